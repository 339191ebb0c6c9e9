// 3D y passes, FP64 (demag.cuh)
#include "demag.cuh"

template int launch_yfwd<double>(const YZArgs<double> &, cudaStream_t);
template int launch_yinv<double>(const YZArgs<double> &, cudaStream_t);
