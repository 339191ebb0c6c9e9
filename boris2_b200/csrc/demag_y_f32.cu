// 3D y passes, FP32 (demag.cuh)
#include "demag.cuh"

template int launch_yfwd<float>(const YZArgs<float> &, cudaStream_t);
template int launch_yinv<float>(const YZArgs<float> &, cudaStream_t);
