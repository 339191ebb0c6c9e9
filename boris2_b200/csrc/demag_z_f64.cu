// 3D z pass, FP64 (demag.cuh)
#include "demag.cuh"

template int launch_zmid<double>(const YZArgs<double> &, cudaStream_t);
