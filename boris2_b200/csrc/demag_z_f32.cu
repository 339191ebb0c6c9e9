// 3D z pass, FP32 (demag.cuh)
#include "demag.cuh"

template int launch_zmid<float>(const YZArgs<float> &, cudaStream_t);
