// y and z passes over many meshes per launch, FP32 (demag.cuh)
#include "demag.cuh"

template int launch_yz_batch<float>(int, int, const YZArgs<float> *, const int2 *, int, int, size_t, cudaStream_t);
