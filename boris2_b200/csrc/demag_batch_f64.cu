// y and z passes over many meshes per launch, FP64 (demag.cuh)
#include "demag.cuh"

template int launch_yz_batch<double>(int, int, const YZArgs<double> *, const int2 *, int, int, size_t, cudaStream_t);
