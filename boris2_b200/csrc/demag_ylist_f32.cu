// 3D y passes over many meshes per launch with long lines, FP32, in scalar sums (demag_ylist.cuh)
#define BM_SCALAR_SUMS
#include "demag_ylist.cuh"

template int launch_ypass_long_batch<float>(int, int, const YZArgs<float> *, const int2 *, int, int, size_t, cudaStream_t);
