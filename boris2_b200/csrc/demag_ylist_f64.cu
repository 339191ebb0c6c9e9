// 3D y passes over many meshes per launch with long lines, FP64 (demag_ylist.cuh)
#include "demag_ylist.cuh"

template int launch_ypass_long_batch<double>(int, int, const YZArgs<double> *, const int2 *, int, int, size_t, cudaStream_t);
