// Stage kernel over many meshes per launch, FP64 (stage.cuh)
#include "stage.cuh"

template int launch_stage_batch<double>(int, const StageArgs<double> *, const int2 *, int, unsigned int, int, size_t, cudaStream_t, int);
