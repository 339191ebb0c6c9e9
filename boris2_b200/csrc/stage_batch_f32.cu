// Stage kernel over many meshes per launch, FP32 (stage.cuh)
#include "stage.cuh"

template int launch_stage_batch<float>(int, const StageArgs<float> *, const int2 *, int, unsigned int, int, size_t, cudaStream_t, int);
