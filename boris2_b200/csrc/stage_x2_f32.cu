// Register stage kernels of x-transform variant 2, FP32 (stage.cuh)
#include "stage.cuh"

template int launch_stage_variant<float, 2>(const StageArgs<float> &, cudaStream_t);
