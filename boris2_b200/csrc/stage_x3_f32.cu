// Register stage kernels of x-transform variant 3, FP32 (stage.cuh)
#include "stage.cuh"

template int launch_stage_variant<float, 3>(const StageArgs<float> &, cudaStream_t);
