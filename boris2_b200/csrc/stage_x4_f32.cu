// Register stage kernels of x-transform variant 4 (FP32 only; stage.cuh, xpair.cuh)
#include "stage.cuh"

template int launch_stage_variant<float, 4>(const StageArgs<float> &, cudaStream_t);
