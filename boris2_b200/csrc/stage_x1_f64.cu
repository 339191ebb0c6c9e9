// Register stage kernels of x-transform variant 1, FP64 (stage.cuh)
#include "stage.cuh"

template int launch_stage_variant<double, 1>(const StageArgs<double> &, cudaStream_t);
