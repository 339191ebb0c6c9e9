// Stage kernel, FP64 (stage.cuh)
#include "stage.cuh"

template int launch_stage<double>(const StageArgs<double> &, cudaStream_t);
