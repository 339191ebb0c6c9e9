// x-length queries of the stage kernel (stage.cuh) and its launcher; the register kernels of each variant
// and precision and the batched launches are translation units of their own, so that they compile in parallel.
#include "stage.cuh"

extern template int launch_stage_variant<float, 0>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 1>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 2>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 3>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<double, 0>(const StageArgs<double> &, cudaStream_t);
extern template int launch_stage_variant<double, 1>(const StageArgs<double> &, cudaStream_t);
extern template int launch_stage_variant<double, 2>(const StageArgs<double> &, cudaStream_t);

// x lengths with a register kernel and their threads per line
int stage_reg_q(int LX, int xv)
{
    if (xv == 3) xv = 2;   // the radix-16 kernel at the lower register cap: the same shape
    switch (LX) {
    case 16: return xv == 2 ? 0 : xv ? 2 : 4;
    case 32: return xv == 2 ? 0 : xv ? 4 : 8;
    case 64: return xv == 2 ? 0 : 8;
    case 128: return xv == 2 ? 0 : 16;
    case 256: return xv == 2 ? 16 : xv ? 32 : 16;
    case 512: return xv == 2 ? 32 : xv ? 64 : 32;
    case 1024: return xv == 2 ? 64 : xv ? 128 : 32;
    case 24: case 48: case 96: case 192: case 384: case 768:
        return xv == 1 ? LX / 12 : 0;   // Stockham only
    default: return 0;
    }
}

bool stage_reg_path(int LX, int xv)
{
    switch (LX) {
    case 16: case 32: case 64: case 128: case 256: case 512: case 1024: return true;
    case 24: case 48: case 96: case 192: case 384: case 768: return xv != 0;
    default: return false;
    }
}

template int launch_stage<float>(const StageArgs<float> &, cudaStream_t);
template int launch_stage<double>(const StageArgs<double> &, cudaStream_t);
