// x-length queries of the stage kernel (stage.cuh) and its launcher; the register kernels of each variant
// and precision and the batched launches are translation units of their own, so that they compile in parallel.
#include "stage.cuh"
#include <cmath>

extern template int launch_stage_variant<float, 0>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 1>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 2>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 3>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<float, 4>(const StageArgs<float> &, cudaStream_t);
extern template int launch_stage_variant<double, 0>(const StageArgs<double> &, cudaStream_t);
extern template int launch_stage_variant<double, 1>(const StageArgs<double> &, cudaStream_t);
extern template int launch_stage_variant<double, 2>(const StageArgs<double> &, cudaStream_t);

// x lengths with a register kernel and their threads per line
int stage_reg_q(int LX, int xv)
{
    if (xv == 4) return (LX == 64 || LX == 128) ? LX / 8 : (LX == 256 || LX == 512 || LX == 1024) ? LX / 16 : 0;
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

std::vector<float> stage_pair_tables(int LX)
{
    std::vector<float> t;
    if (!stage_reg_q(LX, 4)) return t;
    const long double two_pi = 2.0L * 3.141592653589793238462643383279502884L;
    auto put = [&](long double m0, long double m1, long double N, double f) {
        // (c, c', s, s') of 2 pi m / N, FP64 values rounded to FP32
        t.push_back((float)(f * (double)cosl(two_pi * m0 / N)));
        t.push_back((float)(f * (double)cosl(two_pi * m1 / N)));
        t.push_back((float)(f * (double)sinl(two_pi * m0 / N)));
        t.push_back((float)(f * (double)sinl(two_pi * m1 / N)));
    };
    // the split at the mirror butterflies (q, LR - q; 0 and LR / 2) of the first and of the last pass
    const int last = xp_passes(LX) - 1, R0 = xp_radix(LX, 0), RL = xp_radix(LX, last);
    for (int R : {R0, RL})
        for (int r = 0, LR = LX / R; r < R; r++)
            for (int q = 0; q < LR / 2; q++) put(q + r * LR, (q ? LR - q : LR / 2) + r * LR, 2.0L * LX, 0.5);
    for (int p = 1; p <= last; p++) {
        const int R = xp_radix(LX, p), NS = xp_ns(LX, p);
        for (int r = 1; r < R; r++)
            for (int k = 0; k < NS; k += 2) put((long double)r * k, (long double)r * (k + 1), (long double)NS * R, 1.0);
    }
    const int LR = LX / RL;
    for (int r = 1; r < RL; r++)
        for (int q = 0; q < LR / 2; q++) put((long double)r * q, (long double)r * (q ? LR - q : LR / 2), (long double)LX, 1.0);
    return t;
}
