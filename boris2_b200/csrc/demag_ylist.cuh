// 3D y passes over many meshes per launch, long lines: two-level of power-of-two length from 64, and the Stockham
// kernels. A translation unit of its own per precision, since FP32 takes scalar sums here (BM_SCALAR_SUMS): with
// packed ones (common.cuh) these kernels lose, unlike the launches of one mesh. Launch of 24 meshes, FP32, scalar
// against packed sums: Ny = 128 10.7 / 13.6 us, 256 11.8 / 14.9, 512 13.8 / 23.8, 1024 16.4 / 23.5; Stockham 384
// inverse 17.4 / 18.4; Ny = 64 7.3 / 7.6, while 32 and below are the same or slower (7.9 / 7.3).
#include "demag.cuh"

template <typename T, bool INV>
static int ypass_long_dispatch(int Ny, const YZArgs<T> *dargs, const int2 *dwork, int nwork, int nt, size_t smem, cudaStream_t s)
{
    switch (Ny) {
    case 64: return launch_ypass_reg_batch<T, 64, INV>(dargs, dwork, nwork, nt, smem, s);
    case 128: return launch_ypass_reg_batch<T, 128, INV>(dargs, dwork, nwork, nt, smem, s);
    case 256: return launch_ypass_reg_batch<T, 256, INV>(dargs, dwork, nwork, nt, smem, s);
    case 512: return launch_ypass_reg_batch<T, 512, INV>(dargs, dwork, nwork, nt, smem, s);
    case 1024: return launch_ypass_reg_batch<T, 1024, INV>(dargs, dwork, nwork, nt, smem, s);
    default: return 111;
    }
}

template <typename T>
int launch_ypass_long_batch(int kind, int Ny, const YZArgs<T> *dargs, const int2 *dwork, int nwork, int nt, size_t smem,
                            cudaStream_t s)
{
    switch (kind) {
    case BM_BATCH_YFWD_ST: return ypass_st_batch_dispatch<T, false>(Ny, dargs, dwork, nwork, nt, smem, s);
    case BM_BATCH_YINV_ST: return ypass_st_batch_dispatch<T, true>(Ny, dargs, dwork, nwork, nt, smem, s);
    case BM_BATCH_YFWD_REG: return ypass_long_dispatch<T, false>(Ny, dargs, dwork, nwork, nt, smem, s);
    case BM_BATCH_YINV_REG: return ypass_long_dispatch<T, true>(Ny, dargs, dwork, nwork, nt, smem, s);
    default: return 110;
    }
}
