// Length and shape queries of the y and z passes (demag.cuh) and the 2D pass' instantiations. The other
// passes are instantiated one translation unit per pass and precision, so that they compile in parallel.
#include "demag.cuh"

// lengths with a register z pass
bool zmid_has_reg(int Nz)
{
    return Nz == 4 || Nz == 6 || Nz == 8 || Nz == 12 || Nz == 16 || Nz == 24 || Nz == 32 || Nz == 48 || Nz == 64;
}

// whether the parity-split z pass applies: Nz 12, 16, 24, 32, 48 or 64, a tile width of 8 or 16
bool zmid_has_par(int Nz, int W)
{
    return (Nz == 12 || Nz == 16 || Nz == 24 || Nz == 32 || Nz == 48 || Nz == 64) && (W == 8 || W == 16);
}

// whether the z pass on column pairs applies (FP32): even LX (16-byte rows), a register length up to 32, a
// tile width of 8 to 64 within the shared memory
bool zmid_has_pair(int Nz, int W, int LX)
{
    return LX % 2 == 0 && zmid_has_reg(Nz) && Nz <= 32 && (W == 8 || W == 16 || W == 32 || W == 64) &&
           (size_t)6 * Nz * W * 8 + (size_t)6 * (Nz / 2 + 1) * (W + 1) * 4 + (size_t)6 * Nz * 8 + 16 <= 100 * 1024;
}

int ymid2d_reg_threads(int Ny, int W)
{
    const int q = ysplit_q(Ny);
    const int p = Ny / q;
    return 3 * W * (p > q ? p : q);
}

bool ypass_has_reg(int Ny)
{
    return Ny == 8 || Ny == 16 || Ny == 32 || Ny == 64 || Ny == 128 || Ny == 256 || Ny == 512 || Ny == 1024 || Ny == 12 ||
           Ny == 24 || Ny == 48 || Ny == 96 || Ny == 192 || Ny == 384 || Ny == 768;
}

int ypass_reg_threads(int Ny, int W)
{
    const int q = ysplit_q(Ny);
    const int p = Ny / q;
    return W * (p > q ? p : q);
}

bool ypass_has_st(int Ny)
{
    return Ny == 256 || Ny == 512 || Ny == 1024 || Ny == 2048 || Ny == 192 || Ny == 384 || Ny == 768 || Ny == 1536;
}

int ypass_st_threads(int Ny, int W) { return W * (Ny / (Ny % 3 ? 16 : 12)); }

template int launch_ymid2d<float>(const YZArgs<float> &, cudaStream_t);
template int launch_ymid2d<double>(const YZArgs<double> &, cudaStream_t);
