// 3D z pass on two adjacent columns per thread (FP32, even LX): the register z pass of demag.cuh
// (zmid_reg_body) with packed arithmetic (pairfft.cuh).
//
// What bounds the one-column pass: instruction issue (Nz = 32: 61 % issue active, 1997 warp instructions per
// 32 pencil lines, half of them FP32, the rest loads, addresses and predicates). Here a thread carries the
// pencils of two columns: every butterfly, product and sign is one packed instruction for both, every global
// access is 16 bytes, every shared access 16 (spectra) or 8 (kernel) bytes, and the addresses are shared.
// A thread keeps its own component's spectrum in registers, so the 3 x 3 product reads the other two only.
// Measured (film 512 x 512 x 8, Nz = 16, one launch inside a step): 61.6 -> 58.1 us; warp instructions 41.9 -> 28.3 M.
// At Nz = 32 the 128 value registers and 62 KB of spectra leave 9 warps per SM and the one-column form wins (137 against
// 159 us), so the tuner times both and FP64, which would need twice the registers, has none.
// Thread (c, p, wp), wp fastest; block = 3 components x the mirror pencils ky, Ny - ky x WP column pairs.
#pragma once
#include "kernels.h"
#include "pairfft.cuh"

template <int NZ> constexpr size_t zpair_smem(int WP)
{
    // spectra [3][2][NZ][WP] float4, kernel tile [6][NZ/2+1][2 WP], Nyquist column [6][NZ/2+1], and the
    // packed column's outputs [3][2][NZ] complex
    return (size_t)6 * NZ * WP * 16 + (((size_t)6 * (NZ / 2 + 1) * (2 * WP + 1) * 4 + 15) & ~(size_t)15) + (size_t)6 * NZ * 8;
}

template <int NZ, int WP> __device__ __forceinline__ void zpair_body(const YZArgs<float> &a, int bx, int ky)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int KZ1 = NZ / 2 + 1, W = 2 * WP, H = NZ / 2;
    constexpr int lw = WP == 32 ? 5 : WP == 16 ? 4 : WP == 8 ? 3 : 2;
    const int Ny = a.Ny, nz = a.nz, LX = a.LX;
    const int Kx1 = LX + 1, Ky1 = Ny / 2 + 1;
    float4 *sm = reinterpret_cast<float4 *>(smraw);
    float *Ks = reinterpret_cast<float *>(sm + 6 * NZ * WP);
    float *Kn = Ks + 6 * KZ1 * W;
    const int kx0 = bx * W;
    const int kym = ky == 0 ? 0 : Ny - ky;
    const bool single = (ky == kym);
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long kzs = (long long)Ky1 * Kx1, nk = kzs * KZ1;
    // kernel tile (async): column w of component q for every kz
    for (int idx = tid; idx < 6 * W; idx += nt) {
        const int w = idx & (W - 1), q = idx / W;
        const bool ok = kx0 + w < LX;
        const float *src = a.K + q * nk + (long long)ky * Kx1 + (ok ? kx0 + w : 0);
#pragma unroll
        for (int kz = 0; kz < KZ1; kz++) cp_async_real<float>(&Ks[(q * KZ1 + kz) * W + w], src + kz * kzs, ok);
    }
    if (kx0 == 0)
        for (int idx = tid; idx < 6 * KZ1; idx += nt) {
            const int kz = idx % KZ1, q = idx / KZ1;
            cp_async_real<float>(&Kn[q * KZ1 + kz], &a.K[q * nk + kz * kzs + (long long)ky * Kx1 + LX], true);
        }
    const int wp = tid & (WP - 1), j = tid >> lw;
    const int p = j & 1, c = j >> 1;
    const int kx = kx0 + 2 * wp;
    const bool own = (c < 3) && (p == 0 || !single) && (kx < LX);
    const long long gbase = ((long long)c * nz * Ny + (p ? kym : ky)) * LX + kx;
    const long long gstride = (long long)Ny * LX;
    c2 v[NZ];
#pragma unroll
    for (int e = 0; e < NZ; e++) v[e] = {mk<float>(0, 0), mk<float>(0, 0)};
    if (own) {
#pragma unroll
        for (int e = 0; e < H; e++)
            if (e < nz) v[e] = c2_ld(a.S2 + gbase + e * gstride);
    }
    PairFFT<NZ, false>::run(v);
    if (c < 3) {
        float4 *dst = sm + (size_t)(c * 2 + p) * NZ * WP + wp;
#pragma unroll
        for (int e = 0; e < NZ; e++) c2_sts(dst + e * WP, v[e]);
    }
    cp_async_wait_all();
    __syncthreads();
    if (!own) return;
    // row c of the symmetric 3x3 kernel (xx, yy, zz, xy, xz, yz order): the diagonal, and the components
    // c1, c2 of the other two inputs, with the mirror signs of KernelMultiplication_3D_line
    // (DemagKernel.cpp:85): xy odd in y, xz odd in z, yz odd in both
    const int c1 = c == 0 ? 1 : 0, c2i = c == 2 ? 1 : 2;
    const int q1 = c == 2 ? 4 : 3, q2 = c == 0 ? 4 : 5;
    const float sy = p ? -1.f : 1.f;
    const cpx<float> y1 = pk_bc<float>(q1 == 3 ? sy : 1.f), y2 = pk_bc<float>(q2 == 5 ? sy : 1.f);
    const cpx<float> z1 = pk_bc<float>(q1 == 4 ? -1.f : 1.f), z2 = pk_bc<float>(-1.f);   // q2 is xz or yz: odd in z
    const float4 *s1 = sm + (size_t)(c1 * 2 + p) * NZ * WP + wp, *s2 = sm + (size_t)(c2i * 2 + p) * NZ * WP + wp;
    const float *k0p = Ks + (size_t)c * KZ1 * W + 2 * wp, *k1p = Ks + (size_t)q1 * KZ1 * W + 2 * wp,
                *k2p = Ks + (size_t)q2 * KZ1 * W + 2 * wp;
    // the packed column (kx = 0, the first lane of the block's first pair) needs the untouched spectra and is
    // formed through its own slots in a rolled loop: DC (kernel column 0) + i Nyquist (kernel column LX), the z
    // sign following the primary kz so that both mirror halves see the same kernel values
    cpx<float> *O = reinterpret_cast<cpx<float> *>(smraw + (size_t)6 * NZ * WP * 16 +
                                                   (((size_t)6 * KZ1 * (W + 1) * 4 + 15) & ~(size_t)15)) + (c * 2 + p) * NZ;
    if (kx == 0) {
        const int pm = single ? 0 : 1 - p;
        auto S = [&](int cc, int pp, int e) -> cpx<float> {
            const float4 t = sm[(size_t)((cc * 2 + pp) * NZ + e) * WP];
            return mk<float>(t.x, t.z);
        };
        const int q0 = c;
        const int ci[3] = {c, c1, c2i};
#pragma unroll 1
        for (int kz = 0; kz < NZ; kz++) {
            const int kzm = (NZ - kz) % NZ;
            const int akz = kz <= H ? kz : NZ - kz;
            const int kq = single ? (kz <= H ? kz : kzm) : (p == 0 ? kz : kzm);
            const bool neg = kq > H;
            cpx<float> A[3], B[3];
#pragma unroll
            for (int g = 0; g < 3; g++) {
                const cpx<float> C = S(ci[g], p, kz), cj = conj(S(ci[g], pm, kzm));
                A[g] = cscale(C + cj, 0.5f);
                B[g] = cscale(mul_mi(C - cj), 0.5f);
            }
            const float t1 = neg && q1 == 4 ? -1.f : 1.f, t2 = neg ? -1.f : 1.f;
            const float a0 = Ks[(q0 * KZ1 + akz) * W], a1 = t1 * Ks[(q1 * KZ1 + akz) * W], a2 = t2 * Ks[(q2 * KZ1 + akz) * W];
            const float b0 = Kn[q0 * KZ1 + akz], b1 = t1 * Kn[q1 * KZ1 + akz], b2 = t2 * Kn[q2 * KZ1 + akz];
            const cpx<float> Ap = mk<float>(a0 * A[0].x + a1 * A[1].x + a2 * A[2].x, a0 * A[0].y + a1 * A[1].y + a2 * A[2].y);
            const cpx<float> Bp = mk<float>(b0 * B[0].x + b1 * B[1].x + b2 * B[2].x, b0 * B[0].y + b1 * B[1].y + b2 * B[2].y);
            O[kz] = Ap + mul_i(Bp);
        }
    }
#pragma unroll
    for (int kz = 0; kz <= H; kz++) {
        const cpx<float> a0 = pk_ld<float>(k0p + kz * W), a1 = pk_mul(y1, pk_ld<float>(k1p + kz * W)),
                         a2 = pk_mul(y2, pk_ld<float>(k2p + kz * W));
        {
            const c2 m1 = c2_lds(s1 + kz * WP), m2 = c2_lds(s2 + kz * WP);
            v[kz] = {pk_fma(a2, m2.r, pk_fma(a1, m1.r, pk_mul(a0, v[kz].r))),
                     pk_fma(a2, m2.i, pk_fma(a1, m1.i, pk_mul(a0, v[kz].i)))};
        }
        if (kz > 0 && kz < H) {
            const int kn = NZ - kz;
            const cpx<float> b1 = pk_mul(z1, a1), b2 = pk_mul(z2, a2);
            const c2 m1 = c2_lds(s1 + kn * WP), m2 = c2_lds(s2 + kn * WP);
            v[kn] = {pk_fma(b2, m2.r, pk_fma(b1, m1.r, pk_mul(a0, v[kn].r))),
                     pk_fma(b2, m2.i, pk_fma(b1, m1.i, pk_mul(a0, v[kn].i)))};
        }
    }
    if (kx == 0) {
#pragma unroll
        for (int kz = 0; kz < NZ; kz++) {
            const cpx<float> o = O[kz];
            v[kz].r.x = o.x;
            v[kz].i.x = o.y;
        }
    }
    PairFFT<NZ, true>::run(v);
#pragma unroll
    for (int e = 0; e < H; e++)
        if (e < nz) c2_st(a.S2 + gbase + e * gstride, v[e]);
}

template <int NZ, int WP>
__global__ void __launch_bounds__((6 * WP + 31) / 32 * 32) k_zmid_pair(YZArgs<float> a)
{
    pdl_enter();
    if (gated_out<float>(a.st, a.gate)) return;
    zpair_body<NZ, WP>(a, blockIdx.x, blockIdx.y);
}

template <int NZ, int WP> static int launch_zpair_w(const YZArgs<float> &a, cudaStream_t s)
{
    constexpr int nt = (6 * WP + 31) / 32 * 32;
    constexpr size_t smem = zpair_smem<NZ>(WP);
    if constexpr (smem > 200 * 1024) return 105;
    if (smem > BM_SMEM_DEFAULT_SAFE) {
        cudaError_t e = cudaFuncSetAttribute(k_zmid_pair<NZ, WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, BM_SMEM_CAP);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid((a.LX + 2 * WP - 1) / (2 * WP), a.Ny / 2 + 1);
    return launch_pdl(k_zmid_pair<NZ, WP>, grid, nt, smem, s, a, a.pdl);
}

template <int NZ> static int launch_zpair_n(const YZArgs<float> &a, cudaStream_t s)
{
    switch (a.W) {
    case 8: return launch_zpair_w<NZ, 4>(a, s);
    case 16: return launch_zpair_w<NZ, 8>(a, s);
    case 32: return launch_zpair_w<NZ, 16>(a, s);
    case 64: return launch_zpair_w<NZ, 32>(a, s);
    default: return 104;
    }
}

// the z pass on column pairs, or -1 where it does not apply (zmid_has_pair); a template, so that only the z pass'
// translation unit holds its kernels
template <typename T> static int launch_zmid_pair(const YZArgs<T> &a, cudaStream_t s)
{
    if (!zmid_has_pair(a.Nz, a.W, a.LX)) return -1;
    switch (a.Nz) {
    case 4: return launch_zpair_n<4>(a, s);
    case 6: return launch_zpair_n<6>(a, s);
    case 8: return launch_zpair_n<8>(a, s);
    case 12: return launch_zpair_n<12>(a, s);
    case 16: return launch_zpair_n<16>(a, s);
    case 24: return launch_zpair_n<24>(a, s);
    case 32: return launch_zpair_n<32>(a, s);
    default: return -1;
    }
}
