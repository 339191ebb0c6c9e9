// x transforms of the stage kernel on pairs of adjacent butterflies (FP32, power-of-two LX from 64): the packed
// half spectrum of a row to its real values and back, with packed arithmetic (pairfft.cuh).
//
// What bounds the Stockham x transforms of stage.cuh: instruction issue on shared-memory traffic. They stage
// the spectrum row, split it, run the radix passes and join it, 17 shared accesses of 8 bytes per element and
// stage launch with an address each. Here a thread's butterflies come in adjacent pairs (j, j + 1), whose
// inputs, outputs and twiddles are adjacent too, so a shared access carries two elements as (re, re, im, im),
// all arithmetic is packed, the split of the spectrum is formed from global loads in registers (each element
// and its mirror are read where they are needed), and the row leaves as 16-byte stores.
//
// Measured: 38.6 instead of 49.7 M warp instructions on the 512 x 512 x 8 film; stage launch of the 512 x 512 x
// 16 film 188 -> 176 us (of 503 MB: 2.86 TB/s), of the 128 x 64 film 13.4 -> 11.9 us. What bounds it now: the
// shared-memory and L1 pipe (65 % busy) and the latency of the cell rows behind it (long scoreboard 5 per issue).
//
// Shared line: c2 form for the passes (pair i at i + i / 8: conflict-free for every stride used), plain complex
// order between the inverse and the forward transform, where element m is the pair of cells 2m, 2m + 1.
#pragma once
#include "pairfft.cuh"

template <int L> struct xp_shape {
    static constexpr int V = L >= 256 ? 16 : 8;   // values per thread
    static constexpr int T = L / V;               // threads per line
    static constexpr int LSP = L + L / 8 + 2;     // complex values per shared line
};
// radix of pass p (0 past the last): 8 8 8 for 512, 8 8 4 for 256, 8 8 4 4 for 1024, 4 4 4 2 for 128, 4 4 4 for 64
constexpr int xp_radix(int L, int p)
{
    return p < 0 || p > 3 ? 0
         : L == 512 ? (p < 3 ? 8 : 0)
         : L == 256 ? (p < 2 ? 8 : p == 2 ? 4 : 0)
         : L == 1024 ? (p < 2 ? 8 : 4)
         : L == 128 ? (p < 3 ? 4 : 2)
         : L == 64 ? (p < 3 ? 4 : 0) : 0;
}
constexpr int xp_ns(int L, int p) { return p == 0 ? 1 : xp_ns(L, p - 1) * xp_radix(L, p - 1); }
// twiddle table (float4 pairs (c_k, c_k+1, s_k, s_k+1)): the split's pi k / L halved, then per pass p > 0 the
// angles 2 pi r k / (NS R) as [r - 1][k / 2]
constexpr int xp_tw_off(int L, int p) { return p <= 0 ? 0 : p == 1 ? L / 2 : xp_tw_off(L, p - 1) + (xp_radix(L, p - 1) - 1) * xp_ns(L, p - 1) / 2; }
constexpr int xp_passes(int L) { return xp_radix(L, 3) ? 4 : 3; }
constexpr int xp_tw_len(int L) { return xp_tw_off(L, xp_passes(L)); }

__device__ __forceinline__ int xp_at(int i) { return i + (i >> 3); }

template <int T> __device__ __forceinline__ void xp_sync()
{
    if constexpr (T <= 32) __syncwarp();
    else __syncthreads();
}

// the split of one element pair and its mirrors: inverse Z = E + i O from X (conj of the twiddle), forward
// X = E + w O from Z; h: (c / 2, s / 2)
template <bool INV> __device__ __forceinline__ c2 xp_split(c2 x, c2 m, float4 h)
{
    const cpx<float> c = mk<float>(h.x, h.y), s = mk<float>(h.z, h.w), half = pk_bc<float>(0.5f);
    const cpx<float> a = pk_mul(pk_add(x.r, m.r), half), b = pk_mul(pk_sub(x.i, m.i), half);
    const cpx<float> dr = pk_sub(x.r, m.r), di = pk_add(x.i, m.i);
    if (INV) return {pk_sub(a, pk_fma(di, c, pk_mul(dr, s))), pk_fma(dr, c, pk_sub(b, pk_mul(di, s)))};
    return {pk_fma(di, c, pk_sub(a, pk_mul(dr, s))), pk_sub(b, pk_fma(dr, c, pk_mul(di, s)))};
}

// pass p > 0: from the c2 line to the c2 line (or, the last inverse pass, to plain complex elements < nkeep)
template <int L, int P, bool INV>
__device__ __forceinline__ void xp_pass(float4 *line, const float4 *__restrict__ tw, int t, bool act, int nkeep)
{
    constexpr int T = xp_shape<L>::T, R = xp_radix(L, P), NS = xp_ns(L, P), LR2 = L / R / 2, BP = LR2 / T;
    constexpr bool LAST = P + 1 == xp_passes(L);
    const float4 *tp = tw + xp_tw_off(L, P);
    c2 v[BP][R];
    if (act) {
#pragma unroll
        for (int b = 0; b < BP; b++)
#pragma unroll
            for (int r = 0; r < R; r++) v[b][r] = c2_lds(line + xp_at(t + T * b + r * LR2));
    }
    xp_sync<T>();
    if (act) {
#pragma unroll
        for (int b = 0; b < BP; b++) {
            const int jp = t + T * b, kk = jp & (NS / 2 - 1);
#pragma unroll
            for (int r = 1; r < R; r++) {
                const float4 w = tp[(r - 1) * (NS / 2) + kk];
                const cpx<float> c = mk<float>(w.x, w.y), s = mk<float>(w.z, w.w);
                const c2 x = v[b][r];
                if (INV) v[b][r] = {pk_sub(pk_mul(x.r, c), pk_mul(x.i, s)), pk_fma(x.r, s, pk_mul(x.i, c))};
                else v[b][r] = {pk_fma(x.i, s, pk_mul(x.r, c)), pk_sub(pk_mul(x.i, c), pk_mul(x.r, s))};
            }
            PairFFT<R, INV>::run(v[b]);
            const int o = (jp - kk) * R + kk;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int i = o + r * (NS / 2);
                if (INV && LAST) {
                    if (2 * i < nkeep) c2_st(reinterpret_cast<cpx<float> *>(line) + 2 * i, v[b][r]);
                } else {
                    c2_sts(line + xp_at(i), v[b][r]);
                }
            }
        }
    }
    xp_sync<T>();
    if constexpr (!LAST) xp_pass<L, P + 1, INV>(line, tw, t, act, nkeep);
}

// the first pass' outputs (stride 1): butterfly pairs (j, j + 1) to the adjacent elements of each butterfly
template <int R> __device__ __forceinline__ void xp_store0(float4 *line, int jp, const c2 *v)
{
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        line[xp_at(jp * R + r / 2)] = make_float4(v[r].r.x, v[r + 1].r.x, v[r].i.x, v[r + 1].i.x);
        line[xp_at(jp * R + R / 2 + r / 2)] = make_float4(v[r].r.y, v[r + 1].r.y, v[r].i.y, v[r + 1].i.y);
    }
}

// packed half spectrum (global row) -> values as plain complex elements of the line, those below nkeep
template <int L>
__device__ __forceinline__ void xp_inverse(float4 *line, const cpx<float> *__restrict__ src, const float4 *__restrict__ tw, int t,
                                           bool act, int nkeep)
{
    constexpr int T = xp_shape<L>::T, R = xp_radix(L, 0), LR2 = L / R / 2;
    static_assert(LR2 == T, "one butterfly pair per thread in the first pass");
    if (act) {
        c2 v[R], m[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = 2 * (t + r * LR2);
            v[r] = c2_ld(src + k);
            const cpx<float> m0 = src[(L - k) & (L - 1)], m1 = src[L - k - 1];
            m[r] = {mk<float>(m0.x, m1.x), mk<float>(m0.y, m1.y)};
        }
        if (t == 0) {
            // element 0 carries the two real bins (DC, Nyquist): Z = (x + y, x - y) / 2
            v[0].i.x = -v[0].i.x;
            m[0].r.x = 0.f;
            m[0].i.x = 0.f;
        }
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = xp_split<true>(v[r], m[r], tw[t + r * LR2]);
        PairFFT<R, true>::run(v);
        xp_store0<R>(line, t, v);
    }
    xp_sync<T>();
    xp_pass<L, 1, true>(line, tw, t, act, nkeep);
}

// plain complex elements of the line (zero from L / 2 on, not read there) -> packed half spectrum (global row)
template <int L>
__device__ __forceinline__ void xp_forward(float4 *line, cpx<float> *__restrict__ dst, const float4 *__restrict__ tw, int t, bool act)
{
    constexpr int T = xp_shape<L>::T, R = xp_radix(L, 0), LR2 = L / R / 2;
    c2 v[R];
    if (act) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = {mk<float>(0, 0), mk<float>(0, 0)};
            if (2 * r < R) v[r] = c2_ld(reinterpret_cast<const cpx<float> *>(line) + 2 * (t + r * LR2));
        }
    }
    xp_sync<T>();
    if (act) {
        PairFFT<R, false>::run(v);
        xp_store0<R>(line, t, v);
    }
    xp_sync<T>();
    xp_pass<L, 1, false>(line, tw, t, act, L);
    if (act) {
        const float *f = reinterpret_cast<const float *>(line);
#pragma unroll
        for (int q = 0; q < L / 2 / T; q++) {
            const int i = t + T * q;
            const c2 z = c2_lds(line + xp_at(i));
            // mirrors: element L - 2i is the first lane of pair L/2 - i, element L - 2i - 1 the second of the one before
            const float *f0 = f + 4 * xp_at((L / 2 - i) & (L / 2 - 1)), *f1 = f + 4 * xp_at(L / 2 - 1 - i);
            const c2 m = {mk<float>(f0[0], f1[1]), mk<float>(f0[2], f1[3])};
            c2 x = xp_split<false>(z, m, tw[i]);
            if (q == 0 && t == 0) {
                x.r.x = z.r.x + z.i.x;
                x.i.x = z.r.x - z.i.x;
            }
            c2_st(dst + 2 * i, x);
        }
    }
}
