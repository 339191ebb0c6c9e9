// x transforms of the stage kernel on pairs of adjacent butterflies (FP32, power-of-two LX from 64): the packed
// half spectrum of a row to its real values and back, with packed arithmetic (pairfft.cuh).
//
// What bounds the Stockham x transforms of stage.cuh: instruction issue on shared-memory traffic. They stage
// the spectrum row, split it, run the radix passes and join it, 17 shared accesses of 8 bytes per element and
// stage launch with an address each. Here a thread's butterflies come in adjacent pairs (j, j + 1), whose
// inputs, outputs and twiddles are adjacent too, so a shared access carries two elements as (re, re, im, im),
// all arithmetic is packed, and the split of the spectrum happens in registers: where the spectrum is read (the
// inverse's first pass) and written (the forward's last pass) a thread's two lanes take mirror butterflies, so that
// every element meets its mirror there and the spectrum crosses no shared memory.
// Measured on the 512 x 512 x 16 film: stage launch 188 -> 168 us (of 503 MB: 3.0 TB/s), of which 176 -> 168 by the
// mirror butterflies; 38.0 instead of 47.4 M warp instructions on its half. What bounds it now: load latency at a third
// of the SM's warps (80 registers; long scoreboard 4.8 per issue, L1 52 % and DRAM 25 % busy).
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
// Twiddle tables (float4 (c, c', s, s') for the two lanes): the split's angles pi k / L halved, at the first
// pass' elements [r][t] and at the last pass' [r][q] (mirror butterflies, below); per pass p > 0 the angles
// 2 pi r k / (NS R) of adjacent butterflies as [r - 1][k / 2]; the last pass' of mirror butterflies [r - 1][q].
constexpr int xp_tw_off(int L, int p) { return p <= 0 ? 0 : p == 1 ? L : xp_tw_off(L, p - 1) + (xp_radix(L, p - 1) - 1) * xp_ns(L, p - 1) / 2; }
constexpr int xp_passes(int L) { return xp_radix(L, 3) ? 4 : 3; }
constexpr int xp_tw_last(int L) { return xp_tw_off(L, xp_passes(L)); }

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

// Mirror butterflies: a thread's two lanes take butterflies q and LR - q (q = 0: 0 and LR / 2), whose elements
// k = q + r LR and L - k are each other's mirrors, lane and r reversed; the self-mirrored pair of q = 0 pairs
// within its lanes. So the split finds both of its values in the thread. at(r) visits r = 0, R-1, 1, R-2, ...
template <int R, bool INV, typename F> __device__ __forceinline__ void xp_split_all(c2 (&v)[R], bool q0, F h)
{
    c2 z[R];
#pragma unroll
    for (int o = 0; o < R; o++) {
        const int r = (o & 1) ? R - 1 - o / 2 : o / 2, a = R - 1 - r, b = (R - r) % R;
        const c2 m = {mk<float>(q0 ? v[b].r.x : v[a].r.y, q0 ? v[a].r.y : v[a].r.x),
                      mk<float>(q0 ? v[b].i.x : v[a].i.y, q0 ? v[a].i.y : v[a].i.x)};
        c2 x = v[r];
        if (INV && r == 0) {
            // element 0 carries the two real bins (DC, Nyquist): Z = (x + y, x - y) / 2
            c2 mm = m;
            if (q0) {
                x.i.x = -x.i.x;
                mm.r.x = 0.f;
                mm.i.x = 0.f;
            }
            z[r] = xp_split<INV>(x, mm, h(r));
        } else {
            z[r] = xp_split<INV>(x, m, h(r));
            if (!INV && r == 0 && q0) {
                z[r].r.x = x.r.x + x.i.x;
                z[r].i.x = x.r.x - x.i.x;
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = z[r];
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
    // the forward transform's last pass is xp_last
    if constexpr (!LAST && (INV || P + 2 < xp_passes(L))) xp_pass<L, P + 1, INV>(line, tw, t, act, nkeep);
}

// the first pass' outputs (stride 1) of the butterflies ja and jb in the two lanes
template <int R> __device__ __forceinline__ void xp_store0(float4 *line, int ja, int jb, const c2 *v)
{
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        line[xp_at(ja * (R / 2) + r / 2)] = make_float4(v[r].r.x, v[r + 1].r.x, v[r].i.x, v[r + 1].i.x);
        line[xp_at(jb * (R / 2) + r / 2)] = make_float4(v[r].r.y, v[r + 1].r.y, v[r].i.y, v[r + 1].i.y);
    }
}

// packed half spectrum (global row) -> values as plain complex elements of the line, those below nkeep
template <int L>
__device__ __forceinline__ void xp_inverse(float4 *line, const cpx<float> *__restrict__ src, const float4 *__restrict__ tw, int t,
                                           bool act, int nkeep)
{
    constexpr int T = xp_shape<L>::T, R = xp_radix(L, 0), LR = L / R;
    static_assert(LR == 2 * T, "one pair of mirror butterflies per thread in the first pass");
    if (act) {
        const int jb = t ? LR - t : LR / 2;
        c2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const cpx<float> x0 = src[t + r * LR], x1 = src[jb + r * LR];
            v[r] = {mk<float>(x0.x, x1.x), mk<float>(x0.y, x1.y)};
        }
        xp_split_all<R, true>(v, t == 0, [&](int r) { return tw[r * T + t]; });
        PairFFT<R, true>::run(v);
        xp_store0<R>(line, t, jb, v);
    }
    xp_sync<T>();
    xp_pass<L, 1, true>(line, tw, t, act, nkeep);
}

// the forward transform's last pass on mirror butterflies, split and stored to the global row
template <int L>
__device__ __forceinline__ void xp_last(const float4 *line, cpx<float> *__restrict__ dst, const float4 *__restrict__ tw, int t, bool act)
{
    constexpr int P = xp_passes(L) - 1, R = xp_radix(L, P), LR = L / R, T = xp_shape<L>::T, BP = LR / 2 / T;
    static_assert(xp_ns(L, P) == LR, "last pass");
    const float *f = reinterpret_cast<const float *>(line);
    const float4 *tp = tw + xp_tw_last(L), *th = tw + L / 2;
    if (!act) return;
#pragma unroll
    for (int b = 0; b < BP; b++) {
        const int q = t + T * b, jb = q ? LR - q : LR / 2;
        c2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float *fa = f + 4 * xp_at((q >> 1) + r * (LR / 2)) + (q & 1), *fb = f + 4 * xp_at((jb >> 1) + r * (LR / 2)) + (jb & 1);
            v[r] = {mk<float>(fa[0], fb[0]), mk<float>(fa[2], fb[2])};
            if (r > 0) {
                const float4 w = tp[(r - 1) * (LR / 2) + q];
                const cpx<float> c = mk<float>(w.x, w.y), s = mk<float>(w.z, w.w);
                const c2 x = v[r];
                v[r] = {pk_fma(x.i, s, pk_mul(x.r, c)), pk_sub(pk_mul(x.i, c), pk_mul(x.r, s))};
            }
        }
        PairFFT<R, false>::run(v);
        xp_split_all<R, false>(v, q == 0, [&](int r) { return th[r * (LR / 2) + q]; });
#pragma unroll
        for (int r = 0; r < R; r++) {
            dst[q + r * LR] = mk<float>(v[r].r.x, v[r].i.x);
            dst[jb + r * LR] = mk<float>(v[r].r.y, v[r].i.y);
        }
    }
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
        xp_store0<R>(line, 2 * t, 2 * t + 1, v);
    }
    xp_sync<T>();
    xp_pass<L, 1, false>(line, tw, t, act, L);
    xp_last<L>(line, dst, tw, t, act);
}
