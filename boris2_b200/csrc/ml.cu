// Device passes of the multilayered convolution (the reference's SDemag multilayer branch,
// Boris/SDemag.cpp:786-900; GPU twin SDemagCUDA::UpdateField, Boris/SDemagCUDA.cpp:270, with the
// L x L products of Boris/DemagKernelCollectionCUDA_Mult.cu).
//
//   k_ml_gather   weighted mesh transfer in either direction (CSR lists built on the host)
//   k_zmid_ml     one pass over every layer's (kx, +-ky) pencils: forward z FFT of each layer's
//                 three components, Out_d = sum_s K_ds In_s for every destination d, inverse
//                 z FFT, store; in 2D (Nz = 1) the same pass is the plain L x L product
// The spectra are the single-mesh layout [c][z][y][kx] after the x and y passes (column 0 packs
// the DC and Nyquist x bins), one buffer per layer, all on the common N grid.
#include "ml.h"
#include "kernels.h"
#include "regfft.cuh"

template <typename T>
__device__ __forceinline__ bool ml_gated_out(const StepState *st, int gate)
{
    if (gate == BM_GATE_ALWAYS || st == nullptr) return false;
    if (gate == BM_GATE_ACCEPTED) return *((volatile const int *)&st->reject_flag) != 0;
    if (gate == BM_GATE_ES || gate == BM_GATE_ES_ACC)
        return *((volatile const int *)&st->es_mode) != 1 ||
               (gate == BM_GATE_ES_ACC && *((volatile const int *)&st->reject_flag) != 0);
    return *((volatile const int *)&st->need_restore) == 0;
}

// ------------------------------------------------------------------------------ transfers
template <typename T>
__global__ void k_ml_gather(T *__restrict__ dst, long long n_dst, long long dst_plane, const T *__restrict__ src,
                            long long src_plane, const int *__restrict__ ptr, const int *__restrict__ idx,
                            const T *__restrict__ w, StepState *st, int gate, int add)
{
    if (ml_gated_out<T>(st, gate)) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_dst; i += (long long)gridDim.x * blockDim.x) {
        T v0 = 0, v1 = 0, v2 = 0;
        const int q1 = ptr[i + 1];
        for (int q = ptr[i]; q < q1; q++) {
            const long long e = idx[q];
            const T wq = w[q];
            v0 += wq * src[e];
            v1 += wq * src[e + src_plane];
            v2 += wq * src[e + 2 * src_plane];
        }
        if (add) {
            v0 += dst[i];
            v1 += dst[i + dst_plane];
            v2 += dst[i + 2 * dst_plane];
        }
        dst[i] = v0;
        dst[i + dst_plane] = v1;
        dst[i + 2 * dst_plane] = v2;
    }
}

template <typename T>
int launch_ml_gather(T *dst, long long n_dst, long long dst_plane, const T *src, long long src_plane, const int *ptr,
                     const int *idx, const T *w, StepState *st, int gate, cudaStream_t s, int add)
{
    long long b = (n_dst + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    k_ml_gather<T><<<(int)b, 256, 0, s>>>(dst, n_dst, dst_plane, src, src_plane, ptr, idx, w, st, gate, add);
    return (int)cudaGetLastError();
}

template int launch_ml_gather<float>(float *, long long, long long, const float *, long long, const int *, const int *,
                                     const float *, StepState *, int, cudaStream_t, int);
template int launch_ml_gather<double>(double *, long long, long long, const double *, long long, const int *, const int *,
                                      const double *, StepState *, int, cudaStream_t, int);

// ------------------------------------------------------------------------------ fused z pass
// Block: W columns from kx0, the pencil pair ky / Ny - ky (ky <= Ny/2), every layer and component.
// Thread (l, c, p, w), w fastest, owns one z line of NZ points in registers: it loads layer l's
// component c of pencil p, transforms it forward, and after the shared exchange computes layer
// l's output of component c on that same line, row c of sum_s K_ls In_s, then transforms back.
// Shared memory: In [L][3][2][NZ][W], then one tile per unique kernel with its stored values at
// this block's columns (and at the x Nyquist column kx = Nx/2 that column 0 carries), copied by
// cp.async while the forward transforms run. The stored part and the symmetries that give the
// rest (true DFT values of the real-space tensors):
//   self     ky <= Ny/2, kz <= Nz/2, real; Kxy odd in ky, Kxz odd in kz, Kyz odd in both
//   z-shift  ky <= Ny/2, kz <= Nz/2; Kxy, Kyz odd in ky; K(-kz) = conj(K(kz)) for xx, yy, zz,
//            xy and -conj(K(kz)) for xz, yz
//   full     every ky and kz
// pinv: the kernel was computed for the opposite z shift, so Kxz and Kyz change sign.
// The symmetry signs are per (source, component) pairs of multipliers for the real and the
// imaginary part, one for kz <= Nz/2 and one for kz > Nz/2, applied in the unrolled kz loop.

// multipliers (re, im) of a stored self / z-shift value for kz <= Nz/2 (lo) and kz > Nz/2 (hi)
template <typename T>
__device__ __forceinline__ void ml_signs(int kind, int comp, bool ylo, bool inv, cpx<T> &lo, cpx<T> &hi)
{
    T sy = (!ylo && (comp == 3 || comp == 5)) ? (T)-1 : (T)1;
    if (inv && comp >= 4) sy = -sy;
    lo = mk<T>(sy, sy);
    if (kind == BM_MLK_SELF) hi = mk<T>(comp >= 4 ? -sy : sy, (T)0);
    else hi = (comp >= 4) ? mk<T>(-sy, sy) : mk<T>(sy, -sy);
    if (kind == BM_MLK_SELF) lo.y = (T)0;
}

// one stored value of a kernel at (comp, kz, pencil) of column w (w = -1: Nyquist column)
template <typename T, int NZ>
__device__ __forceinline__ cpx<T> ml_tile_get(const unsigned char *tile, int kind, int comp, int kz, int p, bool ylo, bool inv,
                                              int mainb, int w, int lw)
{
    if (kind == BM_MLK_FULL) {
        const cpx<T> *t = reinterpret_cast<const cpx<T> *>(tile);
        cpx<T> v = (w >= 0) ? t[(((comp * NZ + kz) * 2 + p) << lw) + w]
                            : reinterpret_cast<const cpx<T> *>(tile + mainb)[(comp * NZ + kz) * 2 + p];
        if (inv && comp >= 4) v = mk<T>(-v.x, -v.y);
        return v;
    }
    constexpr int KZ1 = NZ / 2 + 1;
    const int akz = kz <= NZ / 2 ? kz : NZ - kz;
    cpx<T> v;
    if (kind == BM_MLK_SELF) {
        const T *t = reinterpret_cast<const T *>(tile);
        v = mk<T>((w >= 0) ? t[((comp * KZ1 + akz) << lw) + w] : reinterpret_cast<const T *>(tile + mainb)[comp * KZ1 + akz], (T)0);
    } else {
        const cpx<T> *t = reinterpret_cast<const cpx<T> *>(tile);
        v = (w >= 0) ? t[((comp * KZ1 + akz) << lw) + w] : reinterpret_cast<const cpx<T> *>(tile + mainb)[comp * KZ1 + akz];
    }
    cpx<T> lo, hi;
    ml_signs<T>(kind, comp, ylo, inv, lo, hi);
    const cpx<T> sg = kz <= NZ / 2 ? lo : hi;
    return mk<T>(v.x * sg.x, v.y * sg.y);
}

template <int NZ> struct zml_bounds {
    static constexpr int blocks = NZ <= 16 ? 2 : 1;
};

// WC: the tile width as a compile-time constant (0: a.W at run time), so that the shared-memory
// addresses of the products become a base plus an immediate offset
template <typename T, int NZ, int WC>
__global__ void __launch_bounds__(bm_lb<T>::v, zml_bounds<NZ>::blocks) k_zmid_ml(MLZArgs<T> a)
{
    if (ml_gated_out<T>(a.st, a.gate)) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int KZ1 = NZ / 2 + 1;
    const int W = WC ? WC : a.W, L = a.L, Ny = a.Ny, nz = a.nz, LX = a.LX;
    const int lw = WC ? (WC == 32 ? 5 : WC == 16 ? 4 : WC == 8 ? 3 : WC == 4 ? 2 : WC == 2 ? 1 : 0) : __ffs(W) - 1;
    const int Kx1 = LX + 1, Ky1 = Ny / 2 + 1;
    cpx<T> *In = reinterpret_cast<cpx<T> *>(smraw);
    unsigned char *Ks = smraw + (size_t)L * 6 * NZ * W * sizeof(cpx<T>);
    auto IDX = [&](int l, int c, int p, int e, int w) -> int { return ((((l * 3 + c) * 2 + p) * NZ + e) << lw) + w; };
    const int kx0 = blockIdx.x * W;
    const int ky = blockIdx.y, kym = (Ny - ky) % Ny;
    const bool single = (ky == kym);
    const int np = single ? 1 : 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    // kernel tiles (async): thread group g (W threads, one column each) copies rows g, g + ng, ...
    // of every unique kernel, one address computation per element
    {
        const int w = tid & (W - 1), g = tid >> lw, ng = nt >> lw;
        const int kx = kx0 + w;
        const bool okx = kx < LX;
        for (int u = 0; u < a.nu; u++) {
            const MLUDesc d = a.u[u];
            unsigned char *tb = Ks + d.sm;
            const int mainb = zmid_ml_tile_main<T>(d.kind, NZ, W);
            if (d.kind == BM_MLK_FULL) {
                const long long nk = (long long)Kx1 * Ny * NZ;
                const cpx<T> *K = reinterpret_cast<const cpx<T> *>(a.K + d.off);
                cpx<T> *t = reinterpret_cast<cpx<T> *>(tb);
                cpx<T> *tn = reinterpret_cast<cpx<T> *>(tb + mainb);
                for (int j = g; j < 12 * NZ; j += ng) {
                    const int pp = j & 1, kz = (j >> 1) % NZ, comp = (j >> 1) / NZ;
                    const bool ok = okx && pp < np;
                    const long long q = comp * nk + ((long long)kz * Ny + (pp ? kym : ky)) * Kx1;
                    cp_async_cpx<T>(&t[(j << lw) + w], ok ? &K[q + kx] : K, ok);
                    if (kx0 == 0 && w == 0) cp_async_cpx<T>(&tn[j], pp < np ? &K[q + LX] : K, pp < np);
                }
            } else if (d.kind == BM_MLK_SELF) {
                const long long nk = (long long)Kx1 * Ky1 * KZ1;
                const T *K = a.K + d.off;
                T *t = reinterpret_cast<T *>(tb);
                T *tn = reinterpret_cast<T *>(tb + mainb);
                for (int j = g; j < 6 * KZ1; j += ng) {
                    const int kz = j % KZ1, comp = j / KZ1;
                    const long long q = comp * nk + ((long long)kz * Ky1 + ky) * Kx1;
                    cp_async_real<T>(&t[(j << lw) + w], okx ? &K[q + kx] : K, okx);
                    if (kx0 == 0 && w == 0) cp_async_real<T>(&tn[j], &K[q + LX], true);
                }
            } else {
                const long long nk = (long long)Kx1 * Ky1 * KZ1;
                const cpx<T> *K = reinterpret_cast<const cpx<T> *>(a.K + d.off);
                cpx<T> *t = reinterpret_cast<cpx<T> *>(tb);
                cpx<T> *tn = reinterpret_cast<cpx<T> *>(tb + mainb);
                for (int j = g; j < 6 * KZ1; j += ng) {
                    const int kz = j % KZ1, comp = j / KZ1;
                    const long long q = comp * nk + ((long long)kz * Ky1 + ky) * Kx1;
                    cp_async_cpx<T>(&t[(j << lw) + w], okx ? &K[q + kx] : K, okx);
                    if (kx0 == 0 && w == 0) cp_async_cpx<T>(&tn[j], &K[q + LX], true);
                }
            }
        }
    }
    cp_async_commit();
    // forward transforms of the owned lines
    const int w = tid & (W - 1);
    const int p = (tid >> lw) & 1;
    const int lc = tid >> (lw + 1);
    const int l = lc / 3, c = lc - 3 * (lc / 3);
    const int kx = kx0 + w;
    const bool line = (l < L);
    const bool own = line && (p < np) && (kx < LX);
    const int kyp = p ? kym : ky;
    const long long gbase = ((long long)c * nz * Ny + kyp) * LX + kx;
    const long long gstride = (long long)Ny * LX;
    cpx<T> v[NZ];
#pragma unroll
    for (int e = 0; e < NZ; e++) v[e] = mk<T>(0, 0);
    if (own) {
        const cpx<T> *S = a.S2[l];
#pragma unroll
        for (int e = 0; e < (NZ + 1) / 2; e++)
            if (e < nz) v[e] = S[gbase + e * gstride];
    }
    RegFFT<T, NZ, false>::run(v, a.twz, 1);
    if (line) {
#pragma unroll
        for (int e = 0; e < NZ; e++) In[IDX(l, c, p, e, w)] = v[e];
    }
    cp_async_wait_all();
    __syncthreads();
    const int cmp[3] = {c == 0 ? 0 : (c == 1 ? 3 : 4), c == 0 ? 3 : (c == 1 ? 1 : 5), c == 0 ? 4 : (c == 1 ? 5 : 2)};
    // row c of sum_s K_ls In_s on this line
    if (own && kx != 0) {
#pragma unroll
        for (int e = 0; e < NZ; e++) v[e] = mk<T>(0, 0);
        for (int s = 0; s < L; s++) {
            const MLUDesc d = a.u[a.pu[l * L + s]];
            const bool inv = a.pinv[l * L + s] != 0;
            const cpx<T> *t = reinterpret_cast<const cpx<T> *>(Ks + d.sm);
            if (d.kind == BM_MLK_FULL) {
#pragma unroll
                for (int cc = 0; cc < 3; cc++) {
                    const T sg = (inv && cmp[cc] >= 4) ? (T)-1 : (T)1;
                    const cpx<T> *row = t + ((cmp[cc] * NZ * 2 + p) << lw) + w;
                    const cpx<T> *in = In + IDX(s, cc, p, 0, w);
#pragma unroll
                    for (int kz = 0; kz < NZ; kz++) v[kz] = v[kz] + cscale(cmul(row[(kz * 2) << lw], in[kz << lw]), sg);
                }
            } else if (d.kind == BM_MLK_SELF) {
#pragma unroll
                for (int cc = 0; cc < 3; cc++) {
                    cpx<T> lo, hi;
                    ml_signs<T>(d.kind, cmp[cc], p == 0, inv, lo, hi);
                    const T *row = reinterpret_cast<const T *>(Ks + d.sm) + ((cmp[cc] * KZ1) << lw) + w;
                    const cpx<T> *in = In + IDX(s, cc, p, 0, w);
#pragma unroll
                    for (int kz = 0; kz < NZ; kz++) {
                        const int akz = kz <= NZ / 2 ? kz : NZ - kz;
                        const T kr = (kz <= NZ / 2 ? lo.x : hi.x) * row[akz << lw];
                        const cpx<T> x = in[kz << lw];
                        v[kz] = mk<T>(v[kz].x + kr * x.x, v[kz].y + kr * x.y);
                    }
                }
            } else {
#pragma unroll
                for (int cc = 0; cc < 3; cc++) {
                    cpx<T> lo, hi;
                    ml_signs<T>(d.kind, cmp[cc], p == 0, inv, lo, hi);
                    const cpx<T> *row = t + ((cmp[cc] * KZ1) << lw) + w;
                    const cpx<T> *in = In + IDX(s, cc, p, 0, w);
#pragma unroll
                    for (int kz = 0; kz < NZ; kz++) {
                        const int akz = kz <= NZ / 2 ? kz : NZ - kz;
                        const cpx<T> sg = kz <= NZ / 2 ? lo : hi;
                        const cpx<T> kr = row[akz << lw];
                        v[kz] = v[kz] + cmul(mk<T>(kr.x * sg.x, kr.y * sg.y), in[kz << lw]);
                    }
                }
            }
        }
    }
    if (kx0 == 0) {
        // column 0 packs the DC (kx = 0) and Nyquist (kx = Nx/2) spectra; both are unpacked with
        // the Hermitian mirror (pencil 0, kz) <-> (pencil pm, -kz), multiplied and re-packed. The
        // results go through a small shared buffer after the tiles so that the kz loop can stay
        // rolled (only the first block column runs this).
        cpx<T> *O = reinterpret_cast<cpx<T> *>(Ks + a.ksm);
        if (own && kx == 0) {
            const int pm = single ? 0 : 1;
            for (int kz = 0; kz < NZ; kz++) {
                const int kr = p == 0 ? kz : (NZ - kz) % NZ;   // frequency in pencil-0 terms
                const int krm = (NZ - kr) % NZ;
                cpx<T> acc = mk<T>(0, 0);
                for (int s = 0; s < L; s++) {
                    const MLUDesc d = a.u[a.pu[l * L + s]];
                    const bool inv = a.pinv[l * L + s] != 0;
                    const unsigned char *tile = Ks + d.sm;
                    const int mainb = zmid_ml_tile_main<T>(d.kind, NZ, W);
                    cpx<T> ap = mk<T>(0, 0), bp = mk<T>(0, 0);
                    for (int cc = 0; cc < 3; cc++) {
                        const cpx<T> C = In[IDX(s, cc, 0, kr, 0)], cj = conj(In[IDX(s, cc, pm, krm, 0)]);
                        const cpx<T> A = cscale(C + cj, (T)0.5), B = cscale(mul_mi(C - cj), (T)0.5);
                        const cpx<T> k0 = ml_tile_get<T, NZ>(tile, d.kind, cmp[cc], kr, 0, true, inv, mainb, 0, lw);
                        const cpx<T> kn = ml_tile_get<T, NZ>(tile, d.kind, cmp[cc], kr, 0, true, inv, mainb, -1, lw);
                        ap = ap + cmul(k0, A);
                        bp = bp + cmul(kn, B);
                    }
                    acc = acc + (p == 0 ? ap + mul_i(bp) : conj(ap) + mul_i(conj(bp)));
                }
                O[((l * 3 + c) * 2 + p) * NZ + kz] = acc;
            }
        }
        __syncthreads();
        if (own && kx == 0) {
#pragma unroll
            for (int e = 0; e < NZ; e++) v[e] = O[((l * 3 + c) * 2 + p) * NZ + e];
        }
    }
    RegFFT<T, NZ, true>::run(v, a.twz, 1);
    if (own) {
        cpx<T> *S = a.S2[l];
#pragma unroll
        for (int e = 0; e < (NZ + 1) / 2; e++)
            if (e < nz) S[gbase + e * gstride] = v[e];
    }
}

template <typename T, int NZ, int WC>
static int launch_zmid_ml_w(const MLZArgs<T> &a, cudaStream_t s)
{
    int nt = (6 * a.L * a.W + 31) & ~31;
    if (nt > bm_lb<T>::v) return 304;
    size_t smem = zmid_ml_smem<T>(a.L, NZ, a.W, a.ksm);
    if (smem > 200 * 1024) return 305;
    if (smem > BM_SMEM_DEFAULT_SAFE) {
        cudaError_t e = cudaFuncSetAttribute(k_zmid_ml<T, NZ, WC>, cudaFuncAttributeMaxDynamicSharedMemorySize, BM_SMEM_CAP);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid((a.LX + a.W - 1) / a.W, a.Ny / 2 + 1);
    k_zmid_ml<T, NZ, WC><<<grid, nt, smem, s>>>(a);
    return (int)cudaGetLastError();
}

template <typename T, int NZ>
static int launch_zmid_ml_t(const MLZArgs<T> &a, cudaStream_t s)
{
    return a.W == 16 ? launch_zmid_ml_w<T, NZ, 16>(a, s) : launch_zmid_ml_w<T, NZ, 0>(a, s);
}

// ------------------------------------------------------------------------------ z pass, whole vectors per thread
// For short z lines without full (in-plane shifted) kernels: thread (l, w), w fastest, owns all three
// components of layer l on both mirror pencils of column w. The one-line form above reads two shared values
// (an input and a kernel value) per complex product: shared-memory bandwidth bounds it (three layers, Nz = 4:
// 9.5 GB of shared reads for 0.49 GB of spectra, 811 us at 1024 x 1024 x 2 cells). Here the six outputs a
// thread accumulates share every input and every kernel value they use (K is symmetric, and the pencils
// ky, -ky share |K|), a third of the shared reads, and the kernel values come straight from global memory:
// a (destination, source) pair of layers uses its kernel once per column, so staging it would only copy it.
// Measured (three layers, 1024 x 1024 x 2 cells, FFT 2048 x 2048 x 4): 811 -> 613 us, 2.59 TB/s of its 1.59 GB.
// Signs: stored values hold ky, kz >= 0. kz > Nz / 2 takes the conjugate (xx, yy, zz, xy) or minus the
// conjugate (xz, yz); ky < 0 changes the sign of xy and yz; a kernel computed for the opposite z shift that
// of xz and yz (a self kernel is real).
template <typename T, int NZ> struct MLVec {
    static constexpr int KZ1 = NZ / 2 + 1;
    // out[c][p][kz] += row products of one source layer; k6: the six components at akz, in: [c][p] at kz
    template <int KZ, bool REAL>
    __device__ __forceinline__ static void add(const cpx<T> k6[6], const cpx<T> in[3][2], cpx<T> out[3][2][NZ])
    {
        constexpr bool hi = KZ > NZ / 2;
        constexpr int q[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int cc = 0; cc < 3; cc++) {
                const int g = q[c][cc];
                const bool oddz = g >= 4, oddy = g == 3 || g == 5;
                // (re, im) of the value at this kz from the stored one
                T kr = hi && oddz ? -k6[g].x : k6[g].x;
                T ki = hi && !oddz ? -k6[g].y : k6[g].y;
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const T r = (p && oddy) ? -kr : kr, i = (p && oddy) ? -ki : ki;
                    const cpx<T> x = in[cc][p];
                    cpx<T> &o = out[c][p][KZ];
                    if (REAL) o = mk<T>(o.x + r * x.x, o.y + r * x.y);
                    else o = mk<T>(o.x + r * x.x - i * x.y, o.y + r * x.y + i * x.x);
                }
            }
    }
};

// the six stored components of unique kernel d at (akz, |ky|, kx)
template <typename T>
__device__ __forceinline__ void ml_k6(const MLZArgs<T> &a, const MLUDesc &d, bool inv, long long nk, long long at, cpx<T> k6[6])
{
    const T s = inv ? (T)-1 : (T)1;
    if (d.kind == BM_MLK_SELF) {
        const T *K = a.K + d.off + at;
#pragma unroll
        for (int g = 0; g < 6; g++) k6[g] = mk<T>(g >= 4 ? s * K[g * nk] : K[g * nk], (T)0);
    } else {
        const cpx<T> *K = reinterpret_cast<const cpx<T> *>(a.K + d.off) + at;
#pragma unroll
        for (int g = 0; g < 6; g++) {
            k6[g] = K[g * nk];
            if (g >= 4) k6[g] = cscale(k6[g], s);
        }
    }
}

template <typename T, int NZ, int KZ>
__device__ __forceinline__ void ml_vec_kz(const cpx<T> k6[6], bool real, const cpx<T> *in, int W, cpx<T> out[3][2][NZ])
{
    cpx<T> x[3][2];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int p = 0; p < 2; p++) x[c][p] = in[((c * 2 + p) * NZ + KZ) * W];
    if (real) MLVec<T, NZ>::template add<KZ, true>(k6, x, out);
    else MLVec<T, NZ>::template add<KZ, false>(k6, x, out);
}
template <typename T, int NZ, int AKZ>
__device__ __forceinline__ void ml_vec_src(const MLZArgs<T> &a, const MLUDesc &d, bool inv, long long nk, long long at, long long kzs,
                                           const cpx<T> *in, int W, cpx<T> out[3][2][NZ])
{
    if constexpr (AKZ <= NZ / 2) {
        cpx<T> k6[6];
        ml_k6<T>(a, d, inv, nk, at + AKZ * kzs, k6);
        const bool real = d.kind == BM_MLK_SELF;
        ml_vec_kz<T, NZ, AKZ>(k6, real, in, W, out);
        if constexpr (AKZ > 0 && 2 * AKZ < NZ) ml_vec_kz<T, NZ, NZ - AKZ>(k6, real, in, W, out);
        ml_vec_src<T, NZ, AKZ + 1>(a, d, inv, nk, at, kzs, in, W, out);
    }
}

template <typename T, int NZ>
__global__ void __launch_bounds__(256) k_zmid_mlv(MLZArgs<T> a)
{
    if (ml_gated_out<T>(a.st, a.gate)) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int KZ1 = NZ / 2 + 1, H = (NZ + 1) / 2;
    const int W = a.W, L = a.L, Ny = a.Ny, nz = a.nz, LX = a.LX, lw = __ffs(W) - 1;
    cpx<T> *In = reinterpret_cast<cpx<T> *>(smraw);                    // [L][3][2][NZ][W]
    cpx<T> *O = In + (size_t)L * 6 * NZ * W;                           // column 0's outputs [L][3][2][NZ]
    const int kx0 = blockIdx.x * W, ky = blockIdx.y, kym = ky == 0 ? 0 : Ny - ky;
    const bool single = (ky == kym);
    const int w = threadIdx.x & (W - 1), l = threadIdx.x >> lw, kx = kx0 + w;
    const bool own = l < L && kx < LX;
    const long long kzs = (long long)(Ny / 2 + 1) * (LX + 1), nk = kzs * KZ1, at = (long long)ky * (LX + 1) + kx;
    const long long gstride = (long long)Ny * LX;
    cpx<T> *S = a.S2[l < L ? l : 0];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int p = 0; p < 2; p++) {
            cpx<T> v[NZ];
#pragma unroll
            for (int e = 0; e < NZ; e++) v[e] = mk<T>(0, 0);
            if (own && !(p && single)) {
                const cpx<T> *src = S + ((long long)c * nz * Ny + (p ? kym : ky)) * LX + kx;
#pragma unroll
                for (int e = 0; e < H; e++)
                    if (e < nz) v[e] = src[e * gstride];
            }
            RegFFT<T, NZ, false>::run(v, a.twz, 1);
            if (l < L) {
#pragma unroll
                for (int e = 0; e < NZ; e++) In[(((l * 3 + c) * 2 + p) * NZ + e) * W + w] = v[e];
            }
        }
    __syncthreads();
    cpx<T> out[3][2][NZ];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int e = 0; e < NZ; e++) out[c][p][e] = mk<T>(0, 0);
    if (own) {
#pragma unroll 1
        for (int s = 0; s < L; s++)
            ml_vec_src<T, NZ, 0>(a, a.u[a.pu[l * L + s]], a.pinv[l * L + s] != 0, nk, at, kzs, In + (size_t)s * 6 * NZ * W + w, W,
                                 out);
    }
    if (kx0 == 0) {
        // column 0 packs the DC (kx = 0) and Nyquist (kx = Nx / 2) spectra: unpacked with the Hermitian mirror
        // (pencil 0, kz) <-> (pencil pm, -kz), multiplied by their own kernel columns, re-packed
        if (own && kx == 0) {
            const int pm = single ? 0 : 1;
#pragma unroll 1
            for (int kz = 0; kz < NZ; kz++) {
                const int kzm = (NZ - kz) % NZ, akz = kz <= NZ / 2 ? kz : NZ - kz;
                const bool hi = kz > NZ / 2;
                cpx<T> ap[3], bp[3];
#pragma unroll
                for (int c = 0; c < 3; c++) ap[c] = bp[c] = mk<T>(0, 0);
#pragma unroll 1
                for (int s = 0; s < L; s++) {
                    const MLUDesc d = a.u[a.pu[l * L + s]];
                    const bool inv = a.pinv[l * L + s] != 0;
                    cpx<T> k0[6], kn[6];
                    ml_k6<T>(a, d, inv, nk, at + akz * kzs, k0);
                    ml_k6<T>(a, d, inv, nk, at + akz * kzs + LX, kn);
#pragma unroll
                    for (int g = 0; g < 6; g++)
                        if (hi) {
                            k0[g] = g >= 4 ? mk<T>(-k0[g].x, k0[g].y) : conj(k0[g]);
                            kn[g] = g >= 4 ? mk<T>(-kn[g].x, kn[g].y) : conj(kn[g]);
                        }
                    constexpr int q[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
                    const cpx<T> *in = In + (size_t)s * 6 * NZ * W;
#pragma unroll
                    for (int cc = 0; cc < 3; cc++) {
                        const cpx<T> C = in[((cc * 2) * NZ + kz) * W], cj = conj(in[((cc * 2 + pm) * NZ + kzm) * W]);
                        const cpx<T> A = cscale(C + cj, (T)0.5), B = cscale(mul_mi(C - cj), (T)0.5);
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            ap[c] = ap[c] + cmul(k0[q[c][cc]], A);
                            bp[c] = bp[c] + cmul(kn[q[c][cc]], B);
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    O[((l * 3 + c) * 2) * NZ + kz] = ap[c] + mul_i(bp[c]);
                    if (!single) O[((l * 3 + c) * 2 + 1) * NZ + kzm] = conj(ap[c]) + mul_i(conj(bp[c]));
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int e = 0; e < NZ; e++)
                        if (!(p && single)) out[c][p][e] = O[((l * 3 + c) * 2 + p) * NZ + e];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int p = 0; p < 2; p++) {
            RegFFT<T, NZ, true>::run(out[c][p], a.twz, 1);
            if (own && !(p && single)) {
                cpx<T> *dst = S + ((long long)c * nz * Ny + (p ? kym : ky)) * LX + kx;
#pragma unroll
                for (int e = 0; e < H; e++)
                    if (e < nz) dst[e * gstride] = out[c][p][e];
            }
        }
}

template <typename T> size_t zmid_mlv_smem(int L, int Nz, int W) { return (size_t)L * 6 * Nz * (W + 1) * sizeof(cpx<T>); }

// whether the whole-vector form applies: z lines that fit the registers (FP32 up to 8 points, FP64 up to 4), no
// full kernels, whole warps of at most 256 threads
template <typename T> bool zmid_ml_has_vec(const MLZArgs<T> &a)
{
    if (!(a.Nz == 1 || a.Nz == 4 || (sizeof(T) == 4 && (a.Nz == 6 || a.Nz == 8)))) return false;
    for (int u = 0; u < a.nu; u++)
        if (a.u[u].kind == BM_MLK_FULL) return false;
    return a.W >= 8 && (a.W & (a.W - 1)) == 0 && a.L * a.W <= 256 && zmid_mlv_smem<T>(a.L, a.Nz, a.W) <= 100 * 1024;
}

template <typename T, int NZ> static int launch_zmid_mlv(const MLZArgs<T> &a, cudaStream_t s)
{
    const int nt = (a.L * a.W + 31) & ~31;
    const size_t smem = zmid_mlv_smem<T>(a.L, NZ, a.W);
    if (smem > BM_SMEM_DEFAULT_SAFE) {
        cudaError_t e = cudaFuncSetAttribute(k_zmid_mlv<T, NZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, BM_SMEM_CAP);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid((a.LX + a.W - 1) / a.W, a.Ny / 2 + 1);
    k_zmid_mlv<T, NZ><<<grid, nt, smem, s>>>(a);
    return (int)cudaGetLastError();
}
template bool zmid_ml_has_vec<float>(const MLZArgs<float> &);
template bool zmid_ml_has_vec<double>(const MLZArgs<double> &);

bool zmid_ml_supported(int Nz)
{
    return Nz == 1 || Nz == 4 || Nz == 6 || Nz == 8 || Nz == 12 || Nz == 16 || Nz == 24 || Nz == 32 || Nz == 48 || Nz == 64;
}

template <typename T> int launch_zmid_ml(const MLZArgs<T> &a, cudaStream_t s)
{
    if (a.W < 1 || (a.W & (a.W - 1)) || a.L < 1 || a.L > BM_ML_MAXL) return 301;
    if (a.vec && zmid_ml_has_vec<T>(a)) {
        if (a.Nz == 1) return launch_zmid_mlv<T, 1>(a, s);
        if (a.Nz == 4) return launch_zmid_mlv<T, 4>(a, s);
        if constexpr (sizeof(T) == 4) return a.Nz == 6 ? launch_zmid_mlv<T, 6>(a, s) : launch_zmid_mlv<T, 8>(a, s);
    }
    switch (a.Nz) {
    case 1: return launch_zmid_ml_t<T, 1>(a, s);
    case 4: return launch_zmid_ml_t<T, 4>(a, s);
    case 6: return launch_zmid_ml_t<T, 6>(a, s);
    case 8: return launch_zmid_ml_t<T, 8>(a, s);
    case 12: return launch_zmid_ml_t<T, 12>(a, s);
    case 16: return launch_zmid_ml_t<T, 16>(a, s);
    case 24: return launch_zmid_ml_t<T, 24>(a, s);
    case 32: return launch_zmid_ml_t<T, 32>(a, s);
    case 48: return launch_zmid_ml_t<T, 48>(a, s);
    case 64: return launch_zmid_ml_t<T, 64>(a, s);
    default: return 302;
    }
}

template int launch_zmid_ml<float>(const MLZArgs<float> &, cudaStream_t);
template int launch_zmid_ml<double>(const MLZArgs<double> &, cudaStream_t);
