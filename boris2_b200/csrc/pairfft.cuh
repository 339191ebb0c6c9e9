// Register FFTs on two lines at once (FP32): a c2 holds the real parts of the two lines' values as one pair
// and the imaginary parts as another, so every butterfly and twiddle product is packed arithmetic
// (pair.cuh) without any exchange between the lanes. Twiddles are compile-time constants, computed here in
// FP64 from the Taylor series on [0, pi / 4] and rounded to FP32, as the host tables are.
#pragma once
#include "pair.cuh"
#include <utility>

struct c2 {
    cpx<float> r, i;
};
__device__ __forceinline__ c2 operator+(c2 a, c2 b) { return {pk_add(a.r, b.r), pk_add(a.i, b.i)}; }
__device__ __forceinline__ c2 operator-(c2 a, c2 b) { return {pk_sub(a.r, b.r), pk_sub(a.i, b.i)}; }
// two adjacent complex values of a line row: (re0, im0, re1, im1)
__device__ __forceinline__ c2 c2_ld(const cpx<float> *p)
{
    const float4 v = *reinterpret_cast<const float4 *>(p);
    return {mk<float>(v.x, v.z), mk<float>(v.y, v.w)};
}
__device__ __forceinline__ void c2_st(cpx<float> *p, c2 v)
{
    *reinterpret_cast<float4 *>(p) = make_float4(v.r.x, v.i.x, v.r.y, v.i.y);
}
// the same two values in shared memory, kept as pairs: (re0, re1, im0, im1)
__device__ __forceinline__ c2 c2_lds(const float4 *p)
{
    const float4 v = *p;
    return {mk<float>(v.x, v.y), mk<float>(v.z, v.w)};
}
__device__ __forceinline__ void c2_sts(float4 *p, c2 v) { *p = make_float4(v.r.x, v.r.y, v.i.x, v.i.y); }

namespace pf {
constexpr double kPi = 3.14159265358979323846;
constexpr double series(double x, bool cosine)   // cos x or sin x, |x| <= pi / 4
{
    double t = cosine ? 1.0 : x, s = t;
    for (int k = cosine ? 1 : 2; k < 24; k += 2) {
        t *= -x * x / (double)(k * (k + 1));
        s += t;
    }
    return s;
}
constexpr double cosn(long long m, long long N)   // cos(2 pi m / N)
{
    m %= N;
    if (m < 0) m += N;
    if (2 * m > N) m = N - m;                          // cos even
    if (4 * m > N) return -cosn(N - 2 * m, 2 * N);     // cos(pi - x) = -cos x
    if (8 * m > N) return series(kPi / 2 - 2 * kPi * (double)m / (double)N, false);
    return series(2 * kPi * (double)m / (double)N, true);
}
constexpr double sinn(long long m, long long N) { return cosn(4 * m - N, 4 * N); }   // cos(x - pi / 2)
}  // namespace pf

// v * exp(-+ 2 pi i M / N) (forward -, inverse +)
template <int M, int N, bool INV> __device__ __forceinline__ c2 c2_tw(c2 v)
{
    constexpr int m = ((M % N) + N) % N;
    if constexpr (m == 0) return v;
    else if constexpr (2 * m == N) return {pk_neg(v.r), pk_neg(v.i)};
    else if constexpr (4 * m == N) return INV ? c2{pk_neg(v.i), v.r} : c2{v.i, pk_neg(v.r)};
    else if constexpr (4 * m == 3 * N) return INV ? c2{v.i, pk_neg(v.r)} : c2{pk_neg(v.i), v.r};
    else {
        constexpr float c = (float)pf::cosn(m, N), s = (float)((INV ? 1.0 : -1.0) * pf::sinn(m, N));
        return {pk_fma(v.i, pk_bc<float>(-s), pk_mul(v.r, pk_bc<float>(c))),
                pk_fma(v.r, pk_bc<float>(s), pk_mul(v.i, pk_bc<float>(c)))};
    }
}

template <int N> struct pf_split {
    static constexpr int n1 = (N % 4 == 0 && N / 4 >= 2) ? 4 : (N % 3 == 0 && N / 3 >= 2) ? 3 : 2;
    static constexpr int n2 = N / n1;
};
// compile-time loop over [0, N)
template <int... I, typename F> __device__ __forceinline__ void pf_for_(std::integer_sequence<int, I...>, F f)
{
    (f(std::integral_constant<int, I>()), ...);
}
template <int N, typename F> __device__ __forceinline__ void pf_for(F f) { pf_for_(std::make_integer_sequence<int, N>(), f); }

// in-place DFT of N = 2^p or 3 * 2^p values, natural order in and out
template <int N, bool INV> struct PairFFT {
    __device__ __forceinline__ static void run(c2 *v)
    {
        constexpr int N1 = pf_split<N>::n1, N2 = pf_split<N>::n2;
        c2 u[N1][N2];
#pragma unroll
        for (int a = 0; a < N1; a++) {
#pragma unroll
            for (int b = 0; b < N2; b++) u[a][b] = v[a + N1 * b];
            PairFFT<N2, INV>::run(u[a]);
        }
        pf_for<N2>([&](auto ib) {
            constexpr int b = decltype(ib)::value;
            c2 t[N1];
            pf_for<N1>([&](auto ia) {
                constexpr int a = decltype(ia)::value;
                t[a] = c2_tw<a * b, N, INV>(u[a][b]);
            });
            PairFFT<N1, INV>::run(t);
#pragma unroll
            for (int a = 0; a < N1; a++) v[b + N2 * a] = t[a];
        });
    }
};
template <bool INV> struct PairFFT<1, INV> {
    __device__ __forceinline__ static void run(c2 *) {}
};
template <bool INV> struct PairFFT<2, INV> {
    __device__ __forceinline__ static void run(c2 *v)
    {
        const c2 a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    }
};
template <bool INV> struct PairFFT<3, INV> {
    __device__ __forceinline__ static void run(c2 *v)
    {
        const cpx<float> c = pk_bc<float>(-0.5f), s = pk_bc<float>(INV ? 0.86602540378443864676f : -0.86602540378443864676f);
        const cpx<float> n = pk_bc<float>(INV ? -0.86602540378443864676f : 0.86602540378443864676f);
        const c2 a = v[0], sum = v[1] + v[2], d = v[1] - v[2];
        const c2 m = {pk_fma(c, sum.r, a.r), pk_fma(c, sum.i, a.i)};
        v[0] = a + sum;
        // m +- (+-i s) d
        v[1] = {pk_fma(n, d.i, m.r), pk_fma(s, d.r, m.i)};
        v[2] = {pk_fma(s, d.i, m.r), pk_fma(n, d.r, m.i)};
    }
};
template <bool INV> struct PairFFT<4, INV> {
    __device__ __forceinline__ static void run(c2 *v)
    {
        const c2 a0 = v[0] + v[2], a1 = v[0] - v[2], b0 = v[1] + v[3], d = v[1] - v[3];
        v[0] = a0 + b0;
        v[2] = a0 - b0;
        const c2 p = {pk_sub(a1.r, d.i), pk_add(a1.i, d.r)}, m = {pk_add(a1.r, d.i), pk_sub(a1.i, d.r)};   // a1 +- i d
        v[1] = INV ? p : m;
        v[3] = INV ? m : p;
    }
};
