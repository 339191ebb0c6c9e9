// Pairs of values handled together: the two x-adjacent cells 2m and 2m + 1 of one packed x element, or the
// real and imaginary parts of a complex value. In FP32 the arithmetic is the sm_100 packed form (two lanes
// per instruction, each rounded as its scalar counterpart): it runs at the scalar lane rate (125 lane
// operations per clock and SM either way) with half the issue slots, which is what bounds these kernels.
#pragma once
#include "common.cuh"

template <typename T> __device__ __forceinline__ cpx<T> pk_bc(T s) { return mk<T>(s, s); }

#define BM_PK2(name, op)                                                                                      \
    __device__ __forceinline__ cpx<float> name(cpx<float> a, cpx<float> b)                                    \
    {                                                                                                         \
        cpx<float> r;                                                                                         \
        asm("{.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" op                      \
            ".f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;}"                                                        \
            : "=f"(r.x), "=f"(r.y)                                                                            \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                        \
        return r;                                                                                             \
    }
BM_PK2(pk_add, "add.rn")
BM_PK2(pk_sub, "sub.rn")
BM_PK2(pk_mul, "mul.rn")
#undef BM_PK2

// a * b + c
__device__ __forceinline__ cpx<float> pk_fma(cpx<float> a, cpx<float> b, cpx<float> c)
{
    cpx<float> r;
    asm("{.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

__device__ __forceinline__ cpx<double> pk_add(cpx<double> a, cpx<double> b) { return mk<double>(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ cpx<double> pk_sub(cpx<double> a, cpx<double> b) { return mk<double>(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cpx<double> pk_mul(cpx<double> a, cpx<double> b) { return mk<double>(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ cpx<double> pk_fma(cpx<double> a, cpx<double> b, cpx<double> c)
{
    return mk<double>(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
template <typename T> __device__ __forceinline__ cpx<T> pk_neg(cpx<T> a) { return mk<T>(-a.x, -a.y); }
// the pair at p, which is aligned to two values
template <typename T> __device__ __forceinline__ cpx<T> pk_ld(const T *p) { return *reinterpret_cast<const cpx<T> *>(p); }
template <typename T> __device__ __forceinline__ void pk_st(T *p, cpx<T> v) { *reinterpret_cast<cpx<T> *>(p) = v; }
