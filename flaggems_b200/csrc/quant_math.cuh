// Arithmetic of the quantisation rules, for the kernels of quant.cu.  All of it is IEEE fp32: the same inputs give
// the same bits in each of them.
#pragma once
#include "common.cuh"

enum { QM_ACT = 0, QM_GROUP = 1, QM_TOKEN = 2, QM_TENSOR_STATIC = 3, QM_TENSOR_DYNAMIC = 4, QM_INT8_TOKEN = 5 };

__device__ __forceinline__ float ceil_pow2_bits(float v) {
    // 2^ceil(log2(v)) for positive normal v: bump the exponent when any mantissa bit is set.
    uint32_t b = __float_as_uint(v);
    uint32_t e = (b >> 23) & 0xffu;
    uint32_t m = b & 0x7fffffu;
    e += (m != 0u) ? 1u : 0u;
    return __uint_as_float(e << 23);
}

template <int MODE>
__device__ __forceinline__ float make_scale(float amax, float eps, int pow2) {
    if constexpr (MODE == QM_ACT) {
        amax = fmaxf(amax, __uint_as_float(0x38d1b717u));                  // 1e-4
        float s = __fmul_rn(amax, __uint_as_float(0x3b124925u));           // fp32(1/448)
        return pow2 ? ceil_pow2_bits(s) : s;
    } else if constexpr (MODE == QM_GROUP) {
        float s = __fdiv_rn(fmaxf(amax, eps), 448.0f);
        if (pow2) s = ceil_pow2_bits(fmaxf(fabsf(s), __uint_as_float(0x2edbe6ffu)));  // floor 1e-10
        return s;
    } else if constexpr (MODE == QM_INT8_TOKEN) {
        return __fdiv_rn(fmaxf(amax, __uint_as_float(0x2edbe6ffu)), 127.0f);
    } else {
        float s = __fdiv_rn(fmaxf(amax, __uint_as_float(0x2edbe6ffu)), 448.0f);
        return fmaxf(s, __uint_as_float(0x36924925u));                      // 1/(448*512)
    }
}

// Per-group constants for turning x into x/s (or x*(1/s) for QM_ACT).
struct Divider {
    float s, r;
    bool exact_div;
};

template <int MODE>
__device__ __forceinline__ Divider make_divider(float s) {
    Divider d;
    d.s = s;
    d.r = __fdiv_rn(1.0f, s);
    d.exact_div = (MODE != QM_ACT) && ((__float_as_uint(s) & 0x7fffffu) == 0x7fffffu);
    return d;
}

template <int MODE>
__device__ __forceinline__ float apply_divider(float x, const Divider& d) {
    if constexpr (MODE == QM_ACT) {
        return __fmul_rn(x, d.r);
    } else {
        if (d.exact_div) return __fdiv_rn(x, d.s);
        float q0 = __fmul_rn(x, d.r);
        float rem = __fmaf_rn(-q0, d.s, x);
        return __fmaf_rn(rem, d.r, q0);
    }
}

// Two elements at a time with the packed fp32 instructions of sm_100 (mul/fma .f32x2): the same
// IEEE operations as apply_divider, half the issue slots.
template <int MODE>
__device__ __forceinline__ void apply_divider2(float x0, float x1, const Divider& d, float& o0, float& o1) {
    if (MODE != QM_ACT && d.exact_div) {
        o0 = __fdiv_rn(x0, d.s);
        o1 = __fdiv_rn(x1, d.s);
        return;
    }
    uint64_t x, r, q;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(__float_as_uint(x0)), "r"(__float_as_uint(x1)));
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "r"(__float_as_uint(d.r)));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(x), "l"(r));
    if constexpr (MODE != QM_ACT) {
        uint64_t ns, rem;
        asm("mov.b64 %0, {%1, %1};" : "=l"(ns) : "r"(__float_as_uint(-d.s)));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rem) : "l"(q), "l"(ns), "l"(x));   // x - q*s, exact
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(q) : "l"(rem), "l"(r), "l"(q));
    }
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(q));
    o0 = __uint_as_float(lo);
    o1 = __uint_as_float(hi);
}

// Pairs of 16-bit inputs kept as raw words: max|x| is exact in the input type.
template <typename T> struct Pair16;
template <> struct Pair16<__nv_bfloat16> {
    using V = __nv_bfloat162;
    static __device__ __forceinline__ V absmax(V m, uint32_t w) {
        return __hmax2(m, __habs2(*reinterpret_cast<const V*>(&w)));
    }
    static __device__ __forceinline__ float reduce(V m) { return fmaxf(__bfloat162float(m.x), __bfloat162float(m.y)); }
    static __device__ __forceinline__ void widen(uint32_t w, float& lo, float& hi) {
        lo = __uint_as_float(w << 16);
        hi = __uint_as_float(w & 0xffff0000u);
    }
};
template <> struct Pair16<__half> {
    using V = __half2;
    static __device__ __forceinline__ V absmax(V m, uint32_t w) {
        return __hmax2(m, __habs2(*reinterpret_cast<const V*>(&w)));
    }
    static __device__ __forceinline__ float reduce(V m) { return fmaxf(__half2float(m.x), __half2float(m.y)); }
    static __device__ __forceinline__ void widen(uint32_t w, float& lo, float& hi) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
        lo = f.x;
        hi = f.y;
    }
};
