// f64_ops.cuh - FP64 operations of the particle kernels that need not run on
// the FP64 pipe.
//
// This GPU issues FP64 arithmetic, comparisons and FP64 conversions at two
// lanes per clock per SM: one warp instruction of them takes as long as some
// 64 of any other kind. The helpers below give the same results from integer
// instructions on the halves of the word (truncation, conversions, halving,
// tests), or with fewer FP64 instructions (several quotients over one
// divisor). The integer ones are complete over all words: a rare case left to
// the FP64 instruction would be predicated in by the compiler and issued always.
#ifndef EMOO_F64_OPS_CUH
#define EMOO_F64_OPS_CUH

#include <cuda_runtime.h>
#include <stdint.h>

namespace emoo {

// x == x
__device__ __forceinline__ bool f64_not_nan(double x) {
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu, lo = (unsigned)__double2loint(x);
    return hi < 0x7ff00000u || (hi == 0x7ff00000u && lo == 0u);
}

__device__ __forceinline__ bool f64_sign(double x) { return __double2hiint(x) < 0; }

// x == 0, from the halves: the word's low 63 bits compared with 0 are made an
// FP64 comparison by the compiler (seven of them took 2.7 % of a thermal run)
__device__ __forceinline__ bool f64_zero(double x) {
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x)) == 0u;
}

// __double2int_rz(t): truncated, saturated, NaN to the smallest.
__device__ __forceinline__ int f64_trunc(double t) {
    const int hi = __double2hiint(t);
    const unsigned lo = (unsigned)__double2loint(t);
    const int e = ((hi >> 20) & 0x7ff) - 1023;
    const unsigned top = ((unsigned)hi << 11) | (lo >> 21) | 0x80000000u;  // the 32 leading bits
    if (e > 30) return hi < 0 || !f64_not_nan(t) ? (int)0x80000000 : 0x7fffffff;
    const int m = e < 0 ? 0 : (int)(top >> (31 - e));
    return hi < 0 ? -m : m;
}

// (double)i
__device__ __forceinline__ double f64_of_int(int i) {
    const unsigned a = i < 0 ? 0u - (unsigned)i : (unsigned)i;
    const int z = __clz((int)a);
    const unsigned m = a << (z & 31);  // the leading one at bit 31
    const unsigned hi = ((1023u + 31u - (unsigned)z) << 20) | ((m >> 11) & 0xfffffu);
    return a ? __hiloint2double((int)(hi | ((unsigned)i & 0x80000000u)), (int)(m << 21)) : 0.0;
}

// 0.5 * x where neither is denormal: one off the exponent (zero, infinity and
// NaN stay).
__device__ __forceinline__ double f64_half(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), e = hi & 0x7ff00000u;
    return __hiloint2double((int)(e - 1u < 0x7fefffffu ? hi - 0x00100000u : hi), __double2loint(x));
}

// (float)x: to nearest, ties to even
__device__ __forceinline__ float f64_to_f32(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned sign = hi & 0x80000000u;
    const int e = (int)((hi >> 20) & 0x7ffu) - 896;  // the float's exponent field
    unsigned b;
    if (e >= 255) {  // too large, infinite or NaN
        b = f64_not_nan(x) ? 0x7f800000u : 0x7fffffffu;
    } else if (e >= 1) {  // a carry out of the mantissa rounds up the exponent
        b = ((unsigned)e << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
        b += (lo & 0x1fffffffu) > 0x10000000u - (b & 1u) ? 1u : 0u;
    } else {  // denormal or zero: the mantissa shifted down, 30 bits at e = 0
        const int s = 30 - e;
        const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
        if (s > 54) {
            b = 0u;
        } else {
            const unsigned long long half = 1ull << (s - 1), rest = m & (2ull * half - 1ull);
            b = (unsigned)(m >> s);
            b += rest > half - (b & 1u) ? 1u : 0u;
        }
    }
    return __uint_as_float(b | sign);
}

// (double)x
__device__ __forceinline__ double f64_of_f32(float x) {
    const unsigned b = __float_as_uint(x), sign = b & 0x80000000u;
    unsigned e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
    if (e == 0u) {  // zero, or a denormal moved up to a leading one
        if (m == 0u) return __hiloint2double((int)b, 0);
        const int z = __clz((int)m) - 8;
        m = (m << z) & 0x7fffffu;
        e = 1u - (unsigned)z;  // below 0: wraps, and back with the bias
    }
    const unsigned hi = e == 255u ? 0x7ff00000u : (e + 896u) << 20;
    return __hiloint2double((int)(sign | hi | (m >> 3)), (int)(m << 29));
}

// A total order on the words that agrees with < on numbers, zeros apart
// (-0 sorts below +0).
__device__ __forceinline__ long long f64_key(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}

// Quotients over one divisor b. With y = 1 / b correctly rounded, q = a y and
// the exact remainder r = a - b q, fma(r, y, q) is a / b correctly rounded
// (P. Markstein, "Computation of elementary functions on the IBM RISC System
// /6000 processor", IBM J. Res. Dev. 34 (1990) 111): three instructions a
// quotient instead of a division's ten. For a (f64_fit) and b in [2^-500, 2^500),
// where neither the remainder nor the quotient leaves the normal range, and for
// a zero a, whose sign the last addition loses and the integer instruction sets.
// The caller divides for others (fields that vanish, a run that is blowing up).
__device__ __forceinline__ bool f64_ordinary(double x) {
    return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 523u < 1000u;
}

struct F64Quot {
    double b, y;
    bool ordinary;
};

__device__ __forceinline__ F64Quot f64_divisor(double b) {
    F64Quot d;
    d.b = b;
    d.ordinary = f64_ordinary(b);
    d.y = __drcp_rn(b);
    return d;
}

// whether f64_quot takes a
__device__ __forceinline__ bool f64_fit(double a) { return f64_ordinary(a) || f64_zero(a); }

__device__ __forceinline__ double f64_quot(double a, const F64Quot &d) {
    const double q = __dmul_rn(a, d.y), v = __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
    const unsigned sign = (unsigned)(__double2hiint(a) ^ __double2hiint(d.b)) & 0x80000000u;
    return __hiloint2double((int)(((unsigned)__double2hiint(v) & 0x7fffffffu) | sign), __double2loint(v));
}

// 1 / sqrt(b) for b in [1, inf) as y0 (1 + c): y0 the approximation instruction
// (about 20 bits, its low word cleared, so that its square is exact), c from
// one step of Householder's third-order iteration, good to 2^-50 of itself.
// Four instructions on the FP64 pipe.
struct F64Rsqrt {
    double y0, c;
};

__device__ __forceinline__ F64Rsqrt f64_rsqrt(double b) {
    F64Rsqrt r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r.y0) : "d"(b));
    r.y0 = __hiloint2double(__double2hiint(r.y0), 0);
    const double e = __fma_rn(-b, __dmul_rn(r.y0, r.y0), 1.0);
    r.c = __dmul_rn(__fma_rn(0.375, e, 0.5), e);
    return r;
}

}  // namespace emoo

#endif
