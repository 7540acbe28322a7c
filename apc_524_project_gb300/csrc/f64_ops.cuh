// f64_ops.cuh - FP64 operations of the particle kernels that need not run on
// the FP64 pipe.
//
// This GPU issues FP64 arithmetic, comparisons and FP64 conversions at two
// lanes per clock per SM: one warp instruction of them takes as long as some
// 64 of any other kind. The helpers below give bit-identical results from
// integer instructions on the halves of the word (truncation, conversion of
// small integers, halving, tests), or with fewer FP64 instructions (several
// quotients over one divisor).
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

// __double2int_rz(t): by shifts for |t| < 2^20, by the conversion above.
__device__ __forceinline__ int f64_trunc(double t) {
    const int hi = __double2hiint(t);
    const int e = ((hi >> 20) & 0x7ff) - 1023;
    if (e >= 20) return __double2int_rz(t);
    const int m = e < 0 ? 0 : ((hi & 0xfffff) | 0x100000) >> (20 - e);
    return hi < 0 ? -m : m;
}

// (double)i: assembled for |i| < 2^20 (every cell index of a grid that fits
// the device), by the conversion above.
__device__ __forceinline__ double f64_of_int(int i) {
    const int a = i < 0 ? -i : i;
    if ((unsigned)a >= (1u << 20)) return (double)i;
    const int e = 31 - __clz(a);  // -1 for 0
    const int hi = a ? ((1023 + e) << 20) | ((a << (20 - e)) & 0xfffff) : 0;
    return __hiloint2double(hi | (i & 0x80000000), 0);
}

// 0.5 * x for x that is normally a positive number of ordinary size: one off
// the exponent; zeros, denormals, infinities, NaN and negatives multiply.
__device__ __forceinline__ double f64_half(double x) {
    const int hi = __double2hiint(x);
    if ((unsigned)(hi - 0x00200000) >= 0x7fd00000u) return 0.5 * x;
    return __hiloint2double(hi - 0x00100000, __double2loint(x));
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
// quotient instead of a division's ten. Used where b is of ordinary size;
// for the others (a run that is blowing up) every quotient is divided out.
struct F64Quot {
    double b, y;
    bool plain;
};

__device__ __forceinline__ F64Quot f64_divisor(double b) {
    F64Quot d;
    d.b = b;
    const unsigned e = ((unsigned)__double2hiint(b) >> 20) & 0x7ffu;
    d.plain = e - 523u > 1000u;  // outside [2^-500, 2^500]
    d.y = __drcp_rn(b);
    return d;
}

__device__ __forceinline__ double f64_quot(double a, const F64Quot &d) {
    if (d.plain) return __ddiv_rn(a, d.b);
    const double q = __dmul_rn(a, d.y);
    return __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
}

}  // namespace emoo

#endif
