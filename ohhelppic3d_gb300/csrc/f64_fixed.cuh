// f64_fixed.cuh -- cell, offset and 2^-48 fixed-point CIC weights of FP64
// coordinates, shared by the FP64 tile kernels (push_f64.cu) and the subdomain
// kernels (subdomain.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ohpic_internal.cuh"

namespace ohpic {
namespace {

constexpr unsigned long long kOne48 = 1ull << 48;

// Cell index and in-cell offset of a coordinate by integer operations on its
// bit pattern.  On GB300 the FP64 pipe bounds this form, and (int)x,
// (double)ix, x - ix and the 48-bit rounding were six of its operations per axis.
// A coordinate is kept as (fr, e): for x >= 1, e is its binary exponent and fr
// the mantissa bits below the binary point, so the offset is fr * 2^(e-52); for
// x in [0, 1) (and -0.0), e = -1 and fr holds the bits of x itself.
struct Split {
    unsigned long long fr;
    int e;
};

// floor(x) for x in [0, 2^30); -1 for anything else (negative, NaN, too large).
__device__ __forceinline__ int split_cell(double x, Split &s)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)(b >> 52);                       // the sign bit makes negatives >= 2048
    if (E < 1023 || b == 0x8000000000000000ull) {       // [0, 1) and -0.0: cell 0, offset x
        s.fr = b;
        s.e = -1;
        return 0;
    }
    s.e = E - 1023;
    if (s.e > 29) return -1;
    const unsigned long long F = (b & ((1ull << 52) - 1)) | (1ull << 52);
    const int sh = 52 - s.e;
    s.fr = F & ((1ull << sh) - 1);
    return (int)(F >> sh);
}

// The offset x - floor(x) as a double, exact (the same bits FP64 subtraction gives).
__device__ __forceinline__ double split_frac(const Split &s)
{
    if (s.e < 0) return __longlong_as_double((long long)s.fr);
    if (s.fr == 0) return 0.0;
    const int p = 63 - __clzll((long long)s.fr);       // top set bit; the value is 2^(p+e-52) * 1.m
    const unsigned long long mant = (s.fr << (52 - p)) & ((1ull << 52) - 1);
    return __longlong_as_double((long long)(((unsigned long long)(p + s.e + 971) << 52) | mant));
}

// A weight in (0, 1] as an integer pair: m * 2^(e - 63) with bit 63 of m set and its
// low 11 bits clear (53 significant bits).  Products of weights are formed and
// rounded (to nearest, ties to even) on the integer pipes, with the bits an FP64
// multiply gives: a multiply occupies an SM partition's FP64 pipe for 64 cycles, its
// integer form issues about 30 instructions on pipes that are otherwise idle.
struct Unit {
    unsigned long long m;
    int e;
};

// f * 2^-k for 0 < f <= 2^k, k <= 52.
__device__ __forceinline__ Unit unit_of(unsigned long long f, int k)
{
    const int lz = __clzll((long long)f);
    return Unit{f << lz, 63 - lz - k};
}

// A positive normal double.
__device__ __forceinline__ Unit unit_of_bits(unsigned long long b)
{
    return Unit{((b << 11) | (1ull << 63)), (int)(b >> 52) - 1023};
}

__device__ __forceinline__ Unit unit_mul(const Unit &a, const Unit &b)
{
    unsigned long long hi = __umul64hi(a.m, b.m), lo = a.m * b.m;
    const int s = (int)(hi >> 63) ^ 1;         // the product's top bit is 63 or 62
    hi = (hi << s) | ((lo >> 63) & (unsigned long long)s);
    lo <<= s;
    hi |= (unsigned long long)(lo != 0);        // sticky: the low 11 bits round
    const unsigned long long t = hi + (0x3ffull + ((hi >> 11) & 1ull));
    Unit r;
    r.e = a.e + b.e + 1 - s;
    r.m = t & ~0x7ffull;
    if (t < hi) {                               // rounded up to the next power of two
        r.m = 1ull << 63;
        ++r.e;
    }
    return r;
}

__device__ __forceinline__ double unit_double(const Unit &a)
{
    return __longlong_as_double((long long)(((unsigned long long)(a.e + 1022) << 52) + (a.m >> 11)));
}

// 1 - x for a positive normal x < 1 (its bits), rounded as the FP64 subtraction rounds
// it: a multiple of 2^-53, exact from x = 1/2 on.
__device__ __forceinline__ Unit unit_one_minus(unsigned long long b)
{
    const unsigned long long M = (b & ((1ull << 52) - 1)) | (1ull << 52);
    const int s = min(1022 - (int)(b >> 52), 63);        // x 2^53 = M 2^-s
    const unsigned long long q = M >> s, rem = M & ((1ull << s) - 1), half = (1ull << s) >> 1;
    unsigned long long R = (1ull << 53) - q;             // 2^53 - x 2^53, its fraction not yet taken off
    R -= rem > half || (rem == half && rem != 0 && (R & 1ull));
    return unit_of(R, 53);
}

// The two weights (r and 1 - r) of an axis; false when either is zero or too small for
// the integer products (an offset that is zero or, in cell 0, below 2^-300).
__device__ __forceinline__ bool split_units(const Split &s, Unit &r, Unit &c)
{
    if (s.e >= 0) {
        const int k = 52 - s.e;
        if (s.fr == 0) return false;
        r = unit_of(s.fr, k);
        c = unit_of((1ull << k) - s.fr, k);
        return true;
    }
    if ((int)(s.fr >> 52) < 1023 - 300 || (long long)s.fr < 0) return false;
    r = unit_of_bits(s.fr);
    c = unit_one_minus(s.fr);
    return true;
}

// round(offset * 2^48), ties up.
__device__ __forceinline__ unsigned long long split_frac48(const Split &s)
{
    if (s.e >= 4) return s.fr << (s.e - 4);
    if (s.e >= 0) {
        const int sh = 4 - s.e;
        return (s.fr + (1ull << (sh - 1))) >> sh;
    }
    const int E = (int)((s.fr >> 52) & 0x7ff);           // x in [0, 1): x * 2^48 = F * 2^(E - 1027)
    if (E == 0) return 0;
    const int sh = 1027 - E;                            // >= 5
    if (sh > 54) return 0;
    const unsigned long long F = (s.fr & ((1ull << 52) - 1)) | (1ull << 52);
    return (F + (1ull << (sh - 1))) >> sh;
}

// round(p * w / 2^48) for p, w <= 2^48, from the 96-bit product.
__device__ __forceinline__ unsigned long long mul48(unsigned long long p, unsigned long long w)
{
    const unsigned long long hi = __umul64hi(p, w), lo = p * w;
    const unsigned long long q = (hi << 16) | (lo >> 48);
    return q + ((lo >> 47) & 1ull);
}

// The 8 weights of a particle whose offsets are Rx, Ry, Rz (units of 2^-48), in
// units of 2^-48, summing to exactly 2^48; order x fastest.
__device__ __forceinline__ void fixed_weights48(int conv, unsigned long long Rx, unsigned long long Ry,
                                                unsigned long long Rz, unsigned long long u[8])
{
    const bool ref = conv == OHPIC_WEIGHTS_REFERENCE;   // node floor(x) takes r (linear_scatter.f90:41-42)
    const unsigned long long X1 = ref ? kOne48 - Rx : Rx, X0 = kOne48 - X1;
    const unsigned long long wy1 = ref ? kOne48 - Ry : Ry, wz1 = ref ? kOne48 - Rz : Rz;
    const unsigned long long Y01 = min(mul48(X0, wy1), X0), Y11 = min(mul48(X1, wy1), X1);
    const unsigned long long Y00 = X0 - Y01, Y10 = X1 - Y11;
    const unsigned long long Z00 = min(mul48(Y00, wz1), Y00), Z10 = min(mul48(Y10, wz1), Y10);
    const unsigned long long Z01 = min(mul48(Y01, wz1), Y01), Z11 = min(mul48(Y11, wz1), Y11);
    u[0] = Y00 - Z00; u[1] = Y10 - Z10; u[2] = Y01 - Z01; u[3] = Y11 - Z11;
    u[4] = Z00; u[5] = Z10; u[6] = Z01; u[7] = Z11;
}

}  // namespace
}  // namespace ohpic
