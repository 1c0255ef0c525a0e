// field_nodes.cuh -- one node of rho from the fixed-point weight sums, shared by the
// field kernels (fields.cu, spectral.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ohpic_internal.cuh"

namespace ohpic {
namespace {

// ---- FP32 form: rho from the fixed-point weight sums ----
//
// rho = sum_s q_s * W_s * 2^-24 (W_s the species' integer weight sum at the
// node), rounded once to FP32.  Each charge is an integer mantissa times a power
// of two (from its bit pattern), so the sum is formed exactly in 128-bit integer
// arithmetic and rounded to nearest, ties to even: no FP64 arithmetic per node.
// Bounds: |m_s| < 2^53, W_s < 2^58 (every count is far below 2^34), the exponent
// spread at most kRhoMaxShift, at most 8 species: the sum stays below 2^126.
// Charges further apart in exponent (or subnormal), and sums outside the normal
// FP32 range, take the FP64 expression instead.
constexpr int kRhoMaxShift = 12;

struct RhoScale {
    long long m[OHPIC_MAX_SPECIES];
    int shift[OHPIC_MAX_SPECIES];
    int K;
    bool ok;
    // Short form, when wbits > 0 and every W_s < 2^wbits: rho = (sum_s f_s W_s) * unit with a
    // 64-bit sum and an exact power of two, so the conversion of the sum is the
    // only rounding (the same one).
    int wbits;
    float unit;
    long long f[OHPIC_MAX_SPECIES];
};

__host__ __device__ inline RhoScale rho_scale(const double *q, int nsp)
{
    RhoScale r;
    r.ok = true;
    r.K = 0x7fffffff;
    int k[OHPIC_MAX_SPECIES];
    for (int s = 0; s < nsp; ++s) {
        union {
            double d;
            unsigned long long u;
        } bits;
        bits.d = q[s];
        const unsigned long long b = bits.u;
        const int e = (int)((b >> 52) & 0x7ffu);
        const long long mant = (long long)(b & ((1ull << 52) - 1));
        r.m[s] = 0;
        k[s] = 0;
        if (e == 0) {
            if (mant != 0) r.ok = false;   // subnormal charge
            continue;
        }
        if (e == 0x7ff) {
            r.ok = false;
            continue;
        }
        const long long m = mant | (1ll << 52);
        r.m[s] = (b >> 63) ? -m : m;
        k[s] = e - 1075 - 24;              // q_s * 2^-24 = m * 2^k
        if (k[s] < r.K) r.K = k[s];
    }
    for (int s = 0; s < nsp; ++s) {
        r.shift[s] = r.m[s] != 0 ? k[s] - r.K : 0;
        if (r.shift[s] > kRhoMaxShift) r.ok = false;
    }
    if (r.K == 0x7fffffff) r.K = 0;        // every charge zero: the sum is 0
    // Short charges (wp^2 / qm / ppc with a power of two per cell has one bit): without
    // their common trailing zeros the products fit 64 bits.
    r.wbits = 0;
    if (r.ok) {
        int tz = 63, top = 0, sp = 0;
        for (int s = 0; s < nsp; ++s) {
            if (r.m[s] == 0) continue;
            const long long v = r.m[s] < 0 ? -r.m[s] : r.m[s];
            int z = 0, n = 0;
            while (!((v >> z) & 1)) ++z;
            while (n < 63 && (v >> n)) ++n;
            if (z + r.shift[s] < tz) tz = z + r.shift[s];
            if (n + r.shift[s] > top) top = n + r.shift[s];
        }
        while ((1 << sp) < nsp) ++sp;
        const int bits = top > tz ? top - tz : 1, K = r.K + tz;
        if (bits <= 20 && K >= -126 && K <= 64) {
            r.wbits = 62 - bits - sp;
            union {
                unsigned u;
                float f;
            } two;
            two.u = (unsigned)(K + 127) << 23;
            r.unit = two.f;
            for (int s = 0; s < nsp; ++s)   // shift - tz may be negative: m has those zeros
                r.f[s] = r.shift[s] >= tz ? r.m[s] << (r.shift[s] - tz) : r.m[s] / (1ll << (tz - r.shift[s]));
        }
    }
    return r;
}

// acc * 2^K rounded to FP32, nearest with ties to even; false outside the
// normal range.
__device__ __forceinline__ bool i128_to_float_rne(__int128 acc, int K, float &out)
{
    if (acc == 0) {
        out = 0.f;
        return true;
    }
    const bool neg = acc < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)(-acc) : (unsigned __int128)acc;
    const unsigned long long hi = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
    int msb = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)lo);
    unsigned int mant;
    if (msb <= 23) {
        mant = (unsigned int)(lo << (23 - msb));
    } else {
        const int sh = msb - 23;
        const unsigned __int128 one = 1;
        const unsigned __int128 rem = a & ((one << sh) - 1);
        const unsigned __int128 half = one << (sh - 1);
        mant = (unsigned int)(a >> sh);
        if (rem > half || (rem == half && (mant & 1u))) {
            ++mant;
            if (mant == (1u << 24)) {
                mant >>= 1;
                ++msb;
            }
        }
    }
    const int be = msb + K + 127;
    if (be < 1 || be > 254) return false;
    out = __uint_as_float((neg ? 0x80000000u : 0u) | ((unsigned)be << 23) | (mant & 0x7fffffu));
    return true;
}

// rho at one node: w[s * stride] is species s's weight sum.
__device__ __forceinline__ float node_rho(const unsigned long long *w, int64_t stride, int nsp, const double *q,
                                          const RhoScale &r)
{
    if (r.wbits > 0) {
        unsigned long long any = 0;
        long long acc = 0;
        for (int s = 0; s < nsp; ++s) {
            const unsigned long long W = w[s * stride];
            any |= W;
            acc += r.f[s] * (long long)W;
        }
        if (any >> r.wbits == 0) return __ll2float_rn(acc) * r.unit;
    }
    if (r.ok) {
        __int128 acc = 0;
        for (int s = 0; s < nsp; ++s) {
            const long long m = r.m[s];
            if (m == 0) continue;
            // |m| * W as one 64 x 64 -> 128-bit product, then the species' shift
            const unsigned long long W = w[s * stride];
            const unsigned long long am = (unsigned long long)(m < 0 ? -m : m);
            unsigned __int128 p = ((unsigned __int128)__umul64hi(am, W) << 64) | (unsigned __int128)(am * W);
            p <<= r.shift[s];
            acc = m < 0 ? acc - (__int128)p : acc + (__int128)p;
        }
        float v;
        if (i128_to_float_rne(acc, r.K, v)) return v;
    }
    double acc = 0.0;
    for (int s = 0; s < nsp; ++s) acc += q[s] * (double)w[s * stride];
    return (float)(acc * kWeightUnit);
}

// node_rho of one or two species whose weight sums are already in registers (W[1] = 0
// for one).  The short form took the kernel's 128-bit products and their rounding, about
// 400 instructions a node, out of the usual case (k_wsum_to_rho at 256^3 105 -> 93 us,
// 6.5 TB/s with the clear).
__device__ __forceinline__ float node_rho2(const unsigned long long W[2], int nsp, const double *q, const RhoScale &r)
{
    if (r.wbits > 0 && (W[0] | W[1]) >> r.wbits == 0) {
        long long acc = r.f[0] * (long long)W[0];
        if (nsp > 1) acc += r.f[1] * (long long)W[1];
        return __ll2float_rn(acc) * r.unit;
    }
    if (r.ok) {
        __int128 acc = 0;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const long long m = s < nsp ? r.m[s] : 0;
            if (m == 0) continue;
            const unsigned long long am = (unsigned long long)(m < 0 ? -m : m);
            unsigned __int128 p = ((unsigned __int128)__umul64hi(am, W[s]) << 64) | (unsigned __int128)(am * W[s]);
            p <<= r.shift[s];
            acc = m < 0 ? acc - (__int128)p : acc + (__int128)p;
        }
        float v;
        if (i128_to_float_rne(acc, r.K, v)) return v;
    }
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s)
        if (s < nsp) acc += q[s] * (double)W[s];
    return (float)(acc * kWeightUnit);
}

__device__ __forceinline__ int wrapn(int i, int n)
{
    i %= n;
    return i < 0 ? i + n : i;
}

}  // namespace
}  // namespace ohpic
