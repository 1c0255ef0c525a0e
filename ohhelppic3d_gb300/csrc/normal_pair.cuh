// normal_pair.cuh -- Box-Muller velocities of the FP32 form without FP64 operations.
//
// The injector's velocity of a particle is v = sigma sqrt(-2 log r1) cos(2 pi' r2) + drift
// (and with sin, and with r3, r4), computed in FP64 and rounded to a float.  The draws are
// 32-bit integers over 2^32, so everything up to the rounding can be had from integers and
// pairs of floats (an unevaluated sum hi + lo; Dekker 1971, Knuth's TAOCP vol. 2): log from
// a table of 128 reciprocals and the series of log(1 + u), sine and cosine from a table of
// 256 angles and the series of the rest.  The pair comes with a bound of its error; when
// both ends of that interval round to the same float, this is the float that the FP64
// computation gives, and otherwise (about 1 particle in 6000) the caller computes in FP64:
// the rounding test of Ziv (ACM TOMS 17, 1991).
#pragma once

#include <math.h>
#include <stdint.h>

namespace ohpic {

struct NormalTables {
    struct alignas(16) Log {
        unsigned inv;   // 1 / (the interval's centre) in units of 2^-10
        float hi, lo;   // log of it
        float pad;
    } log[128];
    struct alignas(16) Trig {
        float shi, slo, chi, clo;   // sin and cos of i / 256 of a turn
    } trig[256];
};

constexpr double series_log(double x)   // log by atanh((x - 1) / (x + 1)), 1 <= x <= 2
{
    const double t = (x - 1.0) / (x + 1.0), t2 = t * t;
    double s = 0.0;
    for (int k = 45; k >= 1; k -= 2) s = s * t2 + 1.0 / k;
    return 2.0 * t * s;
}

constexpr double series_sin(double x)   // Taylor, |x| <= pi / 4
{
    double s = 1.0;
    for (int k = 23; k >= 3; k -= 2) s = 1.0 - s * x * x / (double)(k * (k - 1));
    return x * s;
}

constexpr double series_cos(double x)
{
    double s = 1.0;
    for (int k = 24; k >= 2; k -= 2) s = 1.0 - s * x * x / (double)(k * (k - 1));
    return s;
}

constexpr NormalTables make_normal_tables()
{
    NormalTables t{};
    for (int i = 0; i < 128; ++i) {
        // the interval next to 1 keeps 1 itself: log(1 + u) is then exact relative to u
        const unsigned inv = i == 127 ? 1024u : (unsigned)(1024.0 * 512.0 / (257 + 2 * i) + 0.5);
        const double l = series_log(inv / 1024.0);
        t.log[i].inv = inv;
        t.log[i].hi = (float)l;
        t.log[i].lo = (float)(l - (double)(float)l);
    }
    constexpr double kTurn = 6.283185307179586476925286766559;
    for (int i = 0; i < 256; ++i) {
        const int quarter = (i + 32) / 64 & 3;             // nearest multiple of a quarter turn
        const double x = kTurn * (double)(i - 64 * ((i + 32) / 64)) / 256.0;
        const double s = series_sin(x), c = series_cos(x);
        const double sv = quarter == 0 ? s : quarter == 1 ? c : quarter == 2 ? -s : -c;
        const double cv = quarter == 0 ? c : quarter == 1 ? -s : quarter == 2 ? -c : s;
        t.trig[i].shi = (float)sv;
        t.trig[i].slo = (float)(sv - (double)(float)sv);
        t.trig[i].chi = (float)cv;
        t.trig[i].clo = (float)(cv - (double)(float)cv);
    }
    return t;
}

#if defined(__CUDA_ARCH__)
#define OHPIC_NP_FN __device__ __forceinline__
OHPIC_NP_FN float np_add(float a, float b) { return __fadd_rn(a, b); }
OHPIC_NP_FN float np_mul(float a, float b) { return __fmul_rn(a, b); }
OHPIC_NP_FN float np_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
OHPIC_NP_FN float np_rsqrt(float a) { return rsqrtf(a); }
OHPIC_NP_FN int np_clz(uint32_t a) { return __clz((int)a); }
#else
#define OHPIC_NP_FN inline
OHPIC_NP_FN float np_add(float a, float b) { return a + b; }
OHPIC_NP_FN float np_mul(float a, float b) { return a * b; }
OHPIC_NP_FN float np_fma(float a, float b, float c) { return fmaf(a, b, c); }
OHPIC_NP_FN float np_rsqrt(float a) { return 1.f / sqrtf(a); }
OHPIC_NP_FN int np_clz(uint32_t a) { return __builtin_clz(a); }
#endif

struct FloatPair {
    float hi, lo;
};

// a + b as a pair, exact for |a| >= |b| or a = 0.
OHPIC_NP_FN FloatPair fast_sum(float a, float b)
{
    const float s = np_add(a, b);
    return {s, np_add(b, -np_add(s, -a))};
}

OHPIC_NP_FN FloatPair two_sum(float a, float b)
{
    const float s = np_add(a, b), bb = np_add(s, -a);
    return {s, np_add(np_add(a, -np_add(s, -bb)), np_add(b, -bb))};
}

OHPIC_NP_FN FloatPair pair_mul(const FloatPair &a, const FloatPair &b)
{
    const float p = np_mul(a.hi, b.hi);
    return {p, np_add(np_fma(a.hi, b.hi, -p), np_fma(a.hi, b.lo, np_mul(a.lo, b.hi)))};
}

// sqrt(-2 log(k 2^-32)) for k > 0, to 2^-40 of itself.
OHPIC_NP_FN FloatPair radius(uint32_t k, const NormalTables::Log *table)
{
    const int lz = np_clz(k);
    const uint32_t m = k << lz;
    const NormalTables::Log t = table[m >> 24 & 127];
    // u = m / centre - 1, exact: |u| < 2^-7.8 in units of 2^-42
    const int64_t U = (int64_t)((uint64_t)m * t.inv) - (1ll << 42);
    const FloatPair u = fast_sum(np_mul((float)(int)(U >> 12), 0x1p-30f), np_mul((float)(int)(U & 4095), 0x1p-42f));
    // -log r = lz log 2 + log(1 / centre) - log(1 + u): no term cancels another
    constexpr float kLn2Hi = 0x1.62e4p-1f, kLn2Lo = 0x1.7f7d1cp-20f;   // hi: 15 bits, its multiples are exact
    const float flz = (float)lz, q = np_mul(u.hi, u.hi);
    const float qe = np_fma(u.hi, u.hi, -q) + 2.f * u.hi * u.lo;
    const FloatPair s1 = fast_sum(flz * kLn2Hi, t.hi), s2 = fast_sum(s1.hi, -u.hi), s3 = fast_sum(s2.hi, 0.5f * q);
    const float cubic = u.hi * q * (1.f / 3.f - u.hi * (0.25f - u.hi * (0.2f - u.hi * (1.f / 6.f))));
    const float lo = ((s1.lo + s2.lo + s3.lo) + (t.lo + flz * kLn2Lo)) + ((0.5f * qe - u.lo) - cubic);
    const FloatPair l = fast_sum(s3.hi, lo);
    // one Newton step from rsqrt of twice that
    const float th = 2.f * l.hi, rs = np_rsqrt(th), s = np_mul(th, rs);
    return {s, 0.5f * rs * np_add(np_fma(-s, s, th), 2.f * l.lo)};
}

// Sine and cosine of k 2^-32 turns, to 2^-42.4.
OHPIC_NP_FN void turn(uint32_t k, const NormalTables::Trig *table, FloatPair &sine, FloatPair &cosine)
{
    const uint32_t i = (k + 0x800000u) >> 24;
    const NormalTables::Trig t = table[i];
    const float j = (float)(int)(k - (i << 24));           // |j| <= 2^23
    constexpr float kTurnHi = 0x1.921fb6p-30f, kTurnLo = -0x1.777a5cp-55f;   // 2 pi 2^-32
    const float th = np_mul(j, kTurnHi), tl = np_fma(j, kTurnHi, -th) + j * kTurnLo;
    const float q = np_mul(th, th), qe = np_fma(th, th, -q) + 2.f * th * tl;
    const float sl = tl + th * q * (q * (1.f / 120.f) - 1.f / 6.f);     // sin = th + sl
    const float ch = -0.5f * q, cl = q * q * (1.f / 24.f) - 0.5f * qe;  // cos = 1 + ch + cl
    auto rotate = [&](float ahi, float alo, float bhi, float blo) {     // a cos + b sin
        const float p = np_mul(bhi, th), r = np_mul(ahi, ch);
        const FloatPair x = fast_sum(ahi, p), y = fast_sum(x.hi, r);
        const float lo = ((np_fma(bhi, th, -p) + np_fma(ahi, ch, -r)) + (bhi * sl + blo * th)) +
                         ((ahi * cl + alo * ch) + alo) + (x.lo + y.lo);
        return fast_sum(y.hi, lo);
    };
    sine = rotate(t.shi, t.slo, t.chi, t.clo);
    cosine = rotate(t.chi, t.clo, -t.shi, -t.slo);
}

// (sigma sqrt(-2 log) as a pair) x (sine or cosine) + drift, rounded to a float; false when
// the error bound leaves the rounding open or the magnitude is near the clip at 6 sigma.
// The bound: 1.5 2^-40 of the product for the pair's relative error, 2^-42 of the radius
// for the angle (its own rounding, pi' - pi and the FP64 rounding of 2 pi' r are below
// 2^-45 together), and 2^-45 of the drift for its sum.
OHPIC_NP_FN bool round_velocity(const FloatPair &radius, const FloatPair &b, const FloatPair &drift, float clip, float &v)
{
    const FloatPair p = pair_mul(radius, b);
    const float mag = fabsf(p.hi);
    const FloatPair s = two_sum(p.hi, drift.hi);
    const float lo = s.lo + (p.lo + drift.lo);
    const float err = mag * 0x1.8p-40f + radius.hi * 0x1p-42f + fabsf(drift.hi) * 0x1p-45f;
    v = np_add(s.hi, lo + err);
    return v == np_add(s.hi, lo - err) && mag < clip;
}

}  // namespace ohpic
