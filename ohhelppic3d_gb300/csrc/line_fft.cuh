// line_fft.cuh -- complex FFTs of many equal lines held in a CTA's shared memory.
//
// A Stockham (self-sorting) mixed-radix transform between two shared buffers.  At
// a stage of radix R, with L the product of the radices before it and m = n / R,
// butterfly p of a line (0 <= p < m, k = p mod L) takes the elements p + i m,
// multiplies element i by exp(-2 pi i k i / (L R)), transforms the R of them and
// writes them at (p - k) R + k + i L.  Consecutive threads take consecutive
// lines, so a line's butterflies share their twiddles (a broadcast) and shared
// accesses run across lines.  Radices 2 to 5, 7, 8, 11 and 13 keep a
// butterfly in registers; a larger prime takes one thread per
// output or two.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cmath>
#include <vector>

namespace ohpic {
namespace {

constexpr int kMaxStages = 10;

// x / d for 0 <= x, d < 2^16 with one high multiply.
struct FastDiv {
    unsigned d, m;   // m = ceil(2^32 / d); 0 stands for d = 1
};
inline FastDiv fast_div(unsigned d)
{
    return FastDiv{d, d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d)};
}
__device__ __forceinline__ unsigned div_by(FastDiv f, unsigned x) { return f.m ? __umulhi(x, f.m) : x; }

// The stages of a length-n transform.
struct LinePlan {
    int n, nst;
    int r[kMaxStages];
    FastDiv L[kMaxStages];
};

// False when n has a prime factor above max_prime (at most 67) or does not fit the
// index arithmetic.
inline bool line_plan(int n, LinePlan &p, int max_prime = 31)
{
    p.n = n;
    p.nst = 0;
    if (n < 1 || n > 4096) return false;
    int left = n, L = 1;
    auto take = [&](int r) {
        p.r[p.nst] = r;
        p.L[p.nst] = fast_div((unsigned)L);
        ++p.nst;
        L *= r;
        left /= r;
    };
    for (int q : {67, 61, 59, 53, 47, 43, 41, 37, 31, 29, 23, 19, 17})
        if (q <= max_prime && left % q == 0) {   // a large prime first, where it has no twiddles
            take(q);
            break;
        }
    while (left > 1) {
        if (p.nst == kMaxStages) return false;
        int r = 0;
        if (left == 16) r = 4;             // 4 x 4, not 8 x 2
        else if (left % 8 == 0) r = 8;
        else if (left % 4 == 0) r = 4;
        else
            for (int q : {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67})
                if (q <= max_prime && left % q == 0) {
                    r = q;
                    break;
                }
        if (!r) return false;
        take(r);
    }
    return true;
}

// Appends exp(-2 pi i k / n), k = 0 .. n - 1, as (re, im): the angle is folded into
// the first eighth of the circle, so symmetric entries are exactly symmetric.
inline void line_twiddles(int n, std::vector<double> &t)
{
    const double pi = 3.141592653589793238462643383;
    for (int k = 0; k < n; ++k) {
        const bool conj = 2 * k > n;
        const int m = conj ? n - k : k;                // the angle 2 pi m / n, m <= n / 2
        const bool back = 4 * m > n;                   // second quarter
        const double u = back ? n - 2 * m : 2 * m;     // pi u / n, u <= n / 2
        const bool far = 2 * u > 0.5 * n;              // beyond pi / 4
        const double v = far ? pi * (0.5 * n - u) / n : pi * u / n;
        const double c = far ? std::sin(v) : std::cos(v), s = far ? std::cos(v) : std::sin(v);
        t.push_back(back ? -c : c);
        t.push_back(conj ? s : -s);
    }
}

template <typename V>
__device__ __forceinline__ V cadd(V a, V b)
{
    a.x += b.x;
    a.y += b.y;
    return a;
}
template <typename V>
__device__ __forceinline__ V csub(V a, V b)
{
    a.x -= b.x;
    a.y -= b.y;
    return a;
}
template <typename V>
__device__ __forceinline__ V cmul(V a, V b)
{
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <typename V>
__device__ __forceinline__ V swap_parts(V a)
{
    V r;
    r.x = a.y;
    r.y = a.x;
    return r;
}
// -i a
template <typename V>
__device__ __forceinline__ V cmuli(V a)
{
    V r;
    r.x = a.y;
    r.y = -a.x;
    return r;
}

template <typename V>
__device__ __forceinline__ void dft2(V &a, V &b)
{
    const V t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

template <typename V>
__device__ __forceinline__ void dft4(V &a, V &b, V &c, V &d)
{
    const V s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = cmuli(csub(b, d));
    a = cadd(s, u);
    b = cadd(t, v);
    c = csub(s, u);
    d = csub(t, v);
}

// cos and sin of 2 pi q / R for the odd radices, 0 <= q <= (R - 1) / 2 (folded at
// compile time).
template <int R>
__device__ __forceinline__ constexpr double odd_cos(int q)
{
    if (R == 3)
        return q == 0 ? 1.0 : -0.500000000000000000000;
    if (R == 5)
        return q == 0 ? 1.0 : q == 1 ? 0.309016994374947424102 : 
               -0.809016994374947424102;
    if (R == 7)
        return q == 0 ? 1.0 : q == 1 ? 0.623489801858733530525 : 
               q == 2 ? -0.222520933956314404289 : -0.900968867902419126236;
    if (R == 11)
        return q == 0 ? 1.0 : q == 1 ? 0.841253532831181168862 : 
               q == 2 ? 0.415415013001886425529 : q == 3 ? -0.142314838273285140444 : 
               q == 4 ? -0.654860733945285064057 : -0.959492973614497389890;
    if (R == 13)
        return q == 0 ? 1.0 : q == 1 ? 0.885456025653209895900 : 
               q == 2 ? 0.568064746731155802512 : q == 3 ? 0.120536680255323053349 : 
               q == 4 ? -0.354604887042535625970 : q == 5 ? -0.748510748171101098635 : 
               -0.970941817426052027157;
    return 0.0;
}
template <int R>
__device__ __forceinline__ constexpr double odd_sin(int q)
{
    if (R == 3)
        return q == 0 ? 0.0 : 0.866025403784438646764;
    if (R == 5)
        return q == 0 ? 0.0 : q == 1 ? 0.951056516295153572116 : 
               0.587785252292473129169;
    if (R == 7)
        return q == 0 ? 0.0 : q == 1 ? 0.781831482468029808708 : 
               q == 2 ? 0.974927912181823607018 : 0.433883739117558120476;
    if (R == 11)
        return q == 0 ? 0.0 : q == 1 ? 0.540640817455597582108 : 
               q == 2 ? 0.909631995354518371412 : q == 3 ? 0.989821441880932732376 : 
               q == 4 ? 0.755749574354258283774 : 0.281732556841429697711;
    if (R == 13)
        return q == 0 ? 0.0 : q == 1 ? 0.464723172043768545656 : 
               q == 2 ? 0.822983865893656394580 : q == 3 ? 0.992708874098053992801 : 
               q == 4 ? 0.935016242685414823440 : q == 5 ? 0.663122658240795202377 : 
               0.239315664287557767149;
    return 0.0;
}

// Odd R from the sums and differences of the elements k and R - k.
template <int R, typename V>
__device__ __forceinline__ void dft_odd(V v[R])
{
    using T = decltype(V::x);
    constexpr int H = (R - 1) / 2;
    V a[H + 1], b[H + 1];
    V sum = v[0];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        a[k] = cadd(v[k], v[R - k]);
        b[k] = csub(v[k], v[R - k]);
        sum = cadd(sum, a[k]);
    }
    const V v0 = v[0];
    v[0] = sum;
#pragma unroll
    for (int j = 1; j <= H; ++j) {
        V e = v0, o;
        o.x = T(0);
        o.y = T(0);
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            const int q = (j * k) % R;
            const T c = (T)odd_cos<R>(q <= H ? q : R - q);
            const T s = q <= H ? (T)odd_sin<R>(q) : -(T)odd_sin<R>(R - q);
            e.x += c * a[k].x;
            e.y += c * a[k].y;
            o.x += s * b[k].x;
            o.y += s * b[k].y;
        }
        const V m = cmuli(o);   // -i o
        v[j] = cadd(e, m);
        v[R - j] = csub(e, m);
    }
}

template <int R, typename V>
__device__ __forceinline__ void dft(V v[R])
{
    using T = decltype(V::x);
    if constexpr (R == 2) {
        dft2(v[0], v[1]);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        // even and odd halves of four, the odd ones turned by the eighth roots
        dft4(v[0], v[2], v[4], v[6]);
        dft4(v[1], v[3], v[5], v[7]);
        const T h = (T)0.70710678118654752440;
        V w1, w3;
        w1.x = h * (v[3].x + v[3].y);
        w1.y = h * (v[3].y - v[3].x);
        const V w2 = cmuli(v[5]);
        w3.x = h * (v[7].y - v[7].x);
        w3.y = -h * (v[7].x + v[7].y);
        const V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = cadd(e0, o0);
        v[4] = csub(e0, o0);
        v[1] = cadd(e1, w1);
        v[5] = csub(e1, w1);
        v[2] = cadd(e2, w2);
        v[6] = csub(e2, w2);
        v[3] = cadd(e3, w3);
        v[7] = csub(e3, w3);
    } else {
        dft_odd<R>(v);
    }
}

// One stage over every line: element e of line l sits at l * ls + e * es.  tw is a
// table of n * ts roots, so exp(-2 pi i k / n) is its entry k * ts.
template <int R, typename V>
__device__ __forceinline__ void line_stage(const V *in, V *out, unsigned lines, FastDiv dl, int n, int es, int ls,
                                           FastDiv dL, const V *tw, int ts)
{
    const int L = (int)dL.d, m = n / R, step = n / (L * R) * ts;
    for (unsigned t = threadIdx.x; t < lines * (unsigned)m; t += blockDim.x) {
        const int p = (int)div_by(dl, t), line = (int)t - p * (int)lines;
        const int q = (int)div_by(dL, (unsigned)p), k = p - q * L;
        const V *src = in + line * ls;
        V v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = src[(p + i * m) * es];
        if (L > 1) {
#pragma unroll
            for (int i = 1; i < R; ++i) v[i] = cmul(v[i], tw[k * i * step]);
        }
        dft<R>(v);
        V *dst = out + line * ls + (q * L * R + k) * es;
#pragma unroll
        for (int i = 0; i < R; ++i) dst[i * L * es] = v[i];
    }
}

// A larger prime radix: one thread per output, a running twiddle index.
template <typename V>
__device__ __forceinline__ void line_stage_prime(int R, const V *in, V *out, unsigned lines, FastDiv dl, int n, int es,
                                                 int ls, FastDiv dL, const V *tw, int ts)
{
    const int L = (int)dL.d, m = n / R, step = n / (L * R);
    for (unsigned t = threadIdx.x; t < lines * (unsigned)n; t += blockDim.x) {
        const int o = (int)div_by(dl, t), line = (int)t - o * (int)lines;
        const int i = o / m, p = o - i * m;            // output i of butterfly p
        const int q = (int)div_by(dL, (unsigned)p), k = p - q * L;
        const int inc = (k * step + i * m) % n;         // m = n / R
        const V *src = in + line * ls + p * es;
        V acc = src[0];
        int w = 0;
        for (int s = 1; s < R; ++s) {
            w += inc;
            if (w >= n) w -= n;
            acc = cadd(acc, cmul(src[s * m * es], tw[w * ts]));
        }
        out[line * ls + (q * L * R + k + i * L) * es] = acc;
    }
}

// A larger prime radix as the first stage (no twiddles): one thread per outputs i and
// R - i, from the sums and differences of the elements s and R - s, which are formed
// first, in their place: formed anew for every output, they were half of the stage's
// FP64 operations, which bound it (bounded solve of 201 x 67 x 67, periodic: 853 -> 462 us).
// All threads of the CTA call it.
template <typename V>
__device__ __forceinline__ void line_first_prime(int R, V *in, V *out, unsigned lines, FastDiv dl, int n, int es,
                                                 int ls, const V *tw, int ts)
{
    const int m = n / R, H = (R - 1) / 2;
    for (unsigned t = threadIdx.x; t < lines * (unsigned)(m * H); t += blockDim.x) {
        const int o = (int)div_by(dl, t), line = (int)t - o * (int)lines;
        const int s = o / m + 1, p = o - (s - 1) * m;
        V *u = in + line * ls + (p + s * m) * es, *v = in + line * ls + (p + (R - s) * m) * es;
        const V a = *u, b = *v;
        *u = cadd(a, b);
        *v = csub(a, b);
    }
    __syncthreads();
    for (unsigned t = threadIdx.x; t < lines * (unsigned)(m * (H + 1)); t += blockDim.x) {
        const int o = (int)div_by(dl, t), line = (int)t - o * (int)lines;
        const int i = o / m, p = o - i * m;
        const V *src = in + line * ls + p * es;
        V e = src[0], d;
        d.x = d.y = 0;
        int w = 0;
        for (int s = 1; s <= H; ++s) {
            w += i;
            if (w >= R) w -= R;
            const V c = tw[w * m * ts], a = src[s * m * es], b = src[(R - s) * m * es];
            e.x += c.x * a.x;
            e.y += c.x * a.y;
            d.x -= c.y * b.x;      // c.y = -sin
            d.y -= c.y * b.y;
        }
        V *dst = out + line * ls + p * R * es;
        const V q = cmuli(d);
        dst[i * es] = cadd(e, q);
        if (i) dst[(R - i) * es] = csub(e, q);
    }
}

// Stage s of a plan from in (which a first stage may overwrite) to out (the caller
// synchronises).
template <typename V>
__device__ __forceinline__ void line_fft_stage(const LinePlan &pl, int s, V *in, V *out, unsigned lines,
                                               FastDiv dl, int es, int ls, const V *tw, int ts)
{
    const int R = pl.r[s];
    const FastDiv dL = pl.L[s];
    switch (R) {
    case 2: line_stage<2>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 3: line_stage<3>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 4: line_stage<4>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 5: line_stage<5>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 7: line_stage<7>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 11: line_stage<11>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 13: line_stage<13>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    case 8: line_stage<8>(in, out, lines, dl, pl.n, es, ls, dL, tw, ts); break;
    default:
        if (s == 0) line_first_prime(R, in, out, lines, dl, pl.n, es, ls, tw, ts);
        else line_stage_prime(R, in, out, lines, dl, pl.n, es, ls, dL, tw, ts);
        break;
    }
}

// The transform of every line from a (scratch b, or the other way round); returns
// the buffer that holds the result.  All threads of the CTA call it; the caller
// has synchronised after filling a, and the result is synchronised on return.
template <typename V>
__device__ __forceinline__ V *line_fft(const LinePlan &pl, V *a, V *b, unsigned lines, FastDiv dl, int es, int ls,
                                       const V *tw)
{
    for (int s = 0; s < pl.nst; ++s) {
        line_fft_stage(pl, s, a, b, lines, dl, es, ls, tw, 1);
        __syncthreads();
        V *t = a;
        a = b;
        b = t;
    }
    return a;
}

}  // namespace
}  // namespace ohpic
