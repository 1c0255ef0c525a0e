// line_r2r.cuh -- FFTW's real-to-real transforms of pairs of real lines held in a CTA's
// shared memory as complex lines (one real line in each part).
//
// Every kind maps a real line to a real line and is linear, so one complex line
// carries two.  The complex FFTs are no longer than the line:
//   R2HC, HC2R  one FFT of the line's length; the pair's spectra are separated and
//               combined from elements k and L - k
//   DCT-II      reorder (even elements up, odd ones down), FFT of length L, then
//               Y_k = w^k V_k + conj(w^k) V_{L-k}, w = exp(-i pi / 2L)
//   DCT-III     V_k = conj(w^k) (X_k - i X_{L-k}), inverse FFT of length L, reorder back
//   DST-II/III  the same of the sign-alternated or reversed line
//   DCT-I(N), DST-I(N)  (N intervals) folded about the middle: the outputs of odd
//               index are a DCT-III (DST-III) of length N / 2 of the differences
//               (sums) X_j -+ X_{N-j}, those of even index the same transform
//               with N / 2 intervals of the others.  Folding stops at an odd or
//               small number of intervals, which take one FFT of the even (odd)
//               extension.  The FFTs of every fold run side by side.
// (Makhoul's reordering for the types II and III.)  Against the FFT of the doubled
// line that each kind took before, half as many FP64 operations, which bound
// these transforms on GB300 (two FP64 lanes per SM).
#pragma once
#include <algorithm>
#include <vector>

#include "line_fft.cuh"

namespace ohpic {
namespace {

enum Xform { XF_R2HC, XF_HC2R, XF_DCT1, XF_DST1, XF_DCT2, XF_DCT3, XF_DST2, XF_DST3 };

constexpr int kMaxFolds = 9;      // of up to 4096 intervals, down to kFoldEnd
constexpr int kFoldEnd = 16;
// A prime factor of R costs R operations an element: whole solves (periodic to mixed
// kinds of axis, us) against cuFFT's, and in brackets with 2 R operations, on which the
// line was drawn: 64x53x48 76-123 (98-166) against 250-342, 96x67x64 176-310 (233-423)
// against 263-587, 201x67x67 462-876 (853-1599) against 632-1727; above the line, with
// 2 R, 96x83x64 335-576 against 326-632, 96x101x64 410-746 against 376-745.
constexpr int kMaxPrime = 67;

struct SubFft {
    LinePlan pl;
    int off;           // first element in the line buffers
    int ts;            // table stride: exp(-2 pi i k / n) is entry k * ts
    int base;          // 1: of the extension table
};

// The transforms of one axis.
struct AxisXf {
    int L;             // points
    int N;             // intervals (types I)
    int folds;
    int nf;            // FFTs: one per fold, then the base one (types I), or the only one
    int maxst;
    SubFft f[kMaxFolds + 1];
    int E;             // elements a line buffer holds
    int n1, n2;        // entries of the FFT table and of the extension's own (0: shared)
    const double2 *T;  // FFT table (n1), then w^k (n1), then the extension's table (n2)
};

// The plan of an axis for its forward kind (the backward one uses the same); the
// table's host values are appended to t.  False when a length does not fit.
inline bool axis_plan(int xf, int L, AxisXf &a, std::vector<double> &t)
{
    a = AxisXf{};
    a.L = L;
    const bool type1 = xf == XF_DCT1 || xf == XF_DST1;
    a.N = xf == XF_DCT1 ? L - 1 : L + 1;
    int off = 0, nb = 0;
    if (type1) {
        int n = a.N;
        while (n % 2 == 0 && n > kFoldEnd && a.folds < kMaxFolds) {
            n /= 2;
            SubFft &f = a.f[a.nf++];
            if (!line_plan(n, f.pl, kMaxPrime)) return false;
            f.off = off;
            f.ts = 1 << a.folds;
            off += n;
            ++a.folds;
        }
        a.n1 = a.folds ? a.N / 2 : 0;
        nb = 2 * n;
        SubFft &f = a.f[a.nf++];
        if (!line_plan(nb, f.pl, kMaxPrime)) return false;
        f.off = off;
        f.base = 1;
        off += nb;
        if (a.n1 && a.n1 % nb == 0) {
            f.base = 0;
            f.ts = a.n1 / nb;
        } else {
            f.ts = 1;
            a.n2 = nb;
        }
    } else {
        a.n1 = L;
        a.f[0].ts = 1;
        if (!line_plan(L, a.f[0].pl, kMaxPrime)) return false;
        a.nf = 1;
        off = L;
    }
    for (int i = 0; i < a.nf; ++i) a.maxst = std::max(a.maxst, a.f[i].pl.nst);
    a.E = std::max(off, type1 ? a.N + 1 : L);
    if (a.n1) {
        line_twiddles(a.n1, t);
        // w^k = exp(-i pi k / (2 n1)) is entry k of the table of 4 n1
        std::vector<double> q;
        line_twiddles(4 * a.n1, q);
        t.insert(t.end(), q.begin(), q.begin() + 2 * (size_t)a.n1);
    }
    if (a.n2) line_twiddles(a.n2, t);
    return true;
}

// P complex lines, element e of line l at e * (P + 1) + l of buffers A and B; Tw
// points at the axis' table.  At most kPerThread elements per thread and buffer.
constexpr int kPerThread = 8;

struct LineCtx {
    double2 *A, *B;
    const double2 *Tw;
    int P, Pshift;
};

__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }

// Element k of a fold's (or the only) DCT-III input: conj(w^k) (x_k - i x_{n-k}), parts
// exchanged for the inverse transform; x_n = 0.
__device__ __forceinline__ double2 dct3_in(double2 x, double2 y, double2 w)
{
    return swap_parts(cmul(conj2(w), make_double2(x.x + y.y, x.y - y.x)));
}

// Transform xf of the lines in A (elements 0 .. L - 1), back into A.  All threads.
__device__ __forceinline__ void line_r2r(const AxisXf &a, int xf, const LineCtx &c)
{
    const int S = c.P + 1, P = c.P, sh = c.Pshift, L = a.L;
    double2 *A = c.A, *B = c.B;
    const double2 *W = c.Tw + a.n1;
    const bool type1 = xf == XF_DCT1 || xf == XF_DST1;
    if (type1) {
        // X_j at element j - o: DST-I has no X_0
        const int o = xf == XF_DST1 ? 1 : 0;
        int n = a.N;
        for (int l = 0; l < a.folds; ++l, n /= 2) {
            // j and n - j: the outputs of even index stay at j, those of odd index go to n - j
            const int j0 = o, cnt = (n / 2 + 1 - j0) * P;
            for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
                const int j = j0 + (t >> sh), line = t & (P - 1);
                double2 *p = A + (j - o) * S + line, *q = A + (n - j - o) * S + line;
                const double2 x = *p, y = *q;
                if (2 * j == n) {
                    *p = make_double2(x.x + x.x, x.y + x.y);
                } else {
                    const double2 s = cadd(x, y), d = csub(x, y);
                    *p = o ? d : s;
                    *q = o ? s : d;
                }
            }
            __syncthreads();
        }
        // inputs of every FFT
        n = a.N;
        for (int l = 0; l < a.folds; ++l, n /= 2) {
            const int h = n / 2, st = 1 << l;
            double2 *dst = B + a.f[l].off * S;
            for (int t = threadIdx.x; t < h * P; t += blockDim.x) {
                const int k = t >> sh, line = t & (P - 1);
                // DCT-I: difference k at n - k; DST-I: the reversed sums, element k at h + k
                const double2 x = A[((o ? h + k : n - k) - o) * S + line];
                double2 y = make_double2(0.0, 0.0);
                if (k) y = A[((o ? n - k : h + k) - o) * S + line];
                dst[k * S + line] = dct3_in(x, y, W[k * st]);
            }
        }
        double2 *dst = B + a.f[a.folds].off * S;
        for (int t = threadIdx.x; t < 2 * n * P; t += blockDim.x) {
            const int m = t >> sh, line = t & (P - 1);
            const int j = m <= n ? m : 2 * n - m;
            double2 v = make_double2(0.0, 0.0);
            if (!o || (j > 0 && j < n)) v = A[(j - o) * S + line];
            if (o && m > n) v = make_double2(-v.x, -v.y);
            dst[m * S + line] = v;
        }
    } else {
        for (int t = threadIdx.x; t < L * P; t += blockDim.x) {
            const int m = t >> sh, line = t & (P - 1);
            const double2 *x = A + line;
            double2 v;
            if (xf == XF_R2HC) {
                v = x[m * S];
            } else if (xf == XF_HC2R) {
                // G_k = F_A,k + i F_B,k from the half-complex pairs at k and L - k
                const int kk = m == 0 ? 0 : L - m;
                const double2 p = x[m * S], q = x[kk * S];
                v = kk == m  ? p
                    : m < kk ? make_double2(p.x - q.y, q.x + p.y)
                             : make_double2(q.x + p.y, q.y - p.x);
                v = swap_parts(v);
            } else if (xf == XF_DCT2 || xf == XF_DST2) {
                const int j = 2 * m < L ? 2 * m : 2 * (L - 1 - m) + 1;
                v = x[j * S];
                if (xf == XF_DST2 && (j & 1)) v = make_double2(-v.x, -v.y);
            } else {
                const bool rev = xf == XF_DST3;
                double2 y = make_double2(0.0, 0.0);
                if (m) y = x[(rev ? m - 1 : L - m) * S];
                v = dct3_in(x[(rev ? L - 1 - m : m) * S], y, W[m]);
            }
            B[m * S + line] = v;
        }
    }
    __syncthreads();
    const FastDiv dP{(unsigned)P, sh ? 1u << (32 - sh) : 0u};
    for (int s = 0; s < a.maxst; ++s) {
        for (int i = 0; i < a.nf; ++i) {
            const SubFft &f = a.f[i];
            if (s < f.pl.nst)
                line_fft_stage(f.pl, s, (s & 1 ? A : B) + f.off * S, (s & 1 ? B : A) + f.off * S, (unsigned)P, dP, S, 1,
                               c.Tw + (f.base ? 2 * a.n1 : 0), f.ts);
        }
        __syncthreads();
    }
    double2 r[kPerThread];
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
        const int t = threadIdx.x + u * blockDim.x;
        if (t >= L * P) break;
        const int k = t >> sh, line = t & (P - 1);
        if (type1) {
            const int K = k + (xf == XF_DST1 ? 1 : 0);      // output index
            const int l = K ? min(__ffs(K) - 1, a.folds) : a.folds;
            const SubFft &f = a.f[l];
            const double2 *Z = (f.pl.nst & 1 ? A : B) + f.off * S + line;
            if (l == a.folds) {
                const double2 z = Z[(K >> l) * S];
                r[u] = xf == XF_DST1 ? make_double2(-z.y, z.x) : z;
            } else {
                const int n = f.pl.n, m = K >> (l + 1);
                const double2 z = swap_parts(Z[(m & 1 ? n - 1 - m / 2 : m / 2) * S]);
                r[u] = xf == XF_DST1 && (m & 1) ? make_double2(-z.x, -z.y) : z;
            }
            continue;
        }
        const double2 *Z = (a.f[0].pl.nst & 1 ? A : B) + line;
        if (xf == XF_R2HC) {
            // the pair's spectra at k and L - k, stored half-complex
            const int kk = k == 0 ? 0 : L - k;
            const double2 z = Z[k * S], w = Z[kk * S];
            r[u] = k <= kk ? make_double2(0.5 * (z.x + w.x), 0.5 * (z.y + w.y))
                           : make_double2(0.5 * (w.y - z.y), 0.5 * (z.x - w.x));
        } else if (xf == XF_HC2R) {
            r[u] = swap_parts(Z[k * S]);
        } else if (xf == XF_DCT2 || xf == XF_DST2) {
            const int q = xf == XF_DST2 ? L - 1 - k : k;
            const double2 w = W[q];
            r[u] = cadd(cmul(w, Z[q * S]), cmul(conj2(w), Z[(q ? L - q : 0) * S]));
        } else {
            const double2 z = swap_parts(Z[(k & 1 ? L - 1 - k / 2 : k / 2) * S]);
            r[u] = xf == XF_DST3 && (k & 1) ? make_double2(-z.x, -z.y) : z;
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
        const int t = threadIdx.x + u * blockDim.x;
        if (t < L * P) A[(t >> sh) * S + (t & (P - 1))] = r[u];
    }
    __syncthreads();
}

}  // namespace
}  // namespace ohpic
