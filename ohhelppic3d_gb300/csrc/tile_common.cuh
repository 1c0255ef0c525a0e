// tile_common.cuh -- device helpers shared by the tiled particle kernels
// (work items, the staged E/rho box, gathers, deposits, diagnostics).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "ohpic_internal.cuh"

namespace ohpic {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ void flag_error(DevDiag *d, int code, int info)
{
    if (atomicCAS(&d->err_code, 0, code) == 0) d->err_info = info;
}

// One E node, global to shared, asynchronously: the rows of a box are all in flight at
// once (read through registers, each row's loads were waited for before the next).
__device__ __forceinline__ void copy16(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_node(float4 *dst, const float4 *src) { copy16(dst, src); }
__device__ __forceinline__ void copy_node(dnode *dst, const dnode *src)
{
    copy16(dst, src);
    copy16((char *)dst + 16, (const char *)src + 16);
}
// This thread's copies have landed (the other threads' after the next barrier).
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// CIC weights of node floor(x) (w0) and floor(x)+1 (w1).  The reference
// convention (linear_scatter.f90:41-42, linear_interpolator.f90:54-57) gives
// node floor(x) the weight r = x - floor(x).
template <typename T>
__device__ __forceinline__ void cic(int conv, T r, T &w0, T &w1)
{
    if (conv == OHPIC_WEIGHTS_REFERENCE) {
        w0 = r;
        w1 = T(1) - r;
    } else {
        w0 = T(1) - r;
        w1 = r;
    }
}

// The same with the convention fixed at compile time (the FP32 kernels are
// instantiated per convention: a run-time choice cost two selects per axis).
template <int CONV, typename T>
__device__ __forceinline__ void cic_c(T r, T &w0, T &w1)
{
    if (CONV == OHPIC_WEIGHTS_REFERENCE) {
        w0 = r;
        w1 = T(1) - r;
    } else {
        w0 = T(1) - r;
        w1 = r;
    }
}

// i wrapped into [0, n) by steps of n: for indices at most a few n outside, where a
// division's latency would stall the warp.
__device__ __forceinline__ int wrap_near(int i, int n)
{
    while (i < 0) i += n;
    while (i >= n) i -= n;
    return i;
}

__device__ __forceinline__ int wrapi(int i, int n)
{
    i %= n;
    return i < 0 ? i + n : i;
}

// ---------------------------------------------------------------------------
// Work item of a CTA.
// ---------------------------------------------------------------------------
struct Item {
    int sp;
    int tile;           // -1 when unsorted
    int64_t g0, g1;     // vector-group range [g0, g1)
    int x0, y0, z0;     // tile origin (cells)
};

// Work item b of a launch (b = blockIdx.x for a single context; the multi-run
// kernel passes the item's index within its run).
template <int PPT>
__device__ __forceinline__ bool get_item(const TileArgs &a, int64_t b, Item &it)
{
    if (a.sorted) {
        // (a launch has fewer than 2^31 items)
        const unsigned split = (unsigned)a.split, per_sp = (unsigned)a.g.ntile * split, s = (unsigned)b / per_sp;
        it.sp = a.sp0 + (int)s;
        const unsigned r = (unsigned)b - s * per_sp, ti = split == 1u ? r : r / split;
        it.tile = (int)ti;
        const int part = (int)(r - ti * split);
        const int64_t *tb = a.tile_begin + (int64_t)it.sp * (a.g.ntile + 1);
        const int64_t lo = tb[it.tile] / PPT;
        const int64_t hi = it.tile + 1 == a.g.ntile ? (tb[a.g.ntile] + PPT - 1) / PPT : tb[it.tile + 1] / PPT;
        const int64_t n = hi - lo;
        it.g0 = split == 1u ? lo : lo + n * part / a.split;
        it.g1 = split == 1u ? hi : lo + n * (part + 1) / a.split;
        const unsigned row = ti / (unsigned)a.g.ntx, tz = row / (unsigned)a.g.nty;
        const int tx = (int)(ti - row * (unsigned)a.g.ntx), ty = (int)(row - tz * (unsigned)a.g.nty);
        it.x0 = tx * a.g.tx;
        it.y0 = ty * a.g.ty;
        it.z0 = (int)tz * a.g.tz;
    } else {
        // Unsorted: consecutive chunks of every species, no staging.
        int sp = a.sp0;
        int64_t first = 0;
        for (; sp < a.sp0 + a.nsp; ++sp) {
            const int64_t groups = (a.count[sp] + PPT - 1) / PPT;
            const int64_t blocks = (groups * PPT + a.chunk - 1) / a.chunk;
            if (b < first + blocks) break;
            first += blocks;
        }
        if (sp >= a.sp0 + a.nsp) return false;
        it.sp = sp;
        it.tile = -1;
        const int64_t gseg = a.seg[sp] / PPT;
        const int64_t groups = (a.count[sp] + PPT - 1) / PPT;
        const int64_t gpc = a.chunk / PPT;
        it.g0 = gseg + (b - first) * gpc;
        it.g1 = min(gseg + groups, it.g0 + gpc);
        it.x0 = it.y0 = it.z0 = 0;
    }
    return true;
}

template <int PPT>
__device__ __forceinline__ bool get_item(const TileArgs &a, Item &it)
{
    return get_item<PPT>(a, (int64_t)blockIdx.x, it);
}

// Rows of a box (fixed y, z; sx nodes along x) dealt to the CTA's warps, a row to each
// half of a warp when it fits 16 lanes.  The (y, z) of a lane's next row come by
// addition, and indices wrap by comparison: with a division and two remainders a row,
// the flush of a 13 x 13 x 13 box waited for them 22 times (FP32 push of 64^3 x 32 ppc
// 307 -> 291 us, 128x128x64 1041 -> 987 us, 16^3 x 8 ppc 16.7 -> 14.7 us).
struct RowWalk {
    int lane, step, width, by, cz;
    __device__ __forceinline__ RowWalk(int sx, int sy)
    {
        const int warp = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
        const bool two = sx <= 16;
        width = two ? 16 : 32;
        lane = l & (width - 1);
        step = two ? 2 * nw : nw;
        by = two ? 2 * warp + (l >> 4) : warp;
        cz = 0;
        settle(sy);
    }
    __device__ __forceinline__ void settle(int sy)
    {
        while (by >= sy) {
            by -= sy;
            ++cz;
        }
    }
    __device__ __forceinline__ void next(int sy)
    {
        by += step;
        settle(sy);
    }
};

// Staged box: nodes (x0-halo .. x0+tx+halo) per axis, i.e. the low corners of
// cells x0-halo .. x0+tx+halo-1 ("span" cells), so a cell with box coordinate
// l in [0, span) has both its nodes inside.
struct Box {
    int ox, oy, oz;          // box origin in cells (x0 - halo, ...)
    unsigned spx, spy, spz;  // valid low-corner span per axis
    int sx, sxy;             // node pitches
    bool on;                 // staged at all
    __device__ __forceinline__ int key(int ix, int iy, int iz) const
    {
        const int lx = ix - ox, ly = iy - oy, lz = iz - oz;
        const bool in = on && (unsigned)lx < spx && (unsigned)ly < spy && (unsigned)lz < spz;
        return in ? lx + sx * ly + sxy * lz : -1;
    }
};

__device__ __forceinline__ Box make_box(const Geom &g, const Item &it)
{
    Box b;
    b.ox = it.x0 - g.halo;
    b.oy = it.y0 - g.halo;
    b.oz = it.z0 - g.halo;
    b.spx = (unsigned)(g.tx + 2 * g.halo);
    b.spy = (unsigned)(g.ty + 2 * g.halo);
    b.spz = (unsigned)(g.tz + 2 * g.halo);
    b.sx = g.sx;
    b.sxy = g.sx * g.sy;
    b.on = it.tile >= 0;
    return b;
}

template <typename NodeT, typename T>
__device__ __forceinline__ void stage_tile(const TileArgs &a, const Item &it, NodeT *sE, T *srho, bool need_e,
                                           bool need_rho)
{
    const Geom &g = a.g;
    const int sx = g.sx, sy = g.sy, sz = g.sz, ex = min(sx, g.gx - it.x0);
    const NodeT *E = (const NodeT *)a.epad;
    if (need_e)
        for (RowWalk r(sx, sy); r.cz < sz; r.next(sy)) {
            // padded index of node (x0 - halo + ax) is x0 + ax; the box of a last tile
            // that is shorter than the others reaches past the array
            if (it.z0 + r.cz >= g.gz || it.y0 + r.by >= g.gy) continue;
            const NodeT *src = E + ((int64_t)(it.z0 + r.cz) * g.gy + (it.y0 + r.by)) * g.gx + it.x0;
            const int base = sx * (r.by + sy * r.cz);
            for (int ax = r.lane; ax < ex; ax += r.width) copy_node(sE + base + ax, src + ax);
        }
    if (need_rho)
        for (int i = threadIdx.x; i < sx * sy * sz; i += blockDim.x) srho[i] = T(0);
    copies_landed();
}

// Block-wide reduction of the per-thread diagnostics into DevDiag.  The counts
// reduce with integer warp reductions; the kinetic sums (in FP64, converted per
// thread) only when the push tracks them.  On GB300 an FP64 add runs on the narrow
// FP64 pipe, and reducing all eight tallies in FP64 at the end of every work item
// kept that pipe 4.5% busy in the FP32 push.
template <typename T>
__device__ void flush_diag(const TileArgs &a, int sp, unsigned cx, unsigned cy, unsigned cz, unsigned outside, T ke,
                           T px, T py, T pz)
{
    // The tile kernels run 256 threads (8 warps); the scratch is sized for exactly
    // that and keeps the static shared memory of a (16,8,8) tile at halo 2 within
    // two CTAs per SM.
    __shared__ unsigned cnt[4][kTileWarps];
    __shared__ double kin[4][kTileWarps];
    const bool energy = a.with_energy != 0;
    unsigned u[4] = {cx, cy, cz, outside};
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = __reduce_add_sync(kFull, u[k]);
    double v[4] = {(double)ke, (double)px, (double)py, (double)pz};
    if (energy) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(kFull, v[k], o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0 && warp < kTileWarps) {
        for (int k = 0; k < 4; ++k) {
            cnt[k][warp] = u[k];
            kin[k][warp] = v[k];
        }
    }
    __syncthreads();
    if (warp == 0) {
        const int nw = min((int)(blockDim.x >> 5), kTileWarps);
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = __reduce_add_sync(kFull, lane < nw ? cnt[k][lane] : 0u);
        if (energy) {
            for (int k = 0; k < 4; ++k) {
                double t = lane < nw ? kin[k][lane] : 0.0;
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
                v[k] = t;
            }
        }
        if (lane == 0) {
            DevDiag *d = a.diag;
            if (u[0]) atomicAdd(&d->crossings[0], (unsigned long long)u[0]);
            if (u[1]) atomicAdd(&d->crossings[1], (unsigned long long)u[1]);
            if (u[2]) atomicAdd(&d->crossings[2], (unsigned long long)u[2]);
            if (u[3]) atomicAdd(&d->outside, (unsigned long long)u[3]);
            if (energy) {
                atomicAdd(&d->kin[sp][0], v[0]);
                atomicAdd(&d->kin[sp][1], v[1]);
                atomicAdd(&d->kin[sp][2], v[2]);
                atomicAdd(&d->kin[sp][3], v[3]);
            }
        }
    }
}

// Sign and ">= n" tests of a double on its bit pattern (integer ALU, not the FP64
// pipe).  lt0 is p < 0 (false for -0.0); ge is p >= n for the bits of (double)n > 0.
__device__ __forceinline__ bool lt0(double p)
{
    const long long b = __double_as_longlong(p);
    return b < 0 && b != (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool ge_bits(double p, long long nbits) { return __double_as_longlong(p) >= nbits; }

// Strict FP64 arithmetic: every multiply and add rounds on its own, in the
// reference's operation order (no FMA contraction).
struct StrictOps {
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
};
struct FastOps {
    static __device__ __forceinline__ double mul(double a, double b) { return a * b; }
    static __device__ __forceinline__ double add(double a, double b) { return a + b; }
    static __device__ __forceinline__ double sub(double a, double b) { return a - b; }
};

}  // namespace
}  // namespace ohpic
