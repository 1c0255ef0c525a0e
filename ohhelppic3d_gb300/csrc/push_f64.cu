// push_f64.cu -- the plain FP64 form of the tiled particle kernels.
//
//
// Reference path (per particle, src/ohhelppic3d.f90:311-358):
//   scatter   src/scatter/linear_scatter.f90:32-53
//   interp    src/interpolator/linear_interpolator.f90:33-67
//   move      src/particle_mover/particle_mover_boris.f90:37-62
//   boundary  src/particle_boundary/periodic_particle_boundary.f90:42-53 (twice)
//
// Work decomposition.  Particles of each species are kept sorted by tile-major
// cell index (sort.cu), so the particles of one tile are one contiguous range.
// One CTA takes (species, tile, part): it stages the tile's node E field plus a
// halo of `halo` cells into shared memory, zeroes a shared rho box of the same
// extent, streams its particles, one per thread and iteration, and flushes the box
// to global memory once.  A particle whose cell lies outside the staged box (it
// drifted since the last sort, or wrapped across the periodic edge) gathers
// from and deposits to global memory instead.
//
// Deposit in fixed point.  Each particle's 8 CIC weights are integers in units
// of 2^-48 that sum to exactly 2^48: the fractional offsets are rounded to 48
// bits, and 2^48 is split axis by axis (x, then y within each half, then z
// within each quarter), each child rounded from the product of its parent and
// the axis weight and its sibling taking the difference.  The products are
// 48 x 48 -> 96-bit integer multiplies, so the weights cost no FP64 operations
// beyond the offsets; on GB300 the FP64 pipe is the bottleneck of this form.  A
// particle's weights are added to a shared box kept as 32-bit words, which is
// flushed into per-species 64-bit global sums; from these the solve forms
// rho = sum_s q_s W_s 2^-48 in a fixed species order.  Integer addition is
// associative, so rho does not depend on the order in which atomics land: the
// FP64 form is bit-reproducible.  A node's sum stays below 2^64 up to 65536
// particle weights per species; a flush that would wrap raises
// OHPIC_ERR_CAPACITY.
//
// What bounds the push: the FP64 pipe (two lanes per SM), which each instruction of
// a warp holds for 16 cycles.  So what can be computed exactly elsewhere is: cells,
// offsets and the deposit's weights in integers, the gather's twelve weight products
// in integers too (f64_fixed.cuh), and the rotation without its exactly zero
// products: 44 FP64 instructions per particle with B along z instead of 75.
// 128x128x64 x 32 ppc x 2 species, tiles of 8 x 8 x 8, halo 2 (push, ms):
//   two particles per thread, 64-bit shared atomics (compare-and-swap loops)  11.34
//   + 32-bit words in the shared box                                          10.05
//   + the rotation without zero products                                       8.89
//   + weight products in integers                                              8.97
//   + one particle per thread (its loop fits the instruction cache)            7.75
//   + no sums kept from one particle to the next (17 registers)                7.02
//   + 1 - x of cell 0 in integers, the kinetic sums a compile-time choice      6.54
//   + the next particle copied to shared memory meanwhile                      5.88
// That is 44 FP64 instructions per particle, 82% of the pipe's time.  Also tried: every
// second weight product in FP64 7.23 (for 7.02), the next particle's loads into
// registers an iteration ahead 7.01, three CTAs per SM 7.81, without integer products
// 8.66 (for 7.75), the copy as a run-time choice 6.39 (for 5.88: it spills).
#include "f64_fixed.cuh"
#include "tile_common.cuh"

namespace ohpic {
namespace {

__device__ __forceinline__ void add_checked(unsigned long long *p, unsigned long long v, DevDiag *d)
{
    const unsigned long long old = atomicAdd(p, v);
    if (old + v < old) flag_error(d, OHPIC_ERR_CAPACITY, 20);
}

// The 8 weights of a particle outside the staged box, straight into the global sums.
__device__ __forceinline__ void deposit_global48(const Geom &g, unsigned long long *w, int ix, int iy, int iz,
                                                 const unsigned long long u[8], DevDiag *d)
{
    const int ix1 = ix + 1 == g.nx ? 0 : ix + 1;
    const int iy1 = iy + 1 == g.ny ? 0 : iy + 1;
    const int iz1 = iz + 1 == g.nz ? 0 : iz + 1;
    const int64_t y0 = (int64_t)iy * g.nx, y1 = (int64_t)iy1 * g.nx;
    const int64_t z0 = (int64_t)iz * g.nx * g.ny, z1 = (int64_t)iz1 * g.nx * g.ny;
    add_checked(w + ix + y0 + z0, u[0], d);
    add_checked(w + ix1 + y0 + z0, u[1], d);
    add_checked(w + ix + y1 + z0, u[2], d);
    add_checked(w + ix1 + y1 + z0, u[3], d);
    add_checked(w + ix + y0 + z1, u[4], d);
    add_checked(w + ix1 + y0 + z1, u[5], d);
    add_checked(w + ix + y1 + z1, u[6], d);
    add_checked(w + ix1 + y1 + z1, u[7], d);
}

// The shared box keeps a node's 64-bit sum as two 32-bit words (all low words, then
// all high ones): 32-bit shared atomics are native, while a 64-bit shared atomic
// add is a compare-and-swap loop, and a warp's lanes, holding consecutive particles
// of the cell order, retried it on the same few nodes (11.34 -> 10.05 ms).
struct Box48 {
    unsigned *lo, *hi;
    __device__ __forceinline__ void add8(int key, int sx, int sxy, const unsigned long long u[8]) const
    {
        const int off[8] = {0, 1, sx, sx + 1, sxy, sxy + 1, sxy + sx, sxy + sx + 1};
        unsigned old[8];
#pragma unroll
        for (int v = 0; v < 8; ++v) old[v] = atomicAdd(lo + key + off[v], (unsigned)u[v]);
#pragma unroll
        for (int v = 0; v < 8; ++v)
            atomicAdd(hi + key + off[v], (unsigned)(u[v] >> 32) + (unsigned)(old[v] + (unsigned)u[v] < old[v]));
    }
};

// The shared box into the species' global sums, one atomic per non-zero node.
__device__ __forceinline__ void flush_box48(const TileArgs &a, const Item &it, const Box48 &box)
{
    const Geom &g = a.g;
    unsigned long long *w = a.wsum + (int64_t)it.sp * g.ncell;
    const int sx = g.sx, sy = g.sy, sz = g.sz;
    for (RowWalk r(sx, sy); r.cz < sz; r.next(sy)) {
        const int y = wrap_near(it.y0 - g.halo + r.by, g.ny);
        const int z = wrap_near(it.z0 - g.halo + r.cz, g.nz);
        unsigned long long *row = w + (int64_t)g.nx * (y + (int64_t)g.ny * z);
        const int base = sx * (r.by + sy * r.cz);
        for (int ax = r.lane; ax < sx; ax += r.width) {
            const unsigned long long v = ((unsigned long long)box.hi[base + ax] << 32) | box.lo[base + ax];
            if (v) add_checked(row + wrap_near(it.x0 - g.halo + ax, g.nx), v, a.diag);
        }
    }
}

// The three E components of a node (the padded node's fourth is never read).
struct d3 {
    double x, y, z;
};

__device__ __forceinline__ d3 node3(const dnode *p, bool shared)
{
    d3 r;
    if (shared) {
        const double2 a = *(const double2 *)p;
        r.x = a.x;
        r.y = a.y;
        r.z = p->z;
    } else {
        const double2 a = __ldg((const double2 *)p);
        r.x = a.x;
        r.y = a.y;
        r.z = __ldg(&p->z);
    }
    return r;
}

// E nodes of the cell with low corner (ix, iy, iz): from the staged box when key >= 0.
__device__ __forceinline__ void load_nodes3(const TileArgs &a, const Box &b, int key, int ix, int iy, int iz,
                                            const dnode *sE, d3 nd[8])
{
    const dnode *q;
    int64_t sx, sxy;
    const bool in = key >= 0;
    if (in) {
        q = sE + key;
        sx = b.sx;
        sxy = b.sxy;
    } else {
        const Geom &g = a.g;
        sx = g.gx;
        sxy = (int64_t)g.gx * g.gy;
        q = (const dnode *)a.epad + (ix + g.halo) + sx * (iy + g.halo) + sxy * (iz + g.halo);
    }
    nd[0] = node3(q, in);
    nd[1] = node3(q + 1, in);
    nd[2] = node3(q + sx, in);
    nd[3] = node3(q + sx + 1, in);
    nd[4] = node3(q + sxy, in);
    nd[5] = node3(q + sxy + 1, in);
    nd[6] = node3(q + sxy + sx, in);
    nd[7] = node3(q + sxy + sx + 1, in);
}

// Particle i's words into this thread's slots (one per array, 256 threads apart).  The
// thread reads back only what it copied, so no barrier is needed, and the copy holds
// no registers (loaded a particle ahead into registers, the push spilled).
template <bool VELOCITY>
__device__ __forceinline__ void fetch_f64(double *slots, const PartF64 &p, int64_t i)
{
    double *s = slots + threadIdx.x;
    copy8(s, p.x + i);
    copy8(s + 256, p.y + i);
    copy8(s + 512, p.z + i);
    if (VELOCITY) {
        copy8(s + 768, p.vx + i);
        copy8(s + 1024, p.vy + i);
        copy8(s + 1280, p.vz + i);
    }
}

// Which components of B are zero on the whole grid: the Boris rotation's products with
// a zero component are exact zeros, so leaving them out gives the same bits with
// 8 (B along z) or no FP64 operations instead of 18.
enum Rotation { ROT_FULL, ROT_Z, ROT_NONE };

// ENERGY: the push keeps the kinetic sums (a.with_energy); as a run-time choice their
// six FP64 instructions were issued, predicated off, for every particle.
template <int MODE, bool STRICT, int ROT = ROT_FULL, bool ENERGY = false>
__global__ void __launch_bounds__(256, 2) tiled_f64(TileArgs a, PartF64 p)
{
    using Ops = typename std::conditional<STRICT, StrictOps, FastOps>::type;
    constexpr bool kGather = MODE != MODE_DEPOSIT;
    constexpr bool kMove = MODE == MODE_PUSH || MODE == MODE_MOVE;
    constexpr bool kDeposit = MODE == MODE_PUSH || MODE == MODE_DEPOSIT;

    Item it;
    if (!get_item<1>(a, it)) return;
    const Geom &g = a.g;
    const Box box = make_box(g, it);
    extern __shared__ __align__(32) unsigned char smem[];
    const int s3 = g.sx * g.sy * g.sz;
    dnode *sE = (dnode *)smem;
    // the next particle's coordinates and velocities, copied while this one is computed
    double *next = (double *)(smem + (box.on ? (kGather ? (size_t)s3 * sizeof(dnode) : 0) + (kDeposit ? (size_t)s3 * 8 : 0)
                                             : 0));
    if (it.g0 + threadIdx.x < it.g1) fetch_f64<kGather>(next, p, it.g0 + threadIdx.x);
    Box48 sbox;
    sbox.lo = (unsigned *)(smem + (kGather ? (size_t)s3 * sizeof(dnode) : 0));
    sbox.hi = sbox.lo + s3;
    if (box.on) {
        stage_tile<dnode, unsigned long long>(a, it, sE, (unsigned long long *)sbox.lo, kGather, kDeposit);
        __syncthreads();
    }

    const int sp = it.sp;
    const SpeciesConst &c = a.sc[sp];
    const double fnx = (double)g.nx, fny = (double)g.ny, fnz = (double)g.nz;
    const long long bnx = __double_as_longlong(fnx), bny = __double_as_longlong(fny), bnz = __double_as_longlong(fnz);
    unsigned ncx = 0, ncy = 0, ncz = 0, nout = 0;
    double ke = 0.0, px = 0.0, py = 0.0, pz = 0.0;
    unsigned long long *wsum = a.wsum + (int64_t)sp * g.ncell;

    for (int64_t i = it.g0 + threadIdx.x; i < it.g1; i += blockDim.x) {
        copies_landed();
        const double *own = next + threadIdx.x;
        double x = own[0], y = own[256], z = own[512], vx = 0.0, vy = 0.0, vz = 0.0;
        if (kGather) {
            vx = own[768];
            vy = own[1024];
            vz = own[1280];
        }
        if (i + blockDim.x < it.g1) fetch_f64<kGather>(next, p, i + blockDim.x);
        if (kGather) {
            Split sx_, sy_, sz_;
            const int ix = split_cell(x, sx_), iy = split_cell(y, sy_), iz = split_cell(z, sz_);
            if ((unsigned)ix >= (unsigned)g.nx || (unsigned)iy >= (unsigned)g.ny ||
                (unsigned)iz >= (unsigned)g.nz) {
                flag_error(a.diag, OHPIC_ERR_BOUNDS, 1);
                continue;
            }
            const int key = box.key(ix, iy, iz);
            nout += key < 0;
            d3 nd[8];
            load_nodes3(a, box, key, ix, iy, iz, sE, nd);
            double wx0, wx1, wy0, wy1, wz0, wz1;
            double ex, ey, ez;
            if (STRICT) {
                // x - floor(x) exactly (linear_interpolator.f90:47-52), from the bits
                cic<double>(a.weights, split_frac(sx_), wx0, wx1);
                cic<double>(a.weights, split_frac(sy_), wy0, wy1);
                cic<double>(a.weights, split_frac(sz_), wz0, wz1);
                // ret = ret + v*rx*ry*rz, i (x) outermost (linear_interpolator.f90:62-66).
                const double wxs[2] = {wx0, wx1}, wys[2] = {wy0, wy1}, wzs[2] = {wz0, wz1};
                ex = 0.0; ey = 0.0; ez = 0.0;
#pragma unroll
                for (int ii = 0; ii < 2; ++ii)
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk) {
                            const d3 v = nd[ii + 2 * jj + 4 * kk];
                            ex = Ops::add(ex, Ops::mul(Ops::mul(Ops::mul(v.x, wxs[ii]), wys[jj]), wzs[kk]));
                            ey = Ops::add(ey, Ops::mul(Ops::mul(Ops::mul(v.y, wxs[ii]), wys[jj]), wzs[kk]));
                            ez = Ops::add(ez, Ops::mul(Ops::mul(Ops::mul(v.z, wxs[ii]), wys[jj]), wzs[kk]));
                        }
            } else {
                double ww[8];
                Unit xr, xc, yr, yc, zr, zc;
                if (split_units(sx_, xr, xc) && split_units(sy_, yr, yc) && split_units(sz_, zr, zc)) {
                    // the products (wx wy) wz in integers, bit for bit (f64_fixed.cuh)
                    const bool ref = a.weights == OHPIC_WEIGHTS_REFERENCE;   // node floor(x) takes r
                    const Unit x0 = ref ? xr : xc, x1 = ref ? xc : xr, y0 = ref ? yr : yc, y1 = ref ? yc : yr;
                    const Unit z0 = ref ? zr : zc, z1 = ref ? zc : zr;
                    const Unit a00 = unit_mul(x0, y0), a10 = unit_mul(x1, y0), a01 = unit_mul(x0, y1),
                               a11 = unit_mul(x1, y1);
                    ww[0] = unit_double(unit_mul(a00, z0));
                    ww[1] = unit_double(unit_mul(a10, z0));
                    ww[2] = unit_double(unit_mul(a01, z0));
                    ww[3] = unit_double(unit_mul(a11, z0));
                    ww[4] = unit_double(unit_mul(a00, z1));
                    ww[5] = unit_double(unit_mul(a10, z1));
                    ww[6] = unit_double(unit_mul(a01, z1));
                    ww[7] = unit_double(unit_mul(a11, z1));
                } else {
                    cic<double>(a.weights, split_frac(sx_), wx0, wx1);
                    cic<double>(a.weights, split_frac(sy_), wy0, wy1);
                    cic<double>(a.weights, split_frac(sz_), wz0, wz1);
                    const double a00 = wx0 * wy0, a10 = wx1 * wy0, a01 = wx0 * wy1, a11 = wx1 * wy1;
                    ww[0] = a00 * wz0; ww[1] = a10 * wz0; ww[2] = a01 * wz0; ww[3] = a11 * wz0;
                    ww[4] = a00 * wz1; ww[5] = a10 * wz1; ww[6] = a01 * wz1; ww[7] = a11 * wz1;
                }
                ex = 0.0; ey = 0.0; ez = 0.0;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    ex = fma(nd[n].x, ww[n], ex);
                    ey = fma(nd[n].y, ww[n], ey);
                    ez = fma(nd[n].z, ww[n], ez);
                }
            }
            if (MODE == MODE_INTERP) {
                double *o = a.interp_out + 3 * i;
                o[0] = ex;
                o[1] = ey;
                o[2] = ez;
            }
            if (kMove) {
                // Boris (particle_mover_boris.f90:42-56); t and s are per-species constants.
                // Strict: the half kick (qm*E)*dt2 in the reference's order.  Otherwise
                // hq = qm*dt2 is rounded once on the host and each half kick is one
                // FMA (six FP64 operations fewer per particle on the narrow FP64 pipe).
                double upm0, upm1, upm2;
                if (STRICT) {
                    const double qm = c.qm, dt2 = c.dt2;
                    upm0 = Ops::add(vx, Ops::mul(Ops::mul(qm, ex), dt2));
                    upm1 = Ops::add(vy, Ops::mul(Ops::mul(qm, ey), dt2));
                    upm2 = Ops::add(vz, Ops::mul(Ops::mul(qm, ez), dt2));
                } else {
                    upm0 = fma(c.hq, ex, vx);
                    upm1 = fma(c.hq, ey, vy);
                    upm2 = fma(c.hq, ez, vz);
                }
                double upp0 = upm0, upp1 = upm1, upp2 = upm2;
                if constexpr (ROT == ROT_FULL) {
                    const double upa0 = Ops::add(upm0, Ops::sub(Ops::mul(upm1, c.t[2]), Ops::mul(upm2, c.t[1])));
                    const double upa1 = Ops::add(upm1, Ops::sub(Ops::mul(upm2, c.t[0]), Ops::mul(upm0, c.t[2])));
                    const double upa2 = Ops::add(upm2, Ops::sub(Ops::mul(upm0, c.t[1]), Ops::mul(upm1, c.t[0])));
                    upp0 = Ops::add(upm0, Ops::sub(Ops::mul(upa1, c.s[2]), Ops::mul(upa2, c.s[1])));
                    upp1 = Ops::add(upm1, Ops::sub(Ops::mul(upa2, c.s[0]), Ops::mul(upa0, c.s[2])));
                    upp2 = Ops::add(upm2, Ops::sub(Ops::mul(upa0, c.s[1]), Ops::mul(upa1, c.s[0])));
                } else if constexpr (ROT == ROT_Z) {
                    // (one rounding per product, as the full form leaves them)
                    const double upa0 = __dadd_rn(upm0, __dmul_rn(upm1, c.t[2]));
                    const double upa1 = __dsub_rn(upm1, __dmul_rn(upm0, c.t[2]));
                    upp0 = __dadd_rn(upm0, __dmul_rn(upa1, c.s[2]));
                    upp1 = __dsub_rn(upm1, __dmul_rn(upa0, c.s[2]));
                }
                if (STRICT) {
                    const double qm = c.qm, dt2 = c.dt2;
                    vx = Ops::add(upp0, Ops::mul(Ops::mul(qm, ex), dt2));
                    vy = Ops::add(upp1, Ops::mul(Ops::mul(qm, ey), dt2));
                    vz = Ops::add(upp2, Ops::mul(Ops::mul(qm, ez), dt2));
                } else {
                    vx = fma(c.hq, ex, upp0);
                    vy = fma(c.hq, ey, upp1);
                    vz = fma(c.hq, ez, upp2);
                }
                // Position (:60-62) and the periodic boundary applied twice; the
                // comparisons run on the bit patterns, the rare wraps in FP64.
                x = Ops::add(x, Ops::mul(vx, c.dt));
                y = Ops::add(y, Ops::mul(vy, c.dt));
                z = Ops::add(z, Ops::mul(vz, c.dt));
                const bool wx = lt0(x) || ge_bits(x, bnx);
                const bool wy = lt0(y) || ge_bits(y, bny);
                const bool wz = lt0(z) || ge_bits(z, bnz);
                ncx += wx; ncy += wy; ncz += wz;
                if (wx || wy || wz) {
#pragma unroll
                    for (int rep = 0; rep < 2; ++rep) {
                        if (lt0(x)) x = Ops::add(fnx, x);
                        if (ge_bits(x, bnx)) x = Ops::sub(x, fnx);
                        if (lt0(y)) y = Ops::add(fny, y);
                        if (ge_bits(y, bny)) y = Ops::sub(y, fny);
                        if (lt0(z)) z = Ops::add(fnz, z);
                        if (ge_bits(z, bnz)) z = Ops::sub(z, fnz);
                    }
                }
                if (ENERGY) {
                    ke = fma(vx, vx, fma(vy, vy, fma(vz, vz, ke)));
                    px += vx; py += vy; pz += vz;
                }
                p.x[i] = x; p.y[i] = y; p.z[i] = z;
                p.vx[i] = vx; p.vy[i] = vy; p.vz[i] = vz;
            }
        }
        if (kDeposit) {
            Split tx_, ty_, tz_;
            const int jx = split_cell(x, tx_), jy = split_cell(y, ty_), jz = split_cell(z, tz_);
            if ((unsigned)jx >= (unsigned)g.nx || (unsigned)jy >= (unsigned)g.ny ||
                (unsigned)jz >= (unsigned)g.nz) {
                flag_error(a.diag, OHPIC_ERR_BOUNDS, 2);
                continue;
            }
            // rx*ry*rz of linear_scatter.f90:41-52 in 2^-48 fixed point; the
            // charge amount is applied per species when rho is formed
            unsigned long long w[8];
            fixed_weights48(a.weights, split_frac48(tx_), split_frac48(ty_), split_frac48(tz_), w);
            const int key = box.key(jx, jy, jz);
            if (key >= 0) {
                sbox.add8(key, box.sx, box.sxy, w);
            } else {
                deposit_global48(g, wsum, jx, jy, jz, w, a.diag);
                if (!kGather) ++nout;
            }
        }
    }
    if (kDeposit && box.on) {
        __syncthreads();
        flush_box48(a, it, sbox);
    }
    if (kMove || kGather) flush_diag<double>(a, sp, ncx, ncy, ncz, nout, ke, px, py, pz);
}

}  // namespace

template <typename P>
static void launch_k(ohpic_ctx *c, void (*kernel)(TileArgs, P), const TileArgs &a, int64_t blocks, size_t smem,
                     const P &parts)
{
    if (blocks <= 0) return;
    allow_tile_shared(c, kernel);
    kernel<<<(unsigned)blocks, 256, smem, c->stream>>>(a, parts);
    ++c->launches;
}

template <bool ENERGY>
static auto push_kernel(bool xy_zero, double bz)
{
    return !xy_zero    ? tiled_f64<MODE_PUSH, false, ROT_FULL, ENERGY>
           : bz != 0.0 ? tiled_f64<MODE_PUSH, false, ROT_Z, ENERGY>
                       : tiled_f64<MODE_PUSH, false, ROT_NONE, ENERGY>;
}

void launch_tiled_f64(ohpic_ctx *c, const TileArgs &a, int mode, int strict, int64_t blocks, size_t smem)
{
    const PartF64 &pp = c->p64[c->cur];
    // (move and interp are always strict, push and deposit never)
    switch (mode * 2 + (strict ? 1 : 0)) {
    case MODE_PUSH * 2: {
        const double *b = c->cfg.b0;
        const bool xy = b[0] == 0.0 && b[1] == 0.0;
        if (a.with_energy)
            launch_k(c, push_kernel<true>(xy, b[2]), a, blocks, smem, pp);
        else
            launch_k(c, push_kernel<false>(xy, b[2]), a, blocks, smem, pp);
        break;
    }
    case MODE_MOVE * 2 + 1:
        if (a.with_energy)
            launch_k(c, tiled_f64<MODE_MOVE, true, ROT_FULL, true>, a, blocks, smem, pp);
        else
            launch_k(c, tiled_f64<MODE_MOVE, true>, a, blocks, smem, pp);
        break;
    case MODE_DEPOSIT * 2:
    case MODE_DEPOSIT * 2 + 1: launch_k(c, tiled_f64<MODE_DEPOSIT, false>, a, blocks, smem, pp); break;
    case MODE_INTERP * 2 + 1: launch_k(c, tiled_f64<MODE_INTERP, true>, a, blocks, smem, pp); break;
    }
}

}  // namespace ohpic
