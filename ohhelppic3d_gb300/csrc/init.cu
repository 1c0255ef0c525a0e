// init.cu -- device-side initial conditions with the reference injector's streams.
//
// Reference: the driver seeds one PCG32 stream with (42, 52) and advances it by
// rank*1e8 (src/ohhelppic3d.f90:111-112); each species then draws once for
// random_fix (src/radom/random_generator.f90:45-58) and 7 times per particle:
// x, y, z as rand()*(upper-lower)+lower (position_random_uniform_distribution.f90:38-41)
// and 4 draws for the 3-D Maxwellian (velocity_maxwell_distribution3d.f90:41-56,
// with sigma = vth, no factor 2), clipped to +-6 sigma.
//
// Because every particle consumes exactly 7 draws, thread i jumps its copy of
// the stream ahead by 7*i (O(log i) affine-map squaring) and needs no
// communication.  Positions are bit-identical to a host injector using the same
// streams (exact uniform draws, one rounded multiply and one rounded add);
// velocities use the device's log/sqrt/cos/sin and may differ from a host libm in
// the last bit.
//
// The FP32 form keeps what it can off the FP64 pipe (two lanes per SM), which bounded
// it: some 250 FP64 instructions a particle, 80 times the time of its bytes.  Velocities
// come as pairs of floats and are computed in FP64 only where that leaves their rounding
// open (normal_pair.cuh), positions in a box of whole cells come from integers, and a
// thread jumps ahead once and then strides.  Every stored float is the one that the FP64
// computation rounds to.  The whole call, 2^23 particles: 2888 -> 178 us (468 with a box
// of broken cells); 2^26: 22.5 -> 1.05 ms, of which the bytes are 0.28 ms.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "normal_pair.cuh"
#include "ohpic_internal.cuh"

namespace ohpic {
namespace {

constexpr uint64_t kPcgMult = 6364136223846793005ULL;
constexpr double kRefPi = 3.14159265358979;   // src/utils/science_constants.f90:4

struct Pcg {
    uint64_t state, inc;
};

__host__ __device__ inline uint32_t pcg_next(Pcg &r)
{
    const uint64_t old = r.state;
    r.state = old * kPcgMult + r.inc;
    const uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u);
    const uint32_t rot = (uint32_t)(old >> 59u);
    return (xs >> rot) | (xs << ((32u - rot) & 31u));
}

// delta steps of s -> a*s + c as one such map: compose it with itself by squaring.
__host__ __device__ inline void pcg_jump(uint64_t inc, uint64_t delta, uint64_t &am, uint64_t &ap)
{
    uint64_t cm = kPcgMult, cp = inc;
    am = 1u;
    ap = 0u;
    while (delta) {
        if (delta & 1u) {
            am *= cm;
            ap = ap * cm + cp;
        }
        cp = (cm + 1u) * cp;
        cm *= cm;
        delta >>= 1u;
    }
}

__host__ __device__ inline void pcg_advance(Pcg &r, uint64_t delta)
{
    uint64_t am, ap;
    pcg_jump(r.inc, delta, am, ap);
    r.state = am * r.state + ap;
}

__host__ __device__ inline Pcg pcg_seed(uint64_t initstate, uint64_t initseq)
{
    Pcg r{0u, (initseq << 1u) | 1u};
    r.state = r.state * kPcgMult + r.inc;
    r.state += initstate;
    r.state = r.state * kPcgMult + r.inc;
    return r;
}

// pcg32_random_double_r: a 32-bit draw times 2^-32 (exact).
__host__ __device__ inline double unit_draw(uint32_t k) { return (double)k * 2.3283064365386963e-10; }
__host__ __device__ inline double pcg_double(Pcg &r) { return unit_draw(pcg_next(r)); }

struct InitArgs {
    Pcg base;          // stream position of the species' first particle draw
    int64_t n;
    int64_t dst;       // absolute slot of particle 0
    double lo[3], hi[3];
    double vth;
    double drift[3];
    int nx, ny, nz;
    // FP32 form
    uint64_t jump_mul, jump_add;   // the stream's state 7 x (threads of the grid) draws on
    int whole;                     // the box's faces are whole numbers (first, cells)
    unsigned first[3], cells[3];
    int pairs, cold;               // velocities by pairs of floats, vth = 0
    FloatPair sigma, shift[3];
    float clip;
};

// The velocity from its four uniform draws.
__device__ inline void maxwell(double sigma, const double drift[3], double r1, double r2, double r3, double r4,
                               double vel[3])
{
    const double m1 = sigma * sqrt(-2.0 * log(r1)), m3 = sigma * sqrt(-2.0 * log(r3));
    double v[3] = {m1 * cos(2.0 * kRefPi * r2), m1 * sin(2.0 * kRefPi * r2), m3 * sin(2.0 * kRefPi * r4)};
    for (int d = 0; d < 3; ++d) {
        double c = v[d] < sigma * 6 ? v[d] : sigma * 6;
        c = -sigma * 6 > c ? -sigma * 6 : c;
        vel[d] = c + drift[d];
    }
}

__device__ inline void sample(const InitArgs &a, int64_t i, double pos[3], double vel[3])
{
    Pcg r = a.base;
    pcg_advance(r, (uint64_t)(7 * i));
    for (int d = 0; d < 3; ++d) pos[d] = __dadd_rn(__dmul_rn(pcg_double(r), __dsub_rn(a.hi[d], a.lo[d])), a.lo[d]);
    const double r1 = pcg_double(r), r2 = pcg_double(r), r3 = pcg_double(r), r4 = pcg_double(r);
    maxwell(a.vth, a.drift, r1, r2, r3, r4, vel);
}

__global__ void k_init_f64(InitArgs a, PartF64 p, uint32_t *ids)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        double pos[3], vel[3];
        sample(a, i, pos, vel);
        const int64_t o = a.dst + i;
        p.x[o] = pos[0]; p.y[o] = pos[1]; p.z[o] = pos[2];
        p.vx[o] = vel[0]; p.vy[o] = vel[1]; p.vz[o] = vel[2];
        if (ids) ids[o] = (uint32_t)i;
    }
}

__device__ inline void split(double x, int n, int &c, float &o)
{
    int k = (int)floor(x);
    float f = (float)(x - (double)k);
    if (f >= 1.f) { f = 0.f; ++k; }
    if (k >= n) k -= n;
    if (k < 0) k += n;
    c = k;
    o = f;
}

// What the pairs leave open, out of the loop's registers.
__device__ __noinline__ float3 maxwell_rounded(double sigma, double dx, double dy, double dz, uint32_t k1, uint32_t k2,
                                               uint32_t k3, uint32_t k4)
{
    const double drift[3] = {dx, dy, dz};
    double vel[3];
    maxwell(sigma, drift, unit_draw(k1), unit_draw(k2), unit_draw(k3), unit_draw(k4), vel);
    return make_float3((float)vel[0], (float)vel[1], (float)vel[2]);
}

__device__ const NormalTables kNormal = make_normal_tables();

// CTAs per SM of the FP32 form (64 registers).
constexpr int kInitPerSm = 4;

__global__ void __launch_bounds__(256, kInitPerSm) k_init_f32(const __grid_constant__ InitArgs a, PartF32 p, uint32_t *ids)
{
    __shared__ NormalTables tab;
    for (unsigned k = threadIdx.x; k < sizeof(tab) / 16; k += 256) ((uint4 *)&tab)[k] = ((const uint4 *)&kNormal)[k];
    __syncthreads();

    const int64_t stride = (int64_t)gridDim.x * 256;
    int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;
    Pcg at = a.base;
    if (i < a.n) pcg_advance(at, (uint64_t)(7 * i));
    for (; i < a.n; i += stride) {
        Pcg r = at;
        at.state = a.jump_mul * at.state + a.jump_add;
        int cell[3];
        float off[3];
        const int n[3] = {a.nx, a.ny, a.nz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const uint32_t k = pcg_next(r);
            if (a.whole) {
                // first + k 2^-32 cells has at most 53 bits: the FP64 sum is exact
                const uint64_t x = (uint64_t)k * a.cells[d];
                int c = (int)(a.first[d] + (unsigned)(x >> 32));
                float f = (float)(uint32_t)x * 2.3283064365386963e-10f;
                if (f >= 1.f) { f = 0.f; ++c; }
                cell[d] = c >= n[d] ? c - n[d] : c;
                off[d] = f;
            } else {
                split(__dadd_rn(__dmul_rn(unit_draw(k), __dsub_rn(a.hi[d], a.lo[d])), a.lo[d]), n[d], cell[d], off[d]);
            }
        }
        const uint32_t k1 = pcg_next(r), k2 = pcg_next(r), k3 = pcg_next(r), k4 = pcg_next(r);
        float v[3];
        bool done = false;
        if (a.cold && k1 && k3) {
            done = true;   // 0 sqrt(..) cos(..) clips to +0
            for (int d = 0; d < 3; ++d) v[d] = a.shift[d].hi;
        } else if (a.pairs && k1 && k3) {
            FloatPair sn, cs, sn3, cs3;
            const FloatPair m1 = pair_mul(radius(k1, tab.log), a.sigma);
            turn(k2, tab.trig, sn, cs);
            const FloatPair m3 = pair_mul(radius(k3, tab.log), a.sigma);
            turn(k4, tab.trig, sn3, cs3);
            done = round_velocity(m1, cs, a.shift[0], a.clip, v[0]);
            done &= round_velocity(m1, sn, a.shift[1], a.clip, v[1]);
            done &= round_velocity(m3, sn3, a.shift[2], a.clip, v[2]);
        }
        if (!done) {
            const float3 w = maxwell_rounded(a.vth, a.drift[0], a.drift[1], a.drift[2], k1, k2, k3, k4);
            v[0] = w.x;
            v[1] = w.y;
            v[2] = w.z;
        }
        const int64_t o = a.dst + i;
        p.cell[o] = pack_cell(cell[0], cell[1], cell[2]);
        p.ox[o] = off[0]; p.oy[o] = off[1]; p.oz[o] = off[2];
        p.vx[o] = v[0]; p.vy[o] = v[1]; p.vz[o] = v[2];
        if (ids) ids[o] = (uint32_t)i;
    }
}

FloatPair pair_of(double x)
{
    const float hi = (float)x;
    return {hi, (float)(x - (double)hi)};
}

// Which of the FP32 form's shorter ways are open to a species: integer positions where
// both faces of its box are whole numbers on every axis; pairs where vth and the drift
// lie well inside the floats' range (a drift of 0 too), so that no pair underflows.
void shorten(InitArgs &a)
{
    constexpr double kLeast = 0x1p-60, kMost = 0x1p60;
    a.whole = 1;
    a.pairs = a.vth >= kLeast && a.vth <= kMost;
    for (int d = 0; d < 3; ++d) {
        const bool whole = a.lo[d] >= 0.0 && a.lo[d] <= a.hi[d] && a.hi[d] <= 0x1p20 && a.lo[d] == floor(a.lo[d]) &&
                           a.hi[d] == floor(a.hi[d]);
        a.whole = a.whole && whole;
        a.first[d] = whole ? (unsigned)a.lo[d] : 0u;
        a.cells[d] = whole ? (unsigned)(a.hi[d] - a.lo[d]) : 0u;
        const double size = fabs(a.drift[d]);
        a.pairs = a.pairs && (size == 0.0 || (size >= kLeast && size <= kMost));
    }
    a.cold = a.vth == 0.0;
    a.sigma = pair_of(a.vth);
    for (int d = 0; d < 3; ++d) a.shift[d] = pair_of(0.0 + a.drift[d]);
    a.clip = (float)(5.99 * a.vth);
}

}  // namespace

int draw_particles(const DrawSpec &d, int64_t *counts, std::string *err)
{
    Pcg rng = pcg_seed(d.initstate, d.initseq);
    pcg_advance(rng, d.advance);
    for (int s = 0; s < d.nspecies; ++s) {
        const ohpic_species_init &p = d.spi[s];
        InitArgs a;
        double volume = 1.0;
        for (int k = 0; k < 3; ++k) {
            a.hi[k] = p.hi[k] < (double)d.n[k] ? p.hi[k] : (double)d.n[k];
            a.lo[k] = p.lo[k] > 0.0 ? p.lo[k] : 0.0;
            const double w = a.hi[k] - a.lo[k];
            volume *= w > 0.0 ? w : 0.0;
            a.drift[k] = p.drift[k];
        }
        // random_fix(ppc * volume): one draw decides whether the fraction rounds up.
        const double value = p.ppc * volume;
        const int64_t fixed = (int64_t)value;
        const int64_t count = pcg_double(rng) <= value - (double)fixed ? fixed + 1 : fixed;
        if (d.cap && count > d.cap[s]) {
            if (err) *err = "init: species " + std::to_string(s) + " needs " + std::to_string(count) + " > capacity";
            return OHPIC_ERR_CAPACITY;
        }
        a.base = rng;
        a.n = count;
        a.dst = d.seg ? d.seg[s] : 0;
        a.vth = p.vth;
        a.nx = d.n[0]; a.ny = d.n[1]; a.nz = d.n[2];
        if (!d.counts_only && count > 0) {
            int64_t blocks = (count + 255) / 256;
            if (d.precision == OHPIC_FP64) {
                if (blocks > 152 * 64) blocks = 152 * 64;
                k_init_f64<<<(unsigned)blocks, 256, 0, d.stream>>>(a, d.p64, d.ids);
            } else {
                if (blocks > 152 * kInitPerSm) blocks = 152 * kInitPerSm;
                shorten(a);
                pcg_jump(a.base.inc, (uint64_t)(7 * 256 * blocks), a.jump_mul, a.jump_add);
                k_init_f32<<<(unsigned)blocks, 256, 0, d.stream>>>(a, d.p32, d.ids);
            }
            if (d.launches) ++*d.launches;
        }
        pcg_advance(rng, (uint64_t)(7 * count));
        if (counts) counts[s] = count;
    }
    return OHPIC_OK;
}

int init_particles(ohpic_ctx *c, uint64_t initstate, uint64_t initseq, uint64_t advance,
                   const ohpic_species_init *spi, int64_t *counts)
{
    DrawSpec d;
    d.stream = c->stream;
    d.precision = c->cfg.precision;
    d.n[0] = c->g.nx; d.n[1] = c->g.ny; d.n[2] = c->g.nz;
    d.initstate = initstate;
    d.initseq = initseq;
    d.advance = advance;
    d.nspecies = c->cfg.nspecies;
    d.spi = spi;
    d.seg = c->seg;
    d.cap = c->cap;
    materialize_records(c);
    d.p64 = c->p64[c->cur];
    d.p32 = c->p32[c->cur];
    d.ids = c->ids[c->cur];
    d.launches = &c->launches;
    int64_t cnt[OHPIC_MAX_SPECIES] = {0};
    const int rc = draw_particles(d, cnt, &c->err);
    if (rc != OHPIC_OK) return rc;
    for (int s = 0; s < c->cfg.nspecies; ++s) {
        c->count[s] = cnt[s];
        if (counts) counts[s] = cnt[s];
    }
    c->sorted = false;
    c->rho_valid = false;
    c->kin_valid = false;
    return OHPIC_OK;
}

}  // namespace ohpic
