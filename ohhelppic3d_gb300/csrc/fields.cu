// fields.cu -- spectral Poisson solve and the E stencil.
//
// Reference: t_PoissonFieldSolver%solve (src/field_solver/poisson_field_solver.f90:90-175)
//   phi = rho; forward R2HC x3; divide by the modified wave number
//   sum_d (2 sin(pi k_d / n_d))^2 (poisson_solver3d.f90:104-117, :184-192); zero k = 0
//   (:194-198); backward HC2R x3 and divide by nx*ny*nz (mpi_fftw3_solver.f90:223-236);
//   then E_d[i] = phi[i] - phi[i+e_d] (:131-145) and E_d[i] = (E_d[i-e_d] + E_d[i]) / 2
//   (:157-171), which combine to E_d[i] = 0.5*((phi[i-e] - phi[i]) + (phi[i] - phi[i+e])).
//
// The tensor-product real half-complex basis of the reference and the R2C
// transform used here diagonalise the same periodic 7-point Laplacian, with the
// same eigenvalue per wave vector, so dividing the cuFFT half spectrum by that
// eigenvalue gives the reference's phi up to rounding.  The Green table holds
// 1/(eigenvalue * nx*ny*nz) in FP64 (0 at k = 0) and is built once on the device
// with the reference's truncated pi literal (src/utils/science_constants.f90:4).
#include <cuda_runtime.h>
#include <cufft.h>
#include <stdint.h>

#include "block_sum.cuh"
#include "field_nodes.cuh"
#include "ohpic_internal.cuh"

namespace ohpic {
namespace {

constexpr double kRefPi = 3.14159265358979;

__device__ __forceinline__ double wave_number(int k, int n)
{
    // poisson_solver3d.f90:114-117
    if (k <= n / 2) return 2.0 * sin(kRefPi * k / (double)n);
    return 2.0 * sin(kRefPi * (n - k) / (double)n);
}

__global__ void k_green(Geom g, double *green)
{
    const int64_t total = g.nspec;
    const double norm = (double)g.nx * (double)g.ny * (double)g.nz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int kx = (int)(i % g.nxh);
        const int ky = (int)((i / g.nxh) % g.ny);
        const int kz = (int)(i / ((int64_t)g.nxh * g.ny));
        if (kx == 0 && ky == 0 && kz == 0) {
            green[i] = 0.0;
            continue;
        }
        const double wx = wave_number(kx, g.nx), wy = wave_number(ky, g.ny), wz = wave_number(kz, g.nz);
        const double wn = wx * wx + wy * wy + wz * wz;
        green[i] = 1.0 / (wn * norm);
    }
}

__global__ void k_scale_z(cufftDoubleComplex *spec, const double *green, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double gf = green[i];
        cufftDoubleComplex v = spec[i];
        v.x *= gf;
        v.y *= gf;
        spec[i] = v;
    }
}

// FP32 spectrum scaled by the FP64 table in FP64 arithmetic.
__global__ void k_scale_c(cufftComplex *spec, const double *green, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double gf = green[i];
        cufftComplex v = spec[i];
        v.x = (float)((double)v.x * gf);
        v.y = (float)((double)v.y * gf);
        spec[i] = v;
    }
}

// ---- pooled fields: many runs of one grid size, slot = blockIdx.y; on[slot] == 0 skips ----

// rho of every active slot from its fixed-point weight sums (nsp species per slot,
// charges q[slot * nsp + s]); the sums are cleared for the next deposit.
__global__ void k_pool_rho(unsigned long long *w, int64_t ncell, int nsp, const double *q, const int *on,
                           float *rho)
{
    const int slot = blockIdx.y;
    if (on && !on[slot]) return;
    w += (int64_t)slot * nsp * ncell;
    rho += (int64_t)slot * ncell;
    q += (int64_t)slot * nsp;
    __shared__ RhoScale r;
    if (threadIdx.x == 0) r = rho_scale(q, nsp);
    __syncthreads();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ncell; t += (int64_t)gridDim.x * blockDim.x) {
        rho[t] = node_rho(w + t, ncell, nsp, q, r);
        for (int s = 0; s < nsp; ++s) w[s * ncell + t] = 0ull;
    }
}

__global__ void k_pool_scale(cufftComplex *spec, int64_t nspec, const double *green, const int *on)
{
    const int slot = blockIdx.y;
    if (on && !on[slot]) return;
    spec += (int64_t)slot * nspec;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nspec; i += (int64_t)gridDim.x * blockDim.x) {
        const double gf = green[i];
        cufftComplex v = spec[i];
        v.x = (float)((double)v.x * gf);
        v.y = (float)((double)v.y * gf);
        spec[i] = v;
    }
}

// One n^3 FP64 component array -> that component of every padded E node (uploaded E).
template <typename T, typename NodeT>
__global__ void k_fill_epad(Geom g, const double *src, int comp, NodeT *epad)
{
    const int64_t total = (int64_t)g.gx * g.gy * g.gz;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int px = (int)(t % g.gx);
        const int py = (int)((t / g.gx) % g.gy);
        const int pz = (int)(t / ((int64_t)g.gx * g.gy));
        const int i = wrapn(px - g.halo, g.nx), j = wrapn(py - g.halo, g.ny), k = wrapn(pz - g.halo, g.nz);
        const T v = (T)src[i + (int64_t)g.nx * (j + (int64_t)g.ny * k)];
        if (comp == 0) epad[t].x = v;
        else if (comp == 1) epad[t].y = v;
        else epad[t].z = v;
    }
}

// Interior of the padded E -> one FP64 component array.
template <typename NodeT>
__global__ void k_epad_component(Geom g, const NodeT *epad, int comp, double *out)
{
    const int64_t total = g.ncell;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t % g.nx);
        const int j = (int)((t / g.nx) % g.ny);
        const int k = (int)(t / ((int64_t)g.nx * g.ny));
        const NodeT e = epad[(i + g.halo) + (int64_t)g.gx * ((j + g.halo) + (int64_t)g.gy * (k + g.halo))];
        out[t] = comp == 0 ? (double)e.x : comp == 1 ? (double)e.y : (double)e.z;
    }
}

template <typename T>
__global__ void k_to_double(const T *in, double *out, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)in[i];
}

template <typename T>
__global__ void k_from_double(const double *in, T *out, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (T)in[i];
}

// FP64 reductions: sum of rho and 0.5 * sum |E|^2 over interior nodes.
template <typename T, typename NodeT>
__global__ void k_field_sums(Geom g, const T *rho, const NodeT *epad, double *charge, double *energy)
{
    double q = 0.0, e2 = 0.0;
    // at most 2^31 cells: the node comes from 32-bit divisions
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < g.ncell; t += (int64_t)gridDim.x * blockDim.x) {
        q += (double)rho[t];
        const unsigned row = (unsigned)t / (unsigned)g.nx, k = row / (unsigned)g.ny;
        const int i = (int)((unsigned)t - row * (unsigned)g.nx), j = (int)(row - k * (unsigned)g.ny);
        const NodeT e = epad[(i + g.halo) + (int64_t)g.gx * ((j + g.halo) + (int64_t)g.gy * (k + g.halo))];
        e2 += (double)e.x * (double)e.x + (double)e.y * (double)e.y + (double)e.z * (double)e.z;
    }
    double v[2] = {q, 0.5 * e2};
    double *const out[2] = {charge, energy};
    block_sum_add(v, out);
}

// FP32 form: rho = sum_s q_s * W_s * 2^-24 from the fixed-point weight sums,
// summed exactly and rounded once to FP32 (node_rho).
struct SpeciesCharges {
    double q[OHPIC_MAX_SPECIES];
    int nspecies;
};

// Four nodes per thread per iteration, every weight-sum load of the four issued
// before the first node is formed: one node at a time, the kernel waited on two
// dependent-free loads per node and ran at a third of its bytes' bandwidth.
// The charges' integer form comes from the host (computing it in each block was
// most of the kernel on a small grid), and the sums are cleared for the next
// deposit as they are read, which saves that deposit's clear.
__global__ void k_wsum_to_rho(unsigned long long *w, int64_t ncell, const __grid_constant__ SpeciesCharges sc,
                              const __grid_constant__ RhoScale r, float *rho)
{
    constexpr int U = 4;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ncell; t += U * stride) {
        unsigned long long W[U][2];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = t + u * stride;
            in[u] = i < ncell;
            W[u][0] = in[u] ? w[i] : 0ull;
            W[u][1] = in[u] && sc.nspecies > 1 ? w[ncell + i] : 0ull;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!in[u]) continue;
            const int64_t i = t + u * stride;
            rho[i] = sc.nspecies <= 2 ? node_rho2(W[u], sc.nspecies, sc.q, r) : node_rho(w + i, ncell, sc.nspecies, sc.q, r);
            for (int s = 0; s < sc.nspecies; ++s) w[s * ncell + i] = 0ull;
        }
    }
}

// FP64 form: rho = (sum_s q_s W_s) 2^-48 from the species' 2^-48 fixed-point
// weight sums, the species added in a fixed order, so rho is bit-reproducible.
__global__ void k_wsum_to_rho64(unsigned long long *w, int64_t ncell, SpeciesCharges sc, double *rho)
{
    constexpr double kUnit48 = 1.0 / 281474976710656.0;   // 2^-48
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ncell; t += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long W[OHPIC_MAX_SPECIES];
#pragma unroll
        for (int s = 0; s < OHPIC_MAX_SPECIES; ++s)
            if (s < sc.nspecies) W[s] = w[s * ncell + t];
        double acc = 0.0;
#pragma unroll
        for (int s = 0; s < OHPIC_MAX_SPECIES; ++s)
            if (s < sc.nspecies) {
                acc += sc.q[s] * (double)W[s];
                w[s * ncell + t] = 0ull;
            }
        rho[t] = acc * kUnit48;
    }
}

int blocks_for(int64_t n)
{
    int64_t b = (n + 255) / 256;
    if (b > 152 * 16) b = 152 * 16;
    return b < 1 ? 1 : (int)b;
}

}  // namespace

// Materialise rho from the fixed-point weight sums left by the last deposit, and
// clear them.
void ensure_rho(ohpic_ctx *c)
{
    if (!c->rho_from_wsum) return;
    SpeciesCharges sc;
    sc.nspecies = c->cfg.nspecies;
    for (int s = 0; s < OHPIC_MAX_SPECIES; ++s) sc.q[s] = s < sc.nspecies ? c->cfg.q[s] : 0.0;
    if (c->cfg.precision == OHPIC_FP32)
        k_wsum_to_rho<<<blocks_for(c->g.ncell), 256, 0, c->stream>>>(c->wsum, c->g.ncell, sc,
                                                                     rho_scale(sc.q, sc.nspecies), (float *)c->rho);
    else
        k_wsum_to_rho64<<<blocks_for(c->g.ncell), 256, 0, c->stream>>>(c->wsum, c->g.ncell, sc, (double *)c->rho);
    ++c->launches;
    c->rho_from_wsum = false;
    c->wsum_clear = true;
}

int fields_setup(ohpic_ctx *c)
{
    const Geom &g = c->g;
    cufftResult r;
    if (c->cfg.precision == OHPIC_FP64) {
        r = cufftPlan3d(&c->plan_r2c, g.nz, g.ny, g.nx, CUFFT_D2Z);
        if (r == CUFFT_SUCCESS) r = cufftPlan3d(&c->plan_c2r, g.nz, g.ny, g.nx, CUFFT_Z2D);
    } else {
        r = cufftPlan3d(&c->plan_r2c, g.nz, g.ny, g.nx, CUFFT_R2C);
        if (r == CUFFT_SUCCESS) r = cufftPlan3d(&c->plan_c2r, g.nz, g.ny, g.nx, CUFFT_C2R);
    }
    if (r != CUFFT_SUCCESS) {
        c->err = "cufftPlan3d failed (" + std::to_string((int)r) + ")";
        return OHPIC_ERR_CUDA;
    }
    c->plans_made = true;
    cufftSetStream(c->plan_r2c, c->stream);
    cufftSetStream(c->plan_c2r, c->stream);
    k_green<<<blocks_for(g.nspec), 256, 0, c->stream>>>(g, c->green);
    ++c->launches;
    return OHPIC_OK;
}

void fields_teardown(ohpic_ctx *c)
{
    if (c->plans_made) {
        cufftDestroy(c->plan_r2c);
        cufftDestroy(c->plan_c2r);
        c->plans_made = false;
    }
}

int solve_fields(ohpic_ctx *c, unsigned long long *clear, int nclear)
{
    const Geom &g = c->g;
    ensure_rho(c);
    cufftResult r;
    if (c->cfg.precision == OHPIC_FP64) {
        r = cufftExecD2Z(c->plan_r2c, (cufftDoubleReal *)c->rho, (cufftDoubleComplex *)c->spec);
        if (r != CUFFT_SUCCESS) goto fail;
        k_scale_z<<<blocks_for(g.nspec), 256, 0, c->stream>>>((cufftDoubleComplex *)c->spec, c->green, g.nspec);
        r = cufftExecZ2D(c->plan_c2r, (cufftDoubleComplex *)c->spec, (cufftDoubleReal *)c->phi);
        if (r != CUFFT_SUCCESS) goto fail;
        launch_stencil<double, dnode>(c->stream, g, 1, (const double *)c->phi, (dnode *)c->epad, nullptr, clear,
                                      nclear);
    } else {
        r = cufftExecR2C(c->plan_r2c, (cufftReal *)c->rho, (cufftComplex *)c->spec);
        if (r != CUFFT_SUCCESS) goto fail;
        k_scale_c<<<blocks_for(g.nspec), 256, 0, c->stream>>>((cufftComplex *)c->spec, c->green, g.nspec);
        r = cufftExecC2R(c->plan_c2r, (cufftComplex *)c->spec, (cufftReal *)c->phi);
        if (r != CUFFT_SUCCESS) goto fail;
        launch_stencil<float, float4>(c->stream, g, 1, (const float *)c->phi, (float4 *)c->epad, nullptr, clear,
                                      nclear);
    }
    c->launches += 2;
    return OHPIC_OK;
fail:
    c->err = "cuFFT exec failed (" + std::to_string((int)r) + ")";
    return OHPIC_ERR_CUDA;
}

void launch_zero(ohpic_ctx *c, void *p, int64_t bytes) { cudaMemsetAsync(p, 0, (size_t)bytes, c->stream); }

// ---- pooled solve (serve.cu): returns the number of launches, or -1 on a cuFFT error ----

int pool_green(cudaStream_t st, const Geom &g, double *green)
{
    k_green<<<blocks_for(g.nspec), 256, 0, st>>>(g, green);
    return 1;
}

int pool_solve(cudaStream_t st, const FieldPool &p)
{
    const Geom &g = p.g;
    if (p.spectral) return spectral_solve(*p.spectral, st, p) == cudaSuccess ? 4 : -1;
    const unsigned slots = (unsigned)p.slots;
    auto grid = [&](int64_t n) {
        int64_t b = (n + 255) / 256;
        const int64_t cap = (152 * 16 + slots - 1) / slots;
        if (b > cap) b = cap;
        return dim3((unsigned)(b < 1 ? 1 : b), slots);
    };
    k_pool_rho<<<grid(g.ncell), 256, 0, st>>>(p.wsum, g.ncell, p.nsp, p.q, p.on, p.rho);
    if (cufftExecR2C(p.r2c, p.rho, p.spec) != CUFFT_SUCCESS) return -1;
    k_pool_scale<<<grid(g.nspec), 256, 0, st>>>(p.spec, g.nspec, p.green, p.on);
    if (cufftExecC2R(p.c2r, p.spec, p.phi) != CUFFT_SUCCESS) return -1;
    launch_stencil<float, float4>(st, g, p.slots, p.phi, p.epad, p.on, nullptr, 0);
    return 5;
}

// rho of one slot from its weight sums (the deposit of the run's last step).
void pool_slot_rho(cudaStream_t st, const FieldPool &p, int slot)
{
    const Geom &g = p.g;
    k_pool_rho<<<dim3(blocks_for(g.ncell), 1), 256, 0, st>>>(p.wsum + (int64_t)slot * p.nsp * g.ncell, g.ncell,
                                                             p.nsp, p.q + (int64_t)slot * p.nsp, nullptr,
                                                             p.rho + (int64_t)slot * g.ncell);
}

// One slot's fields as FP64 arrays: rho, phi, Ex, Ey, Ez (5 * ncell doubles).
void pool_slot_fields(cudaStream_t st, const FieldPool &p, int slot, double *dst)
{
    const Geom &g = p.g;
    const int64_t n = g.ncell, npad = (int64_t)g.gx * g.gy * g.gz;
    k_to_double<float><<<blocks_for(n), 256, 0, st>>>(p.rho + slot * n, dst, n);
    k_to_double<float><<<blocks_for(n), 256, 0, st>>>(p.phi + slot * n, dst + n, n);
    for (int c = 0; c < 3; ++c)
        k_epad_component<float4><<<blocks_for(n), 256, 0, st>>>(g, p.epad + slot * npad, c, dst + (2 + c) * n);
}

// Charge and field energy of one slot (FP64 sums into d->charge, d->field_energy).
void pool_slot_sums(cudaStream_t st, const FieldPool &p, int slot, DevDiag *d)
{
    const Geom &g = p.g;
    cudaMemsetAsync(&d->charge, 0, 2 * sizeof(double), st);
    k_field_sums<float, float4><<<blocks_for(g.ncell), 256, 0, st>>>(
        g, p.rho + slot * g.ncell, p.epad + slot * ((int64_t)g.gx * g.gy * g.gz), &d->charge, &d->field_energy);
}

void launch_field_energy(ohpic_ctx *c)
{
    const Geom &g = c->g;
    ensure_rho(c);
    cudaMemsetAsync(&c->diag->charge, 0, 2 * sizeof(double), c->stream);
    if (c->cfg.precision == OHPIC_FP64)
        k_field_sums<double, dnode><<<blocks_for(g.ncell), 256, 0, c->stream>>>(
            g, (const double *)c->rho, (const dnode *)c->epad, &c->diag->charge, &c->diag->field_energy);
    else
        k_field_sums<float, float4><<<blocks_for(g.ncell), 256, 0, c->stream>>>(
            g, (const float *)c->rho, (const float4 *)c->epad, &c->diag->charge, &c->diag->field_energy);
    ++c->launches;
}

// Field transfers through a device staging buffer of >= 3*ncell doubles.
void field_to_double(ohpic_ctx *c, int which, double *dst)
{
    const Geom &g = c->g;
    const bool f64 = c->cfg.precision == OHPIC_FP64;
    if (which == OHPIC_RHO) ensure_rho(c);
    if (which == OHPIC_RHO || which == OHPIC_PHI) {
        const void *src = which == OHPIC_RHO ? c->rho : c->phi;
        if (f64)
            cudaMemcpyAsync(dst, src, sizeof(double) * g.ncell, cudaMemcpyDeviceToDevice, c->stream);
        else
            k_to_double<float><<<blocks_for(g.ncell), 256, 0, c->stream>>>((const float *)src, dst, g.ncell);
    } else {
        const int comp = which - OHPIC_EX;
        if (f64)
            k_epad_component<dnode><<<blocks_for(g.ncell), 256, 0, c->stream>>>(g, (const dnode *)c->epad, comp, dst);
        else
            k_epad_component<float4><<<blocks_for(g.ncell), 256, 0, c->stream>>>(g, (const float4 *)c->epad, comp,
                                                                                 dst);
    }
    ++c->launches;
}

void field_from_double(ohpic_ctx *c, int which, const double *src)
{
    const Geom &g = c->g;
    const bool f64 = c->cfg.precision == OHPIC_FP64;
    if (which == OHPIC_RHO || which == OHPIC_PHI) {
        void *dst = which == OHPIC_RHO ? c->rho : c->phi;
        if (f64)
            cudaMemcpyAsync(dst, src, sizeof(double) * g.ncell, cudaMemcpyDeviceToDevice, c->stream);
        else
            k_from_double<float><<<blocks_for(g.ncell), 256, 0, c->stream>>>(src, (float *)dst, g.ncell);
    } else {
        const int comp = which - OHPIC_EX;
        if (f64)
            k_fill_epad<double, dnode><<<blocks_for((int64_t)g.gx * g.gy * g.gz), 256, 0, c->stream>>>(
                g, src, comp, (dnode *)c->epad);
        else
            k_fill_epad<float, float4><<<blocks_for((int64_t)g.gx * g.gy * g.gz), 256, 0, c->stream>>>(
                g, src, comp, (float4 *)c->epad);
    }
    ++c->launches;
}

}  // namespace ohpic
