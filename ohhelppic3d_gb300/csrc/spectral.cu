// spectral.cu -- the pooled periodic field solve of small grids in four kernels with
// our own FFTs, and the E stencil of every periodic solve.
//
// Reference: t_PoissonFieldSolver%solve (src/field_solver/poisson_field_solver.f90:90-175).
//
//   k_plane_forward   one CTA (or a cluster of two) per z plane and slot: rho from
//                     the weight sums (which it clears), FFT along x of two real
//                     rows per complex line, FFT along y, spectrum out
//   k_pencils         one CTA per few (ky, kx) columns: FFT along z, Green's
//                     function, inverse FFT along z, in place
//   k_plane_inverse   per z plane: inverse FFT along y, then along x two real rows
//                     per complex line, phi out
//   k_stencil_columns E on the padded nodes
//
// The server solves the fields of every run of one grid size together.  Its grids
// are small, so a solve is a chain of kernels that each last as long as their
// latency (rho, three transform kernels each way, scaling, stencil), and a batched
// cuFFT plan transforms every slot of a pool, in use or not.  Here a transform's
// passes between two barriers of the whole grid are one kernel, its data staying
// in shared memory; slots not in use cost an early exit; and each kernel is
// launched while the one before it drains (programmatic dependent launch): it
// loads its twiddles, then waits for its input.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "field_nodes.cuh"
#include "line_fft.cuh"
#include "ohpic_internal.cuh"
#include "pdl.cuh"

namespace ohpic {
namespace {

using V = float2;

// Everything the plane and pencil kernels need of a grid.
struct SpecArgs {
    int nx, ny, nz, nxh;
    int H;                 // row pairs: ceil(ny / 2)
    int CS;                // CTAs (a cluster) per plane
    int Hc, W;             // row pairs and columns per CTA of the cluster: ceil(H / CS), ceil(nxh / CS)
    int px;                // pitch of a row pair's line (odd: lines across threads hit different banks)
    int part;              // elements of one shared buffer
    int C, Cshift;         // columns per pencil CTA, a power of two
    LinePlan lx, ly, lz;
    FastDiv dHc, dW, dnx, dnxh;
    const V *twx, *twy, *twz;
    const double *green;
    int64_t ncell, nspec;
    unsigned long long *wsum;
    int nsp;
    const double *q;       // charges of every slot, [slot][nsp]
    const int *on;         // slot in use
};

__device__ __forceinline__ V *stage_twiddles(V *dst, const V *src, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
    return dst + n;
}

__device__ __forceinline__ float node_value(const SpecArgs &a, const RhoScale &r, const double *q,
                                            unsigned long long *w)
{
    if (a.nsp <= 2) {
        const unsigned long long W[2] = {w[0], a.nsp > 1 ? w[a.ncell] : 0ull};
        return node_rho2(W, a.nsp, q, r);
    }
    return node_rho(w, a.ncell, a.nsp, q, r);
}

// One plane (k_plane_forward, k_plane_inverse): a cluster of CS CTAs, rank r holding
// row pairs [r Hc, (r + 1) Hc) while transforming along x and columns [r W, (r + 1) W)
// while transforming along y, exchanged through distributed shared memory (CL;
// CS = 1 has no exchange).
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

// Stores v at shared offset p of CTA `rank` of the cluster.
__device__ __forceinline__ void store_peer(float2 *p, unsigned rank, float2 v)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(r), "f"(v.x), "f"(v.y) : "memory");
}
template <bool CL>
__global__ void k_plane_forward(const __grid_constant__ SpecArgs a, float *rho, V *spec)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ RhoScale scale;
    V *twx = (V *)smem, *twy = twx + a.nx, *A = twy + a.ny, *B = A + a.part;
    stage_twiddles(twx, a.twx, a.nx);
    stage_twiddles(twy, a.twy, a.ny);
    const int slot = blockIdx.y;
    const int plane = CL ? (int)blockIdx.x / a.CS : (int)blockIdx.x, rank = CL ? (int)blockIdx.x - plane * a.CS : 0;
    pdl_wait();
    if (a.on && !a.on[slot]) return;   // the same for every CTA of a cluster
    const int64_t z0 = (int64_t)plane * a.nx * a.ny;
    rho += slot * a.ncell + z0;
    const double *q = a.q + (int64_t)slot * a.nsp;
    if (threadIdx.x == 0) scale = rho_scale(q, a.nsp);
    __syncthreads();
    unsigned long long *w = a.wsum + (int64_t)slot * a.nsp * a.ncell + z0;
    const int h0 = rank * a.Hc;
    // two real rows per complex line
    for (unsigned t = threadIdx.x; t < (unsigned)(a.Hc * a.nx); t += blockDim.x) {
        const int hl = (int)div_by(a.dnx, t), x = (int)t - hl * a.nx;
        float v[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int y = 2 * (h0 + hl) + j;
            if (y >= a.ny) continue;
            const int i = y * a.nx + x;
            v[j] = node_value(a, scale, q, w + i);
            rho[i] = v[j];
            for (int s = 0; s < a.nsp; ++s) w[s * a.ncell + i] = 0ull;
        }
        V c;
        c.x = v[0];
        c.y = v[1];
        A[hl * a.px + x] = c;
    }
    __syncthreads();
    V *R = line_fft(a.lx, A, B, (unsigned)a.Hc, a.dHc, 1, a.px, twx);
    V *F = R == A ? B : A;
    if (CL) cluster_sync();   // every CTA is done with its F
    // the two rows' spectra, kx = 0 .. nx / 2, to the CTA that holds column kx
    for (unsigned t = threadIdx.x; t < (unsigned)(a.Hc * a.nxh); t += blockDim.x) {
        const int hl = (int)div_by(a.dnxh, t), k = (int)t - hl * a.nxh;
        const int y = 2 * (h0 + hl);
        if (y >= a.ny) break;
        const V u = R[hl * a.px + k], m = R[hl * a.px + (k ? a.nx - k : 0)];
        V c, d;
        c.x = 0.5f * (u.x + m.x);
        c.y = 0.5f * (u.y - m.y);
        d.x = 0.5f * (u.y + m.y);
        d.y = 0.5f * (m.x - u.x);
        if (CL) {
            const int to = (int)div_by(a.dW, (unsigned)k), kk = k - to * a.W;
            store_peer(F + y * a.W + kk, (unsigned)to, c);
            if (y + 1 < a.ny) store_peer(F + (y + 1) * a.W + kk, (unsigned)to, d);
        } else {
            F[y * a.nxh + k] = c;
            if (y + 1 < a.ny) F[(y + 1) * a.nxh + k] = d;
        }
    }
    if (CL) cluster_sync();
    else __syncthreads();
    const int k0 = rank * a.W, own = min(a.W, a.nxh - k0);
    const V *S = line_fft(a.ly, F, R, (unsigned)a.W, a.dW, a.W, 1, twy);
    pdl_launch();
    spec += slot * a.nspec + (int64_t)plane * a.ny * a.nxh;
    for (unsigned t = threadIdx.x; t < (unsigned)(a.ny * a.W); t += blockDim.x) {
        const int y = (int)div_by(a.dW, t), kk = (int)t - y * a.W;
        if (kk < own) spec[y * a.nxh + k0 + kk] = S[t];
    }
}

__global__ void k_pencils(const __grid_constant__ SpecArgs a, V *spec)
{
    extern __shared__ __align__(16) unsigned char smem[];
    V *tw = (V *)smem, *A = tw + a.nz, *B = A + a.nz * a.C;
    stage_twiddles(tw, a.twz, a.nz);
    pdl_wait();
    if (a.on && !a.on[blockIdx.y]) return;
    const int cols = a.ny * a.nxh, c0 = blockIdx.x * a.C, total = a.nz * a.C;
    spec += (int64_t)blockIdx.y * a.nspec;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int z = i >> a.Cshift, c = c0 + (i & (a.C - 1));
        V v;
        v.x = v.y = 0.f;
        if (c < cols) v = spec[(int64_t)z * cols + c];
        A[i] = v;
    }
    __syncthreads();
    const FastDiv dC{(unsigned)a.C, a.C > 1 ? 1u << (32 - a.Cshift) : 0u};
    V *S = line_fft(a.lz, A, B, (unsigned)a.C, dC, a.C, 1, tw);
    // times the Green's function; the inverse transform is the forward one of
    // the values with real and imaginary parts exchanged
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int z = i >> a.Cshift, c = c0 + (i & (a.C - 1));
        const double g = c < cols ? a.green[(int64_t)z * cols + c] : 0.0;
        const V v = S[i];
        V r;
        r.x = (float)((double)v.y * g);
        r.y = (float)((double)v.x * g);
        S[i] = r;
    }
    __syncthreads();
    const V *Z = line_fft(a.lz, S, S == A ? B : A, (unsigned)a.C, dC, a.C, 1, tw);
    pdl_launch();
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int z = i >> a.Cshift, c = c0 + (i & (a.C - 1));
        if (c < cols) spec[(int64_t)z * cols + c] = Z[i];   // parts still exchanged
    }
}

template <bool CL>
__global__ void k_plane_inverse(const __grid_constant__ SpecArgs a, const V *spec, float *phi)
{
    extern __shared__ __align__(16) unsigned char smem[];
    V *twx = (V *)smem, *twy = twx + a.nx, *A = twy + a.ny, *B = A + a.part;
    stage_twiddles(twx, a.twx, a.nx);
    stage_twiddles(twy, a.twy, a.ny);
    const int plane = CL ? (int)blockIdx.x / a.CS : (int)blockIdx.x, rank = CL ? (int)blockIdx.x - plane * a.CS : 0;
    pdl_wait();
    const int slot = blockIdx.y;
    if (a.on && !a.on[slot]) return;
    const int k0 = rank * a.W, own = min(a.W, a.nxh - k0), h0 = rank * a.Hc;
    spec += slot * a.nspec + (int64_t)plane * a.ny * a.nxh;
    for (unsigned t = threadIdx.x; t < (unsigned)(a.ny * a.W); t += blockDim.x) {
        const int y = (int)div_by(a.dW, t), kk = (int)t - y * a.W;
        V v;
        v.x = v.y = 0.f;
        if (kk < own) v = spec[y * a.nxh + k0 + kk];
        A[t] = v;
    }
    __syncthreads();
    V *S = line_fft(a.ly, A, B, (unsigned)a.W, a.dW, a.W, 1, twy);
    V *U = S, *G = S == A ? B : A;   // the rows' spectra, and where the packed lines go
    if (CL) {
        // every row to the CTA that holds it
        U = G;
        G = S;
        cluster_sync();
        for (unsigned t = threadIdx.x; t < (unsigned)(a.ny * a.W); t += blockDim.x) {
            const int y = (int)div_by(a.dW, t), kk = (int)t - y * a.W;
            const int to = (int)div_by(a.dHc, (unsigned)(y >> 1));
            if (kk < own) store_peer(U + (y - 2 * to * a.Hc) * a.nxh + k0 + kk, (unsigned)to, S[t]);
        }
        cluster_sync();
    }
    // rows 2h and 2h + 1 (spectra a_k, b_k) as one line g_k = a_k + i b_k; a real
    // row's spectrum has a real mean and (even nx) a real last mode
    for (unsigned t = threadIdx.x; t < (unsigned)(a.Hc * a.nx); t += blockDim.x) {
        const int hl = (int)div_by(a.dnx, t), k = (int)t - hl * a.nx;
        const int y = 2 * (h0 + hl);
        const bool lower = k < a.nxh;
        const int kk = lower ? k : a.nx - k;
        V u, v;
        u.x = u.y = v.x = v.y = 0.f;
        if (y < a.ny) u = swap_parts(U[2 * hl * a.nxh + kk]);
        if (y + 1 < a.ny) v = swap_parts(U[(2 * hl + 1) * a.nxh + kk]);
        if (kk == 0 || 2 * kk == a.nx) u.y = v.y = 0.f;
        V g;   // exchanged again for the forward transform below
        g.y = lower ? u.x - v.y : u.x + v.y;
        g.x = lower ? u.y + v.x : v.x - u.y;
        G[hl * a.px + k] = g;
    }
    __syncthreads();
    const V *R = line_fft(a.lx, G, U, (unsigned)a.Hc, a.dHc, 1, a.px, twx);
    pdl_launch();
    phi += slot * a.ncell + (int64_t)plane * a.nx * a.ny;
    for (unsigned t = threadIdx.x; t < (unsigned)(a.Hc * a.nx); t += blockDim.x) {
        const int hl = (int)div_by(a.dnx, t), x = (int)t - hl * a.nx;
        const int y = 2 * (h0 + hl);
        if (y >= a.ny) break;
        const V r = R[hl * a.px + x];
        phi[y * a.nx + x] = r.y;
        if (y + 1 < a.ny) phi[(y + 1) * a.nx + x] = r.x;
    }
}

// E on the padded nodes, kStencilZ planes per thread (one padded column of x and y):
// the thread's phi column is read once, and every load of its planes is in flight
// before the first node is formed.  Blocks are numbered over a plane's nodes
// first, then groups of planes, then slots, so the divisions are 32-bit and one
// chain serves kStencilZ nodes.  Bound by the padded E's write: 256^3 FP32 150 ->
// 65 us (5.4 TB/s), 64x64x256 13.6 -> 7.3 us, against one node per thread found by
// two 64-bit divisions.  clear, when given, are 8-byte words to zero (the push's
// tallies).
constexpr int kStencilZ = 4;

template <typename T, typename NodeT>
__global__ void __launch_bounds__(256) k_stencil_columns(const __grid_constant__ Geom g, const T *phi, NodeT *epad,
                                                         const int *on, unsigned long long *clear, int nclear)
{
    const unsigned plane = (unsigned)(g.gx * g.gy), nb = (plane + 255u) / 256u;
    const unsigned b1 = blockIdx.x / nb, nzb = (unsigned)(g.gz + kStencilZ - 1) / kStencilZ, slot = b1 / nzb;
    const unsigned t = (blockIdx.x - b1 * nb) * 256u + threadIdx.x;
    const int z0 = (int)(b1 - slot * nzb) * kStencilZ;
    const unsigned py = t / (unsigned)g.gx, px = t - py * (unsigned)g.gx;
    const int i = wrapn((int)px - g.halo, g.nx), j = wrapn((int)py - g.halo, g.ny);
    const int im = i == 0 ? g.nx - 1 : i - 1, ip = i + 1 == g.nx ? 0 : i + 1;
    const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j + 1 == g.ny ? 0 : j + 1;
    int k = wrapn(z0 - 1 - g.halo, g.nz);
    pdl_wait();
    if (clear && blockIdx.x == 0)
        for (int c = threadIdx.x; c < nclear; c += 256) clear[c] = 0ull;
    if (t >= plane || (on && !on[slot])) return;
    phi += slot * g.ncell;
    const int64_t nxy = (int64_t)g.nx * g.ny;
    const int at = i + g.nx * j, axm = im + g.nx * j, axp = ip + g.nx * j, aym = i + g.nx * jm, ayp = i + g.nx * jp;
    T c[kStencilZ + 2], xm[kStencilZ], xp[kStencilZ], ym[kStencilZ], yp[kStencilZ];
#pragma unroll
    for (int u = 0; u < kStencilZ + 2; ++u) {
        const T *p = phi + k * nxy;
        c[u] = p[at];
        if (u >= 1 && u <= kStencilZ) {
            xm[u - 1] = p[axm];
            xp[u - 1] = p[axp];
            ym[u - 1] = p[aym];
            yp[u - 1] = p[ayp];
        }
        k = k + 1 == g.nz ? 0 : k + 1;
    }
    pdl_launch();
    epad += (int64_t)slot * g.gz * plane + (int64_t)z0 * plane + t;
#pragma unroll
    for (int u = 0; u < kStencilZ; ++u) {
        if (z0 + u >= g.gz) break;
        const T p0 = c[u + 1];
        NodeT e;
        e.x = T(0.5) * ((xm[u] - p0) + (p0 - xp[u]));
        e.y = T(0.5) * ((ym[u] - p0) + (p0 - yp[u]));
        e.z = T(0.5) * ((c[u] - p0) + (p0 - c[u + 2]));
        e.w = T(0);
        epad[(int64_t)u * plane] = e;
    }
}

}  // namespace

// The plan of one grid: the kernels' arguments and the twiddles' device memory.
struct Spectral {
    SpecArgs a;
    void *tw;
    size_t plane_smem, pencil_smem;
    int plane_threads, pencil_threads;
};

namespace {

// Shared memory of a plane CTA (two buffers and the twiddles): two CTAs per SM.
constexpr size_t kPlaneSmem = 100 * 1024;

// The CTAs per plane (a cluster; 0: the grid stays with cuFFT), such that two CTAs
// share an SM.  One solve, E included, against cuFFT with a kernel each for rho,
// scaling and stencil (us): 16^3 11.8 (33), 32^3 15.5 (37), 64^3 20.6 (37), 96^3
// 37 (62), 128^3 65 (82).  A plane that needs more than two CTAs stays with cuFFT,
// which is bound by memory there (160^2: 133 against 120; 256^2: 390 against 262).
int plane_cluster(const SpecArgs &a)
{
    for (int cs = 1; cs <= 2; ++cs) {
        const int64_t Hc = (a.H + cs - 1) / cs, W = (a.nxh + cs - 1) / cs;
        const int64_t part = std::max(std::max(Hc * a.px, (int64_t)a.ny * W), 2 * Hc * a.nxh);
        if (part <= 32768 && sizeof(V) * (size_t)(2 * part + a.nx + a.ny) <= kPlaneSmem) return cs;
    }
    return 0;
}

}  // namespace

Spectral *spectral_create(const Geom &g, const double *green)
{
    SpecArgs a = {};
    a.nx = g.nx; a.ny = g.ny; a.nz = g.nz;
    a.nxh = g.nxh;
    a.H = (g.ny + 1) / 2;
    a.px = g.nx | 1;
    if (!line_plan(g.nx, a.lx) || !line_plan(g.ny, a.ly) || !line_plan(g.nz, a.lz)) return nullptr;
    a.CS = plane_cluster(a);
    if (!a.CS) return nullptr;
    a.Hc = (a.H + a.CS - 1) / a.CS;
    a.W = (a.nxh + a.CS - 1) / a.CS;
    a.part = (int)std::max(std::max((int64_t)a.Hc * a.px, (int64_t)a.ny * a.W), 2 * (int64_t)a.Hc * a.nxh);
    const size_t plane_smem = sizeof(V) * (size_t)(2 * a.part + a.nx + a.ny);
    // enough pencil CTAs for the chip, at least 4 columns (one 32-byte sector) each
    const int cols = a.ny * a.nxh;
    a.C = 4;
    a.Cshift = 2;
    while (a.C < 32 && cols / (2 * a.C) >= 152 && sizeof(V) * (size_t)(4 * a.C + 1) * a.nz <= 96 * 1024) {
        a.C *= 2;
        ++a.Cshift;
    }
    const size_t pencil_smem = sizeof(V) * (size_t)(2 * a.C + 1) * a.nz;
    if (pencil_smem > kPlaneSmem) return nullptr;
    a.dHc = fast_div((unsigned)a.Hc);
    a.dW = fast_div((unsigned)a.W);
    a.dnx = fast_div((unsigned)a.nx);
    a.dnxh = fast_div((unsigned)a.nxh);
    a.green = green;
    a.ncell = g.ncell;
    a.nspec = g.nspec;
    std::vector<double> t;
    for (int n : {a.nx, a.ny, a.nz}) line_twiddles(n, t);
    const std::vector<float> tf(t.begin(), t.end());
    void *tw = nullptr;
    if (cudaMalloc(&tw, sizeof(float) * tf.size()) != cudaSuccess ||
        cudaMemcpy(tw, tf.data(), sizeof(float) * tf.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        if (tw) cudaFree(tw);
        return nullptr;
    }
    a.twx = (const V *)tw;
    a.twy = a.twx + a.nx;
    a.twz = a.twy + a.ny;
    auto threads = [](int64_t elements) {   // about four elements per thread, whole warps
        return (int)std::min<int64_t>(std::max<int64_t>((elements / 4 + 31) / 32 * 32, 64), 512);
    };
    // (always: the 48 KB that need no opt-in hold a kernel's static shared memory too)
    auto allow = [](auto k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlaneSmem) == cudaSuccess;
    };
    if (!(allow(k_plane_forward<false>) && allow(k_plane_forward<true>) && allow(k_plane_inverse<false>) &&
          allow(k_plane_inverse<true>) && allow(k_pencils))) {
        cudaGetLastError();
        cudaFree(tw);
        return nullptr;
    }
    return new Spectral{a, tw, plane_smem, pencil_smem, threads(a.part), threads((int64_t)a.nz * a.C)};
}

void spectral_destroy(Spectral *s)
{
    if (!s) return;
    if (s->tw) cudaFree(s->tw);
    delete s;
}

// The E stencil over `slots` grids of one size.
template <typename T, typename NodeT>
void launch_stencil(cudaStream_t st, const Geom &g, int slots, const T *phi, NodeT *epad, const int *on,
                    unsigned long long *clear, int nclear)
{
    const int64_t nb = ((int64_t)g.gx * g.gy + 255) / 256, nzb = (g.gz + kStencilZ - 1) / kStencilZ;
    launch_overlapped(st, dim3((unsigned)(nb * nzb * slots)), dim3(256), 0, 1, k_stencil_columns<T, NodeT>, g, phi, epad,
                      on, clear, nclear);
}

template void launch_stencil<float, float4>(cudaStream_t, const Geom &, int, const float *, float4 *, const int *,
                                            unsigned long long *, int);
template void launch_stencil<double, dnode>(cudaStream_t, const Geom &, int, const double *, dnode *, const int *,
                                            unsigned long long *, int);

cudaError_t spectral_solve(const Spectral &s, cudaStream_t st, const FieldPool &p)
{
    SpecArgs a = s.a;
    a.wsum = p.wsum;
    a.nsp = p.nsp;
    a.q = p.q;
    a.on = p.on;
    const dim3 planes((unsigned)(a.nz * a.CS), (unsigned)p.slots);
    const dim3 pencils((unsigned)((a.ny * a.nxh + a.C - 1) / a.C), (unsigned)p.slots);
    // (the chain's first kernel may follow other streams' work: a plain dependency)
    launch_clusters<false>(st, planes, dim3(s.plane_threads), s.plane_smem, a.CS,
                           a.CS > 1 ? k_plane_forward<true> : k_plane_forward<false>, a, p.rho, (V *)p.spec);
    launch_overlapped(st, pencils, dim3(s.pencil_threads), s.pencil_smem, 1, k_pencils, a, (V *)p.spec);
    launch_overlapped(st, planes, dim3(s.plane_threads), s.plane_smem, a.CS,
                      a.CS > 1 ? k_plane_inverse<true> : k_plane_inverse<false>, a, (const V *)p.spec, p.phi);
    launch_stencil<float, float4>(st, p.g, p.slots, p.phi, p.epad, p.on, nullptr, 0);
    return cudaGetLastError();
}

}  // namespace ohpic
