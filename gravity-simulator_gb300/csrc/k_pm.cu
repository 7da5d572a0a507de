// k_pm.cu -- particle-mesh gravity (src/acceleration_PM.c:15-391) and the
// cosmological leapfrog (src/integrator_cosmology_leapfrog.c:24-255).
//
// One evaluation on a g^3 periodic mesh:
//   deposit        cloud-in-cell deposit of the masses, eight FP64 atomic adds per
//                  particle (the reference's OpenMP loop has unsynchronised += here);
//   the potential  the density contrast rho / (V_cell rho_mean) - 1, formed where the
//                  mesh is first read (a deposit into a mesh of -1 would round every
//                  addition to the contrast's last bit), convolved with -1/k^2 (0 at
//                  k = 0), from a table by the integer |n|^2: in place for the sizes
//                  of k_fft.cu, otherwise cuFFT D2Z (FFTW's layout: g x g x (g/2+1)),
//                  k_pm_green, and cuFFT Z2D, unnormalised;
//   k_pm_gradient  fourth-order central differences of phi into the
//                  acceleration mesh, without their constant factor;
//   interpolation  cloud-in-cell, back to the particles; the caller's multiplier
//                  carries the factor.
// A step of the cosmological leapfrog is one particle kernel between two
// evaluations (k_pm_particles): interpolation, the kick that ends a step, the kick
// and the drift that begin the next, the periodic wrap, and the deposit at the
// new positions.  As five kernels these took 463 us a step at 128^3 particles, with
// the accelerations and momenta written and read in between; fused, 409 us; with
// the cells and fractions of the deposit kept for the interpolation at the same
// positions, and the two kicks in one, 336 us (80 FP64 operations a particle, 98
// before).
// Every kernel computes the reference's quantity in FP64.  The FP64 pipe of
// this GPU runs at 1/64 of the FP32 rate and bounds the particle kernels, so
// they use algebraically equal forms with fewer FP64 operations than the
// reference's expressions: weight products shared between the eight
// corners, fused multiply-adds, the cell index by a directed addition of 2^52,
// constant factors folded into one multiplier, comparisons on the bits (an FP64
// comparison costs as much as an add).  These round
// differently from the reference's order by a few ulps, far below the
// differences of the transforms (against FFTW's) and of the atomic
// deposit order.  The file is compiled with --fmad=false; the fused
// operations are the explicit fma() calls.
//
// Memory: delta / phi g^3 doubles, the acceleration mesh 3 g^3 doubles: 32 g^3
// bytes, 537 MB at g = 256; with cuFFT also the spectrum g^2 (g/2+1) complex.
#include "gs_fft.h"
#include "gs_fp64.cuh"
#include "gs_internal.h"

#include <cufft.h>

#include <cmath>
#include <cstdio>
#include <memory>

namespace gs {
namespace {

constexpr int TPB = 256;
inline unsigned blocks(long long n) { return (unsigned)((n + TPB - 1) / TPB); }

const char *cufft_name(cufftResult r)
{
    switch (r) {
    case CUFFT_SUCCESS: return "CUFFT_SUCCESS";
    case CUFFT_INVALID_PLAN: return "CUFFT_INVALID_PLAN";
    case CUFFT_ALLOC_FAILED: return "CUFFT_ALLOC_FAILED";
    case CUFFT_INVALID_VALUE: return "CUFFT_INVALID_VALUE";
    case CUFFT_INTERNAL_ERROR: return "CUFFT_INTERNAL_ERROR";
    case CUFFT_EXEC_FAILED: return "CUFFT_EXEC_FAILED";
    case CUFFT_SETUP_FAILED: return "CUFFT_SETUP_FAILED";
    case CUFFT_INVALID_SIZE: return "CUFFT_INVALID_SIZE";
    default: return "cuFFT error";
    }
}

#define GS_CUFFT(call)                                                                   \
    do {                                                                                 \
        cufftResult r_ = (call);                                                         \
        if (r_ != CUFFT_SUCCESS)                                                         \
            return GS_RAISE(r_ == CUFFT_ALLOC_FAILED ? GRAV_MEMORY_ERROR : GRAV_FAILURE,   \
                            "%s failed: %s", #call, cufft_name(r_));                     \
    } while (0)

// Mesh geometry of one evaluation (src/acceleration_PM.c:35-37).
struct PmGeom {
    double cx, cy, cz;   // box centre
    double half;         // box_length / 2
    double inv_cell;     // 1 / (box_length / g)
    double half_cells;   // g / 2
    int g;
};

__device__ __forceinline__ int wrap_index(int n, int g)
{
    // the reference indexes n % g; n >= 0 inside the box.  A particle
    // outside it (n < 0) wraps here instead of indexing out of bounds.
    const int r = n % g;
    return r < 0 ? r + g : r;
}

// Cell indices and weights of one particle (src/acceleration_PM.c:44-58).  Inside
// the box the cell is the integer part of u = (x - c + half) / cell, formed as
// (x - c) / cell + g / 2 (x - c first, so that a box far from the origin loses
// nothing) and taken by adding 2^52 rounded down: six FP64 operations a dimension.
__device__ __forceinline__ void cic_cell(const double xi[3], const PmGeom &G, int idx[2][3],
                                         double w[2][3])
{
    const double c[3] = {G.cx, G.cy, G.cz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double u = fma(xi[d] - c[d], G.inv_cell, G.half_cells);
        if ((unsigned)__double2hiint(u) < 0x41d00000u) {   // 0 <= u < 2^30
            const double t = __dadd_rd(u, 0x1p52);
            const int nd = __double2loint(t);
            w[1][d] = u - (t - 0x1p52);
            w[0][d] = 1.0 - w[1][d];
            idx[0][d] = nd < G.g ? nd : nd % G.g;
            idx[1][d] = idx[0][d] + 1 < G.g ? idx[0][d] + 1 : 0;
        } else {
            const double normalized = (xi[d] - c[d] + G.half) * G.inv_cell;
            const int nd = (int)normalized;
            const double weight = normalized - nd;
            w[1][d] = weight;
            w[0][d] = 1.0 - weight;
            idx[0][d] = wrap_index(nd, G.g);
            idx[1][d] = wrap_index(nd + 1, G.g);
        }
    }
}

// Cells and fractions of every particle at its last deposit, which are those of
// the interpolation that follows at the same positions: 15 of its 54 FP64
// operations for 32 bytes a particle (null: not kept).
struct CicKept {
    double *w;       // 3n: the weight of the upper cell on each axis
    ushort4 *cell;   // n: the lower cell (a mesh has at most 1,290 cells a side)
};

__device__ __forceinline__ void keep_cic(const CicKept &K, int i, const int idx[2][3],
                                         const double w[2][3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) K.w[3 * (size_t)i + d] = w[1][d];
    K.cell[i] = make_ushort4(idx[0][0], idx[0][1], idx[0][2], 0);
}

__device__ __forceinline__ void kept_cic(const CicKept &K, int i, int g, int idx[2][3], double w[2][3])
{
    const ushort4 c = K.cell[i];
    idx[0][0] = c.x;
    idx[0][1] = c.y;
    idx[0][2] = c.z;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        w[1][d] = K.w[3 * (size_t)i + d];
        w[0][d] = 1.0 - w[1][d];
        idx[1][d] = idx[0][d] + 1 < g ? idx[0][d] + 1 : 0;
    }
}

// Corner order of the reference's eight terms: bit 0 x, bit 1 y, bit 2 z
// (a constant in unrolled loops, so the per-corner arrays stay in registers).
__host__ __device__ constexpr int corner_bits(int c)
{
    return c == 3 ? 4 : (c == 4 ? 3 : c);
}

__device__ __forceinline__ void deposit_one(const double xi[3], double mi, const PmGeom &G,
                                            double *__restrict__ delta, const CicKept &K, int i)
{
    int idx[2][3];
    double w[2][3];
    cic_cell(xi, G, idx, w);
    if (K.w) keep_cic(K, i, idx, w);
    const long long g = G.g, g2 = g * g;
    double mx[2], mxy[2][2];
#pragma unroll
    for (int bx = 0; bx < 2; ++bx) {
        mx[bx] = mi * w[bx][0];
#pragma unroll
        for (int by = 0; by < 2; ++by) mxy[bx][by] = mx[bx] * w[by][1];
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int bx = corner_bits(c) & 1, by = (corner_bits(c) >> 1) & 1,
                  bz = (corner_bits(c) >> 2) & 1;
        const long long cell = idx[bx][0] * g2 + idx[by][1] * g + idx[bz][2];
        atomicAdd(delta + cell, mxy[bx][by] * w[bz][2]);
    }
}

// src/acceleration_PM.c:112-210, in units of the gradient mesh
__device__ __forceinline__ void interp_one(const int idx[2][3], const double w[2][3], const PmGeom &G,
                                           const double *__restrict__ acc, double s[3])
{
    const long long g = G.g, g2 = g * g;
    double wxy[2][2];
#pragma unroll
    for (int bx = 0; bx < 2; ++bx)
#pragma unroll
        for (int by = 0; by < 2; ++by) wxy[bx][by] = w[bx][0] * w[by][1];
    s[0] = s[1] = s[2] = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int bx = corner_bits(c) & 1, by = (corner_bits(c) >> 1) & 1,
                  bz = (corner_bits(c) >> 2) & 1;
        const long long cell = idx[bx][0] * g2 + idx[by][1] * g + idx[bz][2];
        const double wc = wxy[bx][by] * w[bz][2];
        const double *ac = acc + cell * 3;
        s[0] = fma(ac[0], wc, s[0]);
        s[1] = fma(ac[1], wc, s[1]);
        s[2] = fma(ac[2], wc, s[2]);
    }
}

__global__ void k_pm_deposit(const double *__restrict__ x, const double *__restrict__ m, int n,
                             PmGeom G, double *__restrict__ delta, CicKept K)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double xi[3] = {x[3 * (size_t)i], x[3 * (size_t)i + 1], x[3 * (size_t)i + 2]};
    deposit_one(xi, m[i], G, delta, K, i);
}

// The contrast where the library's transforms read the mesh.
__global__ void k_pm_contrast(double *__restrict__ mesh, long long cells, MeshScale scale)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < cells) mesh[i] = contrast(mesh[i], scale.device ? *scale.device : scale.value);
}

// -1 / (|n|^2 (2 pi / L)^2) by the integer |n|^2 of a mode (src/acceleration_PM.c:
// 321-345), 0 for the mean; the division is made once per value instead of once
// per mode (25 us a transform at 128^3).
__global__ void k_pm_green_table(double *__restrict__ table, int len, double two_pi_over_l2)
{
    const int k2 = blockIdx.x * blockDim.x + threadIdx.x;
    if (k2 >= len) return;
    const double k_sq = (double)k2 * two_pi_over_l2;   // 0 also where it underflows
    table[k2] = k_sq == 0.0 ? 0.0 : -1.0 / k_sq;
}

__global__ void k_pm_green(double2 *__restrict__ spec, int g, const double *__restrict__ table)
{
    // fewer than 2^31 modes: 32-bit index arithmetic
    const unsigned h = g / 2 + 1, ug = g;
    const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ug * ug * h) return;
    const unsigned ij = e / h;
    const int k = (int)(e - ij * h);
    const int i = (int)(ij / ug), j = (int)(ij - (unsigned)i * ug);
    const int kx = (i < (int)h) ? i : i - g;
    const int ky = (j < (int)h) ? j : j - g;
    const double kernel = __ldg(table + kx * kx + ky * ky + k * k);
    double2 v = spec[e];
    v.x *= kernel;
    v.y *= kernel;
    spec[e] = v;
}

// src/acceleration_PM.c:212-272 without the constant factor / (12 cell_length):
// phi[-2] - 8 phi[-1] + 8 phi[+1] - phi[+2] as (phi[-2] - phi[+2]) +
// 8 (phi[+1] - phi[-1]).
__global__ void k_pm_gradient(const double *__restrict__ phi, int g, double *__restrict__ acc)
{
    // at most 2^31 cells: 32-bit index arithmetic
    const unsigned ug = g, g2 = ug * ug;
    const unsigned index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= g2 * ug) return;
    const unsigned ij = index / ug;
    const int k = (int)(index - ij * ug), i = (int)(ij / ug), j = (int)(ij - (unsigned)i * ug);
    const int c[3] = {i, j, k};
    const unsigned st[3] = {g2, ug, 1u};
    // c + o on the periodic axis, o in [-2, 2] (twice for g = 1)
    auto at = [&](int cd, int o) {
        int q = cd + o;
        q += q < 0 ? g : 0;
        q += q < 0 ? g : 0;
        q -= q >= g ? g : 0;
        q -= q >= g ? g : 0;
        return (unsigned)q;
    };
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const unsigned b = index - (unsigned)c[d] * st[d];
        const double pm2 = phi[b + at(c[d], -2) * st[d]], pm1 = phi[b + at(c[d], -1) * st[d]];
        const double pp1 = phi[b + at(c[d], 1) * st[d]], pp2 = phi[b + at(c[d], 2) * st[d]];
        acc[3 * (size_t)index + d] = fma(8.0, pp1 - pm1, pm2 - pp2);
    }
}

__global__ void k_pm_interp(const double *__restrict__ x, int n, PmGeom G,
                            const double *__restrict__ acc, double scale, double *__restrict__ a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double xi[3] = {x[3 * (size_t)i], x[3 * (size_t)i + 1], x[3 * (size_t)i + 2]};
    double s[3];
    int idx[2][3];
    double w[2][3];
    cic_cell(xi, G, idx, w);
    interp_one(idx, w, G, acc, s);
#pragma unroll
    for (int d = 0; d < 3; ++d) a[3 * (size_t)i + d] = s[d] * scale;
}

// Total mass, by a fixed tree (the host's one-by-one sum of 2 million masses took
// 2 ms of a run), then 1 / (V_cell rho_mean) into *inv, rho_mean = mass / volume
// (src/integrator_cosmology_leapfrog.c:66-70).
constexpr int MS_BLOCKS = 256, MS_THREADS = 256;
__device__ __forceinline__ double block_sum(double v, double *sh)
{
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int w = MS_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    return sh[0];
}

__global__ void __launch_bounds__(MS_THREADS)
k_pm_mass_parts(const double *__restrict__ m, int n, double *__restrict__ part)
{
    __shared__ double sh[MS_THREADS];
    double v = 0.0;
    for (long long i = (long long)blockIdx.x * MS_THREADS + threadIdx.x; i < n;
         i += (long long)MS_BLOCKS * MS_THREADS)
        v += m[i];
    v = block_sum(v, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// *inv = 1 / (V_cell rho_mean) from the mass parts
__global__ void __launch_bounds__(MS_THREADS)
k_pm_mass_inv(const double *__restrict__ part, double volume, double cell_volume,
              double *__restrict__ inv)
{
    static_assert(MS_BLOCKS == MS_THREADS, "a part per thread");
    __shared__ double sh[MS_THREADS];
    const double total = block_sum(part[threadIdx.x], sh);
    if (threadIdx.x == 0) *inv = 1.0 / (cell_volume * (total / volume));
}

// ---- cosmological leapfrog (src/integrator_cosmology_leapfrog.c) -----------
// src/system.c:1337-1375 for one coordinate.
__device__ __forceinline__ double periodic(double xv, double c, double bw)
{
    const double p = xv - c;
    // inside, tested on the bits (NaN goes on and fails both comparisons)
    if (abs_bits(p) <= __double_as_longlong(bw)) return xv;
    if (p < -bw) {
        xv = ((int)(p / bw) % 2 != 0) ? fmod(p, bw) + bw : fmod(p, bw);
        xv += c;
    } else if (p > bw) {
        xv = ((int)(p / bw) % 2 != 0) ? fmod(p, bw) - bw : fmod(p, bw);
        xv += c;
    }
    return xv;
}

__global__ void k_cosmo_wrap(double *__restrict__ x, int len, double cx, double cy, double cz,
                             double bw)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    const int d = k % 3;
    x[k] = periodic(x[k], d == 0 ? cx : (d == 1 ? cy : cz), bw);
}

// momentum = a^2 v (:92-98)
__global__ void k_cosmo_momentum(double *__restrict__ p, const double *__restrict__ v, int len,
                                 double t)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    p[k] = t * t * v[k];
}

// velocity = momentum / a^2 at a snapshot (:200-209)
__global__ void k_cosmo_velocity(double *__restrict__ v, const double *__restrict__ p, int len,
                                 double t)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    v[k] = p[k] / (t * t);
}

// The particles between two evaluations: accelerations interpolated from the
// gradient mesh (GATHER) or read from `a`, the kick that ends a step,
// p -= k1 a (:176-183), and with MOVE the kick and the drift that begin the next,
// p -= k2 a (:142-149), x += c p (:152-160), wrapped (:163), and its deposit.
// Both kicks have the same accelerations and are one, p -= (k1 + k2) a.
// k1 and k2 carry 0.5 dt / da and the acceleration's constant factor,
// c = dt / (a^2 da).  Without MOVE the accelerations are kept in `a`.
template <bool GATHER, bool MOVE>
__global__ void k_pm_particles(double *__restrict__ x, double *__restrict__ p,
                               const double *__restrict__ m, double *__restrict__ a, int n,
                               PmGeom G, const double *__restrict__ acc, double k1, double k2,
                               double c, double bw, double *__restrict__ delta, CicKept K)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t q = 3 * (size_t)i;
    double s[3];
    if (GATHER) {
        int idx[2][3];
        double w[2][3];
        kept_cic(K, i, G.g, idx, w);
        interp_one(idx, w, G, acc, s);
    } else {
        for (int d = 0; d < 3; ++d) s[d] = a[q + d];
    }
    const double centre[3] = {G.cx, G.cy, G.cz};
    const double kick = -((GATHER ? k1 : 0.0) + (MOVE ? k2 : 0.0));
    double xi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double pd = fma(kick, s[d], p[q + d]);
        if (MOVE) {
            xi[d] = periodic(fma(c, pd, x[q + d]), centre[d], bw);
            x[q + d] = xi[d];
        } else {
            a[q + d] = s[d];
        }
        p[q + d] = pd;
    }
    if (MOVE) deposit_one(xi, m[i], G, delta, K, i);
}

}  // namespace

// One particle-mesh solver per grid size: cuFFT plans and the meshes.
class PmSolver {
  public:
    ~PmSolver()
    {
        if (fwd_) cufftDestroy(fwd_);
        if (inv_) cufftDestroy(inv_);
    }

    ErrorStatus setup(int g)
    {
        if (g == g_) return ok();
        if (fwd_) cufftDestroy(fwd_);
        if (inv_) cufftDestroy(inv_);
        fwd_ = inv_ = 0;
        g_ = 0;
        const long long cells = (long long)g * g * g;
        GS_TRY(mesh_.reserve((size_t)cells * sizeof(double)));
        GS_TRY(acc_.reserve((size_t)cells * 3 * sizeof(double)));
        if (convolve_supports(g)) {
            GS_TRY(tw_.reserve((size_t)g * sizeof(double2)));
        } else {
            const long long half = (long long)g * g * (g / 2 + 1);
            GS_TRY(spec_.reserve((size_t)half * sizeof(double2)));
            GS_CUFFT(cufftPlan3d(&fwd_, g, g, g, CUFFT_D2Z));
            GS_CUFFT(cufftPlan3d(&inv_, g, g, g, CUFFT_Z2D));
        }
        g_ = g;
        return ok();
    }

    // A run's constants: geometry and the Green's function table.
    ErrorStatus prepare(const double *box_center, double box_width, int g, cudaStream_t s)
    {
        GS_TRY(setup(g));
        const double box_length = box_width * 2.0;
        cell_length_ = box_length / g;
        geom_.cx = box_center[0];
        geom_.cy = box_center[1];
        geom_.cz = box_center[2];
        geom_.half = box_length / 2.0;
        geom_.inv_cell = 1.0 / cell_length_;
        geom_.half_cells = 0.5 * g;
        geom_.g = g;
        const int top = g / 2;
        const int len = 3 * top * top + 1;
        GS_TRY(green_.reserve((size_t)len * sizeof(double)));
        k_pm_green_table<<<blocks(len), TPB, 0, s>>>(green_.as<double>(), len,
                                                     4.0 * M_PI * M_PI / (box_length * box_length));
        GS_CUDA(cudaGetLastError());
        if (convolve_supports(g)) GS_TRY(convolve_table(g, tw_.as<double2>(), s));
        return ok();
    }

    // 1 / (V_cell rho_mean) with rho_mean given.
    void set_mean_density(double rho_mean)
    {
        scale_ = {nullptr, 1.0 / (cell_length_ * cell_length_ * cell_length_ * rho_mean)};
    }

    // The same with rho_mean the total mass over the box's volume.
    ErrorStatus mean_density_of(const double *d_m, int n, double box_width, cudaStream_t s)
    {
        GS_TRY(part_.reserve((MS_BLOCKS + 1) * sizeof(double)));
        double *inv = part_.as<double>() + MS_BLOCKS;
        k_pm_mass_parts<<<MS_BLOCKS, MS_THREADS, 0, s>>>(d_m, n, part_.as<double>());
        k_pm_mass_inv<<<1, MS_THREADS, 0, s>>>(
            part_.as<double>(), (box_width * 2) * (box_width * 2) * (box_width * 2),
            cell_length_ * cell_length_ * cell_length_, inv);
        GS_CUDA(cudaGetLastError());
        scale_ = {inv, 0.0};
        return ok();
    }

    // The mesh ready for a deposit.
    ErrorStatus clear(cudaStream_t s)
    {
        GS_CUDA(cudaMemsetAsync(mesh_.p, 0, (size_t)g_ * g_ * g_ * sizeof(double), s));
        return ok();
    }

    // src/acceleration_PM.c:311-380 from the deposited mesh to the gradient mesh.
    ErrorStatus solve(cudaStream_t s)
    {
        double *mesh = mesh_.as<double>();
        const long long cells = (long long)g_ * g_ * g_;
        if (convolve_supports(g_)) {
            GS_TRY(convolve_mesh(mesh, g_, scale_, green_.as<double>(), tw_.as<double2>(), s));
        } else {
            k_pm_contrast<<<blocks(cells), TPB, 0, s>>>(mesh, cells, scale_);
            GS_CUDA(cudaGetLastError());
            GS_CUFFT(cufftSetStream(fwd_, s));
            GS_CUFFT(cufftExecD2Z(fwd_, mesh, spec_.as<cufftDoubleComplex>()));
            const long long half = (long long)g_ * g_ * (g_ / 2 + 1);
            k_pm_green<<<blocks(half), TPB, 0, s>>>(spec_.as<double2>(), g_, green_.as<double>());
            GS_CUDA(cudaGetLastError());
            GS_CUFFT(cufftSetStream(inv_, s));
            GS_CUFFT(cufftExecZ2D(inv_, spec_.as<cufftDoubleComplex>(), mesh));
        }
        k_pm_gradient<<<blocks(cells), TPB, 0, s>>>(mesh, g_, acc_.as<double>());
        GS_CUDA(cudaGetLastError());
        return ok();
    }

    // Kernels of this library in a step: the particles, the potential (the contrast
    // and the Green's function beside cuFFT) and the gradient.
    int kernels_per_step() const { return 2 + (convolve_supports(g_) ? kConvolveLaunches : 2); }

    // The gradient mesh's constant factor.
    double scale(double H0, double omega_m, double scale_factor) const
    {
        const double cells = (double)((long long)g_ * g_ * g_);
        return ((3.0 / 2.0) * omega_m * H0 * H0) / (scale_factor * cells) / (12.0 * cell_length_);
    }

    const PmGeom &geom() const { return geom_; }
    double *mesh() const { return mesh_.as<double>(); }
    const double *acc() const { return acc_.as<double>(); }

  private:
    int g_ = 0;
    double cell_length_ = 1.0;
    PmGeom geom_{};
    cufftHandle fwd_ = 0, inv_ = 0;
    MeshScale scale_{nullptr, 1.0};
    DBuf mesh_, spec_, acc_, green_, tw_, part_;
};

namespace {

struct PmCall {
    cudaStream_t stream = nullptr;
    PmSolver solver;
    DBuf x, m, a;
    cudaEvent_t ev[2] = {nullptr, nullptr};   // around the step loop
    double loop_ms = 0.0;
    int64_t loop_steps = 0;
    ~PmCall()
    {
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
        if (stream) cudaStreamDestroy(stream);
    }
};

thread_local std::unique_ptr<PmCall> tl_pm;

ErrorStatus pm_call(PmCall **out)
{
    if (!tl_pm) {
        const DeviceInfo *d = nullptr;
        GS_TRY(device_info(&d));
        std::unique_ptr<PmCall> c(new PmCall());
        GS_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        GS_CUDA(cudaEventCreate(&c->ev[0]));
        GS_CUDA(cudaEventCreate(&c->ev[1]));
        tl_pm = std::move(c);
    }
    *out = tl_pm.get();
    return ok();
}

ErrorStatus pm_check(int n, const double *x, const double *m, const double *box_center,
                     int g)
{
    if (!x || !m || !box_center) return GS_RAISE(GRAV_POINTER_ERROR, "NULL array");
    if (n <= 0)
        return GS_RAISE(GRAV_VALUE_ERROR, "Number of particles must be positive. Got: %d", n);
    if (g <= 0) return GS_RAISE(GRAV_VALUE_ERROR, "pm_grid_size must be positive. Got: %d", g);
    if ((long long)g * g * g > (1LL << 31))
        return GS_RAISE(GRAV_VALUE_ERROR, "pm_grid_size %d gives more than 2^31 cells", g);
    return ok();
}

}  // namespace

ErrorStatus pm_acceleration_host(double *a, int n, const double *x, const double *m,
                                 const double *box_center, double box_width, double H0,
                                 double omega_m, double mean_bkg_density, int g,
                                 double scale_factor)
{
    if (!a) return GS_RAISE(GRAV_POINTER_ERROR, "Acceleration array is NULL");
    GS_TRY(pm_check(n, x, m, box_center, g));
    PmCall *c = nullptr;
    GS_TRY(pm_call(&c));
    const size_t b3 = (size_t)n * 3 * sizeof(double);
    GS_TRY(c->x.reserve(b3));
    GS_TRY(c->a.reserve(b3));
    GS_TRY(c->m.reserve((size_t)n * sizeof(double)));
    GS_CUDA(cudaMemcpyAsync(c->x.p, x, b3, cudaMemcpyHostToDevice, c->stream));
    GS_CUDA(cudaMemcpyAsync(c->m.p, m, (size_t)n * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
    PmSolver &pm = c->solver;
    GS_TRY(pm.prepare(box_center, box_width, g, c->stream));
    pm.set_mean_density(mean_bkg_density);
    GS_TRY(pm.clear(c->stream));
    k_pm_deposit<<<blocks(n), TPB, 0, c->stream>>>(c->x.as<double>(), c->m.as<double>(), n, pm.geom(),
                                                   pm.mesh(), CicKept{nullptr, nullptr});
    GS_CUDA(cudaGetLastError());
    GS_TRY(pm.solve(c->stream));
    k_pm_interp<<<blocks(n), TPB, 0, c->stream>>>(c->x.as<double>(), n, pm.geom(), pm.acc(),
                                                  pm.scale(H0, omega_m, scale_factor),
                                                  c->a.as<double>());
    GS_CUDA(cudaGetLastError());
    GS_CUDA(cudaMemcpyAsync(a, c->a.p, b3, cudaMemcpyDeviceToHost, c->stream));
    GS_CUDA(cudaStreamSynchronize(c->stream));
    return ok();
}

// src/integrator_cosmology_leapfrog.c:24-255.  x is advanced in HBM; the
// host v is written only at snapshots (v = p / a^2), as the reference
// writes it, and is otherwise left as given.
ErrorStatus pm_leapfrog_cosmology(CosmologicalSystem *system, SimulationStatus *status,
                                  OutputParam *op, const bool *is_exit, double dt, double a_begin,
                                  double a_final, int g)
{
    const int n = system->num_particles;
    GS_TRY(pm_check(n, system->x, system->m, system->box_center, g));
    const double H0 = system->h * 100.0;
    const double omega_m = system->omega_m, omega_lambda = system->omega_lambda;
    const double *c = system->box_center;
    const double bw = system->box_width;
    PmCall *pc = nullptr;
    GS_TRY(pm_call(&pc));
    cudaStream_t s = pc->stream;
    const int L = 3 * n;
    const size_t b3 = (size_t)L * sizeof(double);
    DBuf x, v, m, p, a;
    GS_TRY(x.reserve(b3));
    GS_TRY(v.reserve(b3));
    GS_TRY(p.reserve(b3));
    // the kept cells and fractions in the accelerations' allocation
    GS_TRY(a.reserve(2 * b3 + (size_t)n * sizeof(ushort4)));
    const CicKept kept = {a.as<double>() + L, reinterpret_cast<ushort4 *>(a.as<double>() + 2 * (size_t)L)};
    GS_TRY(m.reserve((size_t)n * sizeof(double)));
    GS_CUDA(cudaMemcpyAsync(x.p, system->x, b3, cudaMemcpyHostToDevice, s));
    GS_CUDA(cudaMemcpyAsync(v.p, system->v, b3, cudaMemcpyHostToDevice, s));
    GS_CUDA(cudaMemcpyAsync(m.p, system->m, (size_t)n * sizeof(double), cudaMemcpyHostToDevice, s));

    double t = a_begin;
    if (status) status->t = t;
    // snapshots (:49-52, :76-88): the initial one of the caller's arrays
    const bool is_output = op && op->method != OUTPUT_METHOD_DISABLED;
    double next_output_time = is_output ? op->output_interval : 0.0;
    if (is_output && op->output_initial) GS_TRY(output_snapshot_cosmology(op, system, t));
    PmSolver &pm = pc->solver;
    GS_TRY(pm.prepare(c, bw, g, s));
    GS_TRY(pm.mean_density_of(m.as<double>(), n, bw, s));
    k_cosmo_wrap<<<blocks(L), TPB, 0, s>>>(x.as<double>(), L, c[0], c[1], c[2], bw);
    k_cosmo_momentum<<<blocks(L), TPB, 0, s>>>(p.as<double>(), v.as<double>(), L, t);
    GS_CUDA(cudaGetLastError());
    GS_TRY(pm.clear(s));
    k_pm_deposit<<<blocks(n), TPB, 0, s>>>(x.as<double>(), m.as<double>(), n, pm.geom(), pm.mesh(), kept);
    GS_CUDA(cudaGetLastError());
    GS_TRY(pm.solve(s));
    double factor = pm.scale(H0, omega_m, t);   // of the accelerations now in the mesh
    // ceil((a_final - a_begin) / dt) steps; dt = 0 (allowed by the checks)
    // gives no finite count, and no steps are taken
    const double q = (a_final - a_begin) / dt;
    const int64_t total = (std::isfinite(q) && q >= 0.0) ? (int64_t)std::ceil(q) : 0;
    if (status) status->dt = dt;
    int64_t steps = 0;
    GS_CUDA(cudaEventRecord(pc->ev[0], s));
    double k1 = 0.0;        // the pending kick of the step before
    bool gather = true;     // whether it is pending: the accelerations are in the mesh alone
    while (steps < total) {
        if (t + dt > a_final) dt = a_final - t;
        if (status) status->dt = dt;
        // end of the step before, this step's first kick and its drift
        double da = compute_da(t, H0, omega_m, omega_lambda);
        const double k2 = 0.5 * dt / da * factor;
        t += 0.5 * dt;
        da = compute_da(t, H0, omega_m, omega_lambda);
        GS_TRY(pm.clear(s));
        auto move = gather ? k_pm_particles<true, true> : k_pm_particles<false, true>;
        move<<<blocks(n), TPB, 0, s>>>(x.as<double>(), p.as<double>(), m.as<double>(), a.as<double>(),
                                       n, pm.geom(), pm.acc(), k1, k2, dt / (t * t * da), bw,
                                       pm.mesh(), kept);
        GS_CUDA(cudaGetLastError());
        GS_TRY(pm.solve(s));
        factor = pm.scale(H0, omega_m, t);
        k1 = 0.5 * dt / da * factor;
        ++steps;
        t = a_begin + steps * dt;
        if (status) {
            status->t = t;
            status->num_steps = steps;
        }
        const bool stop = steps >= total || (is_exit && *is_exit);
        const bool snap = is_output && t >= next_output_time;
        gather = !(stop || snap);
        if (!gather) {
            // the step's last kick by itself; the next step's takes the stored
            // accelerations
            k_pm_particles<true, false><<<blocks(n), TPB, 0, s>>>(
                x.as<double>(), p.as<double>(), m.as<double>(), a.as<double>(), n, pm.geom(), pm.acc(),
                k1, 0.0, 0.0, bw, pm.mesh(), kept);
            GS_CUDA(cudaGetLastError());
        }
        if (snap) {
            // the host arrays get x and v = p / a^2, then the snapshot (:198-221)
            k_cosmo_velocity<<<blocks(L), TPB, 0, s>>>(v.as<double>(), p.as<double>(), L, t);
            GS_CUDA(cudaGetLastError());
            GS_CUDA(cudaMemcpyAsync(system->x, x.p, b3, cudaMemcpyDeviceToHost, s));
            GS_CUDA(cudaMemcpyAsync(system->v, v.p, b3, cudaMemcpyDeviceToHost, s));
            GS_CUDA(cudaStreamSynchronize(s));
            GS_TRY(output_snapshot_cosmology(op, system, t));
            next_output_time = op->output_count_ * op->output_interval;
        }
        // the flag may have been set while the snapshot was written, after which the
        // step is complete
        if (stop || (snap && is_exit && *is_exit)) break;
    }
    GS_CUDA(cudaEventRecord(pc->ev[1], s));
    GS_CUDA(cudaMemcpyAsync(system->x, x.p, b3, cudaMemcpyDeviceToHost, s));
    GS_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    GS_CUDA(cudaEventElapsedTime(&ms, pc->ev[0], pc->ev[1]));
    pc->loop_ms = ms;
    pc->loop_steps = steps;
    return ok();
}

ErrorStatus pm_last_timing(double *loop_ms, int64_t *steps, int *kernels)
{
    if (!tl_pm) return GS_RAISE(GRAV_VALUE_ERROR, "no cosmological run on this thread");
    if (loop_ms) *loop_ms = tl_pm->loop_ms;
    if (steps) *steps = tl_pm->loop_steps;
    if (kernels) *kernels = tl_pm->solver.kernels_per_step();
    return ok();
}

}  // namespace gs
