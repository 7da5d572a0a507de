// k_direct.cu -- direct-sum accelerations on sm_103a.
//
// Replaces acceleration_pairwise (src/acceleration.c:177-234).
//
// GRAV_GPU_PAIRWISE (compensated FP32):
//   * positions and masses are packed once per evaluation into a float4
//     array (x, y, z, m) relative to a fixed frame centre, padded to a whole
//     number of 1024-particle tiles with massless far-away particles;
//   * a CTA of 128 threads owns 1024 i-particles (8 per thread, register
//     blocked; two CTAs per SM) and one contiguous j-chunk; j-tiles of 1024
//     particles (16 KiB)
//     stream through a 3-stage shared-memory ring filled by TMA bulk copies
//     (cp.async.bulk + mbarrier complete_tx), read back as broadcast float4;
//   * each pair term is 3 FADD + 3 FFMA + rsqrt + 3 FMUL + 3 FFMA in FP32;
//     each partial sum of 128 pair terms is added into a Kahan-compensated FP32
//     accumulator;
//   * the j-particles are divided in granules of 128 (the length of a plain
//     partial sum), and a row tile's granules into units so that the last wave of
//     resident CTAs is as full as it gets (choose_per); the units' Kahan pairs go
//     to scratch [split][3][N], which a second kernel adds in fixed order, to the
//     precision of an FP64 sum, and scales by G;
//   * up to 20,480 particles the units are 64 rows by 1,024 or 2,048 terms
//     (k_direct_run).
//   Measured at N = 100,000: 3.76 -> 3.51 ms (57 TFLOP/s at 20 per pair term, 0.74
//   of the FP32 FMA peak; the pair term's own ceiling is 20/24 of it).
//
// GRAV_GPU_PAIRWISE_FP64 (reference order): a CTA of a few particles forms
// the pair terms of all other particles, 128 at a time, and sums them in index
// order with every FP64 product, sum, sqrt and quotient rounded separately --
// the same operations as the reference's symmetric loop applies to that
// particle, so the result equals the reference's bit for bit where the
// reference is not FMA-contracted.
#include "gs_fp64.cuh"
#include "gs_internal.h"
#include "gs_ptx.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

namespace gs {

constexpr int DS_THREADS = 128;
constexpr int DS_IPT = 8;
constexpr int DS_ITILE = DS_THREADS * DS_IPT;  // 1024
constexpr int DS_JTILE = 1024;                 // 16 KiB of float4
constexpr int DS_STAGES = 3;
constexpr int DS_SMEM = DS_STAGES * DS_JTILE * 16;
constexpr int DS_GRANULE = 128;                // plain FP32 partials of 128 terms
constexpr int DS_TILE_GRANULES = DS_JTILE / DS_GRANULE;
constexpr int DR_WARPS = 8;                    // k_direct_run
constexpr int DR_THREADS = 32 * DR_WARPS;
constexpr int DR_ROWS = 64;
// k_direct_run up to here, k_direct_sum above: at N = 20,000 159 against 164 us, at
// 24,000 223 against 219 us.
constexpr int DS_RUN_N = 20 * DS_JTILE;
static_assert(DS_ITILE == DS_JTILE, "i and j tiles share the padding unit");

// Padding particle: massless and far from everything (its pair terms are 0).
constexpr float kPadPos = 1.0e15f;

// With a drift (v not null), x += v h first.
__global__ void k_pack_float4(double *__restrict__ x, const double *__restrict__ m,
                              int n, int n_pad, double cx, double cy, double cz,
                              double *__restrict__ xe, const double *__restrict__ v, double h,
                              float4 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    float4 p;
    if (i < n) {
        double y[3] = {x[3 * i + 0], x[3 * i + 1], x[3 * i + 2]};
        if (v) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double e = xe[3 * i + d];
                comp_update(y[d], e, v[3 * i + d], h);
                x[3 * i + d] = y[d];
                xe[3 * i + d] = e;
            }
        }
        p.x = (float)(y[0] - cx);
        p.y = (float)(y[1] - cy);
        p.z = (float)(y[2] - cz);
        p.w = (float)m[i];
    } else {
        p = make_float4(kPadPos, kPadPos, kPadPos, 0.0f);
    }
    out[i] = p;
}

template <bool SOFT>
__device__ __forceinline__ void pair_term(const float4 q, float xi, float yi, float zi,
                                          float eps2, float &ax, float &ay, float &az)
{
    const float dx = q.x - xi;
    const float dy = q.y - yi;
    const float dz = q.z - zi;
    float r2 = fmaf(dx, dx, eps2);
    r2 = fmaf(dy, dy, r2);
    r2 = fmaf(dz, dz, r2);
    float ri = rsqrt_approx(r2);
    if (!SOFT) ri = (r2 > 0.0f) ? ri : 0.0f;   // self term without softening
    const float mr = q.w * ri;
    const float ri2 = ri * ri;
    const float s = mr * ri2;
    ax = fmaf(dx, s, ax);
    ay = fmaf(dy, s, ay);
    az = fmaf(dz, s, az);
}

// Two i-particles per instruction: Blackwell's paired FP32 operations
// (add / mul / fma on float2, each lane rounded as the scalar operation)
// carry the pair terms of particles (k, k+1) together, halving the FP32
// instructions issued per term; the arithmetic of each particle is exactly
// pair_term's (q.x - x_i is formed as q.x + (-x_i)).
template <bool SOFT>
__device__ __forceinline__ void pair_term2(const float4 q, float2 nxi, float2 nyi, float2 nzi,
                                           float2 eps2, float2 &ax, float2 &ay, float2 &az)
{
    const float2 dx = __fadd2_rn(make_float2(q.x, q.x), nxi);
    const float2 dy = __fadd2_rn(make_float2(q.y, q.y), nyi);
    const float2 dz = __fadd2_rn(make_float2(q.z, q.z), nzi);
    float2 r2 = __ffma2_rn(dx, dx, eps2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    float2 ri = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    if (!SOFT) {
        ri.x = (r2.x > 0.0f) ? ri.x : 0.0f;
        ri.y = (r2.y > 0.0f) ? ri.y : 0.0f;
    }
    const float2 mr = __fmul2_rn(make_float2(q.w, q.w), ri);
    const float2 ri2 = __fmul2_rn(ri, ri);
    const float2 sc = __fmul2_rn(mr, ri2);
    ax = __ffma2_rn(dx, sc, ax);
    ay = __ffma2_rn(dy, sc, ay);
    az = __ffma2_rn(dz, sc, az);
}

// One work unit: the IPT * 128 i-particles from pi_tile against the j-particles
// of granules [g0, g1) (128 particles each, the length of a plain FP32 partial
// sum); the unit compensates over its granules, and its Kahan pairs go to
// partial[split][3][plane] at rows row0 + ...
template <bool SOFT>
__device__ __forceinline__ void direct_sum_unit(const float4 *__restrict__ pi_tile,
                                                const float4 *__restrict__ pj, int plane,
                                                int row0, int split, int g0, int g1, float eps2,
                                                float2 *__restrict__ partial,
                                                unsigned *__restrict__ status, float4 *sj,
                                                uint64_t *full_bar)
{
    const int nj = (g1 - g0) * DS_GRANULE;
    const int ntiles = (nj + DS_JTILE - 1) / DS_JTILE;
    const float4 *src = pj + (size_t)g0 * DS_GRANULE;

    float xi[DS_IPT], yi[DS_IPT], zi[DS_IPT];
#pragma unroll
    for (int k = 0; k < DS_IPT; ++k) {
        const float4 p = pi_tile[k * DS_THREADS + threadIdx.x];
        xi[k] = p.x;
        yi[k] = p.y;
        zi[k] = p.z;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < DS_STAGES; ++s) mbar_init(&full_bar[s], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // tile u: DS_JTILE particles, or what is left (whole granules, so every
    // copy is a multiple of 2 KiB)
    auto fetch = [&](int u) {
        const unsigned bytes = (unsigned)min(DS_JTILE, nj - u * DS_JTILE) * 16u;
        mbar_expect_tx(&full_bar[u % DS_STAGES], bytes);
        bulk_g2s(sj + (u % DS_STAGES) * DS_JTILE, src + (size_t)u * DS_JTILE, bytes,
                 &full_bar[u % DS_STAGES]);
    };
    int issued = min(DS_STAGES, ntiles);
    if (threadIdx.x == 0)
        for (int u = 0; u < issued; ++u) fetch(u);

    float sx[DS_IPT], sy[DS_IPT], sz[DS_IPT], cx[DS_IPT], cy[DS_IPT], cz[DS_IPT];
#pragma unroll
    for (int k = 0; k < DS_IPT; ++k) {
        sx[k] = sy[k] = sz[k] = 0.0f;
        cx[k] = cy[k] = cz[k] = 0.0f;
    }
    static_assert(DS_IPT % 2 == 0, "i-particles are paired");
    float2 nx2[DS_IPT / 2], ny2[DS_IPT / 2], nz2[DS_IPT / 2];
#pragma unroll
    for (int k = 0; k < DS_IPT / 2; ++k) {
        nx2[k] = make_float2(-xi[2 * k], -xi[2 * k + 1]);
        ny2[k] = make_float2(-yi[2 * k], -yi[2 * k + 1]);
        nz2[k] = make_float2(-zi[2 * k], -zi[2 * k + 1]);
    }
    const float2 eps2v = make_float2(eps2, eps2);

    int t = 0;
    for (; t < ntiles; ++t) {
        const int st = t % DS_STAGES;
        const unsigned parity = (unsigned)(t / DS_STAGES) & 1u;
        const bool ready = mbar_wait(&full_bar[st], parity);
        if (!__syncthreads_and(ready)) {
            if (threadIdx.x == 0) atomicOr(status, ST_WAIT_TIMEOUT);
            break;
        }
        const float4 *tile = sj + st * DS_JTILE;
        const int jn = min(DS_JTILE, nj - t * DS_JTILE);
        for (int j0 = 0; j0 < jn; j0 += DS_GRANULE) {
            float2 ax[DS_IPT / 2], ay[DS_IPT / 2], az[DS_IPT / 2];
#pragma unroll
            for (int k = 0; k < DS_IPT / 2; ++k)
                ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
#pragma unroll 8
            for (int j = j0; j < j0 + DS_GRANULE; ++j) {
                const float4 q = tile[j];
#pragma unroll
                for (int k = 0; k < DS_IPT / 2; ++k)
                    pair_term2<SOFT>(q, nx2[k], ny2[k], nz2[k], eps2v, ax[k], ay[k], az[k]);
            }
#pragma unroll
            for (int k = 0; k < DS_IPT / 2; ++k) {
                kahan_add(sx[2 * k], cx[2 * k], ax[k].x);
                kahan_add(sy[2 * k], cy[2 * k], ay[k].x);
                kahan_add(sz[2 * k], cz[2 * k], az[k].x);
                kahan_add(sx[2 * k + 1], cx[2 * k + 1], ax[k].y);
                kahan_add(sy[2 * k + 1], cy[2 * k + 1], ay[k].y);
                kahan_add(sz[2 * k + 1], cz[2 * k + 1], az[k].y);
            }
        }
        __syncthreads();   // every thread is done with stage st
        if (issued < ntiles) {
            if (threadIdx.x == 0) fetch(issued);
            ++issued;
        }
    }
    if (t < ntiles) {
        // Timed out: let copies already issued land before the CTA exits.
        if (threadIdx.x == 0) {
            for (int u = t; u < issued; ++u)
                (void)mbar_wait(&full_bar[u % DS_STAGES], (unsigned)(u / DS_STAGES) & 1u);
        }
        __syncthreads();
        return;
    }

    float2 *out = partial + (size_t)split * 3 * (size_t)plane;
#pragma unroll
    for (int k = 0; k < DS_IPT; ++k) {
        const size_t i = (size_t)row0 + k * DS_THREADS + threadIdx.x;
        out[0 * (size_t)plane + i] = make_float2(sx[k], cx[k]);
        out[1 * (size_t)plane + i] = make_float2(sy[k], cy[k]);
        out[2 * (size_t)plane + i] = make_float2(sz[k], cz[k]);
    }
}

// a + b = sum + err exactly (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float a, float b, float &err)
{
    const float t = __fadd_rn(a, b), v = __fsub_rn(t, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, v)), __fsub_rn(b, v));
    return t;
}

// A unit's Kahan pair (s, c), whose value is s - c, added to the running sum
// h + l + t: h and l exactly, t holds what they leave (72 bits in all).
__device__ __forceinline__ void add_pair(float &h, float &l, float &t, const float2 sc)
{
    float e, f, g;
    h = two_sum(h, sc.x, e);
    l = two_sum(l, two_sum(e, -sc.y, f), g);
    t = __fadd_rn(t, __fadd_rn(f, g));
}

// Work units: unit (itile, split) takes granules [split * per, (split + 1) * per).
template <bool SOFT>
__global__ void __launch_bounds__(DS_THREADS, 2)
k_direct_sum(const float4 *__restrict__ pj, int n_pad, int i_tiles, int per, int granules,
             float eps2, float2 *__restrict__ partial, unsigned *__restrict__ status)
{
    extern __shared__ __align__(128) unsigned char ds_smem[];
    __shared__ __align__(8) uint64_t full_bar[DS_STAGES];
    const int itile = blockIdx.x % i_tiles;
    const int split = blockIdx.x / i_tiles;
    const int row0 = itile * DS_ITILE;
    direct_sum_unit<SOFT>(pj + row0, pj, n_pad, row0, split, split * per,
                          min(granules, (split + 1) * per), eps2, partial, status,
                          reinterpret_cast<float4 *>(ds_smem), full_bar);
}

// Direct sum of a system too small to give every SM units of 1024 rows.  A
// unit is 64 rows (two per lane) by one compensated run of `run` granules: the
// eight warps take a granule each, and the run is then added up in granule order
// from shared memory, so that the Kahan sequence of a row is that of a thread that
// takes the granules one after the other, and the units are small enough to fill
// the GPU (12,000 particles: 2,256 units where units of 1024 x 1024 made 144).
// Two rows per lane beat four and eight at every size (58 against 62 and 63 us at
// N = 12,000): the FP32 pipe has enough warps, and smaller units waste less at the
// end.  With packing and reduction, in a graph: 10.1 us at N = 1,500 (72 before),
// 22 at 6,000, 62.5 at 12,000 (76 before), 159 at 20,000 (k_direct_sum: 164).
template <bool SOFT>
__global__ void __launch_bounds__(DR_THREADS)
k_direct_run(const float4 *__restrict__ pj, int n_pad, int i_tiles, int run, int granules,
             float eps2, float2 *__restrict__ partial, unsigned *__restrict__ status)
{
    __shared__ __align__(128) float4 sj[DS_JTILE];
    __shared__ float part[DR_WARPS][3][DR_ROWS];
    __shared__ __align__(8) uint64_t bar;
    static_assert(DR_WARPS * DS_GRANULE == DS_JTILE && 3 * DR_ROWS <= DR_THREADS,
                  "a granule per warp, a thread per row and component");
    const int itile = blockIdx.x % i_tiles, r = blockIdx.x / i_tiles;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = itile * DR_ROWS;
    const int g0 = r * run, g1 = min(granules, g0 + run);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    const float4 p0 = pj[row0 + lane], p1 = pj[row0 + 32 + lane];
    const float2 nx = make_float2(-p0.x, -p1.x), ny = make_float2(-p0.y, -p1.y),
                 nz = make_float2(-p0.z, -p1.z), e2 = make_float2(eps2, eps2);
    const int e = threadIdx.x;   // this thread's component and row of the run's sums
    float s = 0.0f, c = 0.0f;
    unsigned parity = 0;
    for (int g = g0; g < g1; g += DR_WARPS, parity ^= 1u) {
        const int here = min(DR_WARPS, g1 - g);
        if (threadIdx.x == 0) {
            mbar_expect_tx(&bar, here * DS_GRANULE * 16);
            bulk_g2s(sj, pj + (size_t)g * DS_GRANULE, here * DS_GRANULE * 16, &bar);
        }
        const bool ready = mbar_wait(&bar, parity);
        if (!__syncthreads_and(ready)) {
            if (threadIdx.x == 0) atomicOr(status, ST_WAIT_TIMEOUT);
            // the copy lands before the CTA exits
            if (threadIdx.x == 0) (void)mbar_wait(&bar, parity);
            __syncthreads();
            return;
        }
        if (w < here) {
            float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
            const float4 *tile = sj + w * DS_GRANULE;
#pragma unroll 8
            for (int j = 0; j < DS_GRANULE; ++j) pair_term2<SOFT>(tile[j], nx, ny, nz, e2, ax, ay, az);
            part[w][0][lane] = ax.x;
            part[w][0][32 + lane] = ax.y;
            part[w][1][lane] = ay.x;
            part[w][1][32 + lane] = ay.y;
            part[w][2][lane] = az.x;
            part[w][2][32 + lane] = az.y;
        }
        __syncthreads();
        if (e < 3 * DR_ROWS)
            for (int q = 0; q < here; ++q) kahan_add(s, c, part[q][e / DR_ROWS][e % DR_ROWS]);
        __syncthreads();   // the tile and the partials are free again
    }
    if (e < 3 * DR_ROWS)
        partial[((size_t)r * 3 + e / DR_ROWS) * (size_t)n_pad + row0 + e % DR_ROWS] =
            make_float2(s, c);
}

// Direct sum for a separate list of target particles pi [ni_pad] (padded to
// whole 1024-particle tiles) against all sources pj: the sampled rows of the
// learned method's training targets and per-step judge.
template <bool SOFT>
__global__ void __launch_bounds__(DS_THREADS, 2)
k_direct_rows(const float4 *__restrict__ pi, int ni_pad, const float4 *__restrict__ pj,
              int i_tiles, int per, int granules, float eps2, float2 *__restrict__ partial,
              unsigned *__restrict__ status)
{
    extern __shared__ __align__(128) unsigned char ds_smem[];
    __shared__ __align__(8) uint64_t full_bar[DS_STAGES];
    const int itile = blockIdx.x % i_tiles;
    const int split = blockIdx.x / i_tiles;
    const int row0 = itile * DS_ITILE;
    direct_sum_unit<SOFT>(pi + row0, pj, ni_pad, row0, split, split * per,
                          min(granules, (split + 1) * per), eps2, partial, status,
                          reinterpret_cast<float4 *>(ds_smem), full_bar);
}

// Sum over the splits, in split order, of component k of row i: in FP32 with the
// rounding errors kept, which is an FP64 sum's precision and more.  FP64
// conversions and adds cost a whole warp's time on a pipe of 1/64 of the FP32 rate:
// 72 of them per thread in a unit's epilogue took 4 us of a 65 us launch at
// N = 12,000.  A sum that leaves the FP32 range (or is not finite) is one of FP64.
__device__ __forceinline__ double reduce_row(const float2 *__restrict__ partial, int splits,
                                             size_t plane, int k, int i)
{
    const float2 *p = partial + k * plane + i;
    float h = 0.0f, l = 0.0f, t = 0.0f;
#pragma unroll 8
    for (int q = 0; q < splits; ++q) add_pair(h, l, t, p[(size_t)q * 3 * plane]);
    const double sum = (double)h + ((double)l + (double)t);
    if (finite_bits(sum)) return sum;
    double wide = 0.0;
#pragma unroll 1
    for (int q = 0; q < splits; ++q) {
        const float2 sc = p[(size_t)q * 3 * plane];
        wide += (double)sc.x - (double)sc.y;
    }
    return wide;
}

// a_i = G * sum_s partial[s][.][i]; a thread per component.
__global__ void k_reduce_splits(const float2 *__restrict__ partial, int splits, int n,
                                int n_pad, double G, double *__restrict__ a, Kick kick)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (i < n)
        store_and_kick(a, 3 * (size_t)i + k, G * reduce_row(partial, splits, n_pad, k, i), kick);
}

// FP64, reference operation order (see file comment).  A CTA of eight warps,
// two per SM sub-partition, owns P particles.  For 128 consecutive j the warps
// form the pair terms of the P particles (each term is independent; a warp takes
// 32 j of one particle at a time); then lane 3p + c of warp 0 subtracts the
// component-c terms of particle p from its accumulator one by one in j order,
// which is the order the reference's loop adds them to a_i, while the other warps
// form the next 128.  (The own term and those past the end are +0, which leave
// the accumulator as it is.)
//
// An FP64 instruction holds its sub-partition for 64 cycles whatever its lanes
// do, so the time is the instructions of the busiest one: 32 per 32 terms and one
// per j for the ordered sums of all P particles.  With a warp per particle the
// ordered sums, three lanes wide, took as many instructions as the terms; the
// shares below make the four sub-partitions' counts equal, 32 (P + 1) per round.
// Leapfrog step: N = 1,024 163 -> 91 us, 4,096 2.13 -> 1.15 ms, 33,000 81 -> 74 ms.
constexpr int RF_THREADS = 256;             // two warps per sub-partition
constexpr int RF_CHUNK = 128;              // j per round
constexpr int RF_ROW = RF_CHUNK + 1;       // stride of a component's terms (bank spread)
constexpr int RF_MAX_P = 10;               // 30 lanes of ordered sums

__host__ __device__ constexpr size_t rf_smem(int P)
{
    return ((size_t)2 * 3 * P * RF_ROW + 3 * RF_MAX_P) * sizeof(double);
}

__global__ void __launch_bounds__(RF_THREADS)
k_direct_fp64_reference_order(const double *__restrict__ x, const double *__restrict__ m,
                              int n, int P, double G, double eps2, double *__restrict__ a,
                              Kick kick)
{
    extern __shared__ __align__(16) double rf_terms[];   // [2][3 P][RF_ROW], then x_i
    double *xi = rf_terms + 2 * 3 * P * RF_ROW;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * P;
    const int np = min(P, n - i0);
    if (threadIdx.x < 3 * np) xi[threadIdx.x] = x[3 * (size_t)i0 + threadIdx.x];
    __syncthreads();
    // items of a round: (32 j, particle), particles fastest; the sub-partition of
    // warp 0, which adds, takes np - 3 of the 4 np (warp 4), the others np + 1 each
    const int own = max(0, np - 3);
    const int per = (4 * np - own + 2) / 3;
    const int sub = w & 3;
    int e0 = sub == 0 ? 0 : min(4 * np, own + (sub - 1) * per);
    int e1 = sub == 0 ? own : min(4 * np, e0 + per);
    const int half = sub == 0 ? e0 : e0 + (e1 - e0 + 1) / 2;
    (w < 4 ? e1 : e0) = half;
    auto produce = [&](int chunk) {
        double *buf = rf_terms + (chunk & 1) * 3 * P * RF_ROW;
        int quarter = -1, j = 0;
        double xj0 = 0.0, xj1 = 0.0, xj2 = 0.0, mj = 0.0;
        for (int e = e0; e < e1; ++e) {
            const int q = e / np, p = e - q * np;
            if (q != quarter) {
                quarter = q;
                j = chunk * RF_CHUNK + q * 32 + lane;
                if (j < n) {
                    xj0 = x[3 * (size_t)j + 0];
                    xj1 = x[3 * (size_t)j + 1];
                    xj2 = x[3 * (size_t)j + 2];
                    mj = m[j];
                }
            }
            double t0 = 0.0, t1 = 0.0, t2 = 0.0;
            if (j < n && j != i0 + p) {
                const double r0 = __dsub_rn(xi[3 * p + 0], xj0);
                const double r1 = __dsub_rn(xi[3 * p + 1], xj1);
                const double r2 = __dsub_rn(xi[3 * p + 2], xj2);
                const double s = __dadd_rn(
                    __dadd_rn(__dadd_rn(__dmul_rn(r0, r0), __dmul_rn(r1, r1)), __dmul_rn(r2, r2)),
                    eps2);
                const double rn = __dsqrt_rn(s);
                const double t = __ddiv_rn(G, __dmul_rn(__dmul_rn(rn, rn), rn));
                t0 = __dmul_rn(__dmul_rn(t, r0), mj);
                t1 = __dmul_rn(__dmul_rn(t, r1), mj);
                t2 = __dmul_rn(__dmul_rn(t, r2), mj);
            }
            double *out = buf + 3 * p * RF_ROW + q * 32 + lane;
            out[0] = t0;
            out[RF_ROW] = t1;
            out[2 * RF_ROW] = t2;
        }
    };
    const int chunks = (n + RF_CHUNK - 1) / RF_CHUNK;
    double acc = 0.0;   // lane 3p + c < 3 np of warp 0: component c of a_(i0 + p)
    produce(0);
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
        if (w == 0 && lane < 3 * np) {
            const double *tc = rf_terms + ((c & 1) * 3 * P + lane) * RF_ROW;
            const int cnt = min(RF_CHUNK, n - c * RF_CHUNK);
#pragma unroll 16
            for (int q = 0; q < cnt; ++q) acc = __dsub_rn(acc, tc[q]);
        }
        __syncwarp();
        if (c + 1 < chunks) produce(c + 1);
        __syncthreads();
    }
    if (w == 0 && lane < 3 * np) store_and_kick(a, 3 * (size_t)i0 + lane, acc, kick);
}

// ------------------------------------------------------------------------
namespace {

// Granules per unit of a direct sum: the row tiles' granules are divided by the
// time a unit takes.  Whole waves of resident CTAs take a unit each; in the last,
// partial wave an SM whose slots are not all taken gives the CTAs it has a larger
// share of its pipes, so a wave that is a quarter full costs less than a full one.
// A unit is charged 0.15 granules to start and end; every split adds the traffic
// of its partial sums (48 bytes a row, written and read) where it has its own.
// One granule of a full wave takes 13.9 us, and this form follows the sweep of 1
// to 64 splits at N = 12,000 to 100,000 within 3 %.  (Counting whole waves only
// took 232 us instead of 220 at N = 24,000.)
int choose_per(int i_tiles, int granules, int per_sm, long slots, double split_cost)
{
    int best_per = granules;
    double best = 1e300;
    for (int s = 1; s <= std::min(granules, 64); ++s) {
        const int per = (granules + s - 1) / s;
        const int used = (granules + per - 1) / per;
        const long units = (long)i_tiles * used;
        const long left = units % slots;
        const double filled = std::ceil((double)left / (double)slots * per_sm) / per_sm;
        const double waves = (double)(units / slots) + (left ? 0.1 + 0.9 * filled : 0.0);
        const double cost = waves * (0.5 * (per + (double)granules / used) + 0.15) + split_cost * used;
        if (cost < best - 1e-9) {
            best = cost;
            best_per = per;
        }
    }
    return best_per;
}

// Splits and source tiles per split where a unit takes whole tiles: the whole
// number of waves that needs the fewest tiles per CTA.
void choose_tiles(int i_tiles, int tiles, long slots, int max_splits, int *splits, int *chunk)
{
    double best = 1e300;
    for (int s = 1; s <= std::min(tiles, max_splits); ++s) {
        const int c = (tiles + s - 1) / s;
        const int used = (tiles + c - 1) / c;
        const double cost = (double)(((long)i_tiles * used + slots - 1) / slots) * (c + 0.25);
        if (cost < best - 1e-9) {
            best = cost;
            *splits = used;
            *chunk = c;
        }
    }
}

// Resident CTAs of a kernel on the current device.
template <class Kernel>
ErrorStatus resident_ctas(Kernel kernel, int *per_sm)
{
    GS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM));
    GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, DS_THREADS, DS_SMEM));
    *per_sm = std::max(*per_sm, 1);
    return ok();
}

class DirectEngine final : public Engine {
  public:
    explicit DirectEngine(bool fp64) : fp64_(fp64) {}

    ErrorStatus setup(int n, double G, const AccelerationParam &p) override
    {
        n_ = n;
        G_ = G;
        eps_ = p.softening_length;
        const DeviceInfo *dev = nullptr;
        GS_TRY(device_info(&dev));
        if (fp64_) {
            // particles per CTA: the fewest instructions of the busiest SM.  Per round
            // of 128 j and CTA, in units of 32: P + 1 (four at least, the ordered sums
            // alone), and once the first round's terms, on three warps.
            const long rounds = (n + RF_CHUNK - 1) / RF_CHUNK;
            long best = 0;
            for (int P = 1; P <= RF_MAX_P; ++P) {
                const long ctas = (n + P - 1) / P;
                const long first = (4 * P - std::max(0, P - 3) + 2) / 3;
                const long cost = (ctas + dev->sm_count - 1) / dev->sm_count *
                                  (rounds * std::max(4, P + 1) + first);
                if (best == 0 || cost <= best) {
                    best = cost;
                    p_ = P;
                }
            }
            GS_CUDA(cudaFuncSetAttribute(k_direct_fp64_reference_order,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)rf_smem(RF_MAX_P)));
            return ok();
        }
        n_pad_ = ((n + DS_ITILE - 1) / DS_ITILE) * DS_ITILE;
        granules_ = (n + DS_GRANULE - 1) / DS_GRANULE;
        if (n <= DS_RUN_N) {
            // Compensated runs of 1,024 terms; of 2,048 from 17,409 particles on,
            // where both take the same time and half the partial sums are stored.
            // Leapfrog step with runs of 1,024 and 2,048: N = 12,000 68.3 and 72.4 us,
            // 16,000 110 and 115, 17,000 121.9 and 121.6, 18,000 136 and 137, 19,000
            // 150 and 149, 20,480 173 and 175.
            per_ = (n <= 17 * DS_JTILE ? 1 : 2) * DS_TILE_GRANULES;
            i_tiles_ = (n + DR_ROWS - 1) / DR_ROWS;
        } else {
            int per_sm = 1;
            GS_TRY(resident_ctas(k_direct_sum<true>, &per_sm));
            GS_TRY(resident_ctas(k_direct_sum<false>, &per_sm));
            i_tiles_ = n_pad_ / DS_ITILE;
            per_ = choose_per(i_tiles_, granules_, per_sm, (long)dev->sm_count * per_sm, 7e-7 * n);
        }
        splits_ = (granules_ + per_ - 1) / per_;
        GS_TRY(pj_.reserve((size_t)n_pad_ * sizeof(float4)));
        GS_TRY(partial_.reserve((size_t)splits_ * 3 * n_pad_ * sizeof(float2)));
        GS_TRY(status_.reserve(sizeof(unsigned)));
        GS_CUDA(cudaMemset(status_.p, 0, sizeof(unsigned)));
        return ok();
    }

    void set_frame_centre(double cx, double cy, double cz) override
    {
        c_[0] = cx;
        c_[1] = cy;
        c_[2] = cz;
    }

    ErrorStatus compute(const double *d_x, const double *d_m, double *d_a, cudaStream_t s,
                        ForceTimer *timer) override
    {
        // without a drift k_pack_float4 only reads the positions
        const StepState q = {const_cast<double *>(d_x), nullptr, nullptr, nullptr, n_};
        return forces(q, d_m, d_a, 0.0, s, timer);
    }

    // Drift inside the packing kernel, kick inside the reduction (FP64: the force
    // kernel): three launches a step instead of five, two instead of three.
    // A step of 1,000 particles takes 15.4 us instead of 17.5, of 8,000 42.6 instead
    // of 45.1, of 1,024 in FP64 88.7 instead of 90.6.
    ErrorStatus leapfrog(const StepState &q, const double *d_m, double *d_a, double h,
                         cudaStream_t s, ForceTimer *timer) override
    {
        if (fp64_) launch_comp_update(q.x, q.xe, q.v, h, 1.0, 3 * q.n, s);
        return forces(q, d_m, d_a, h, s, timer);
    }

    int kernels_per_eval() const override { return fp64_ ? 1 : 3; }
    int kernels_per_leapfrog() const override { return fp64_ ? 2 : 3; }

  private:
    // Accelerations at q.x; with q.v, after its drift (FP32 only) and before its kick.
    ErrorStatus forces(const StepState &q, const double *d_m, double *d_a, double h, cudaStream_t s,
                       ForceTimer *timer)
    {
        const Kick kick = {q.v, q.ve, h};
        if (fp64_) {
            if (timer) GS_TRY(timer->begin(s));
            k_direct_fp64_reference_order<<<(n_ + p_ - 1) / p_, RF_THREADS, rf_smem(p_), s>>>(
                q.x, d_m, n_, p_, G_, eps_ * eps_, d_a, kick);
            GS_CUDA(cudaGetLastError());
            if (timer) GS_TRY(timer->end(s));
            return ok();
        }
        const float eps2 = (float)(eps_ * eps_);
        const int grid = i_tiles_ * splits_;
        const bool soft = eps2 > 0.0f;
        k_pack_float4<<<(n_pad_ + 127) / 128, 128, 0, s>>>(q.x, d_m, n_, n_pad_, c_[0], c_[1], c_[2],
                                                           q.xe, q.v, h, pj_.as<float4>());
        GS_CUDA(cudaGetLastError());
        if (timer) GS_TRY(timer->begin(s));
        if (n_ <= DS_RUN_N) {
            auto run = soft ? k_direct_run<true> : k_direct_run<false>;
            run<<<grid, DR_THREADS, 0, s>>>(pj_.as<float4>(), n_pad_, i_tiles_, per_, granules_, eps2,
                                            partial_.as<float2>(), status_.as<unsigned>());
        } else {
            auto sum = soft ? k_direct_sum<true> : k_direct_sum<false>;
            sum<<<grid, DS_THREADS, DS_SMEM, s>>>(pj_.as<float4>(), n_pad_, i_tiles_, per_, granules_,
                                                  eps2, partial_.as<float2>(),
                                                  status_.as<unsigned>());
        }
        GS_CUDA(cudaGetLastError());
        if (timer) GS_TRY(timer->end(s));
        k_reduce_splits<<<dim3((n_ + 127) / 128, 3), 128, 0, s>>>(partial_.as<float2>(), splits_, n_,
                                                                  n_pad_, G_, d_a, kick);
        GS_CUDA(cudaGetLastError());
        return ok();
    }

  public:
    ErrorStatus check_status(cudaStream_t s) override
    {
        if (fp64_) return ok();
        unsigned h = 0;
        GS_CUDA(cudaMemcpyAsync(&h, status_.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        GS_CUDA(cudaStreamSynchronize(s));
        if (h & ST_WAIT_TIMEOUT)
            return GS_RAISE(GRAV_FAILURE, "direct-sum kernel: shared-memory tile wait timed out");
        return ok();
    }

  private:
    bool fp64_;
    int p_ = 1;   // particles per CTA of the FP64 kernel
    int n_ = 0, n_pad_ = 0, i_tiles_ = 0, granules_ = 1, per_ = 1, splits_ = 1;
    double G_ = 1.0, eps_ = 0.0;
    double c_[3] = {0.0, 0.0, 0.0};
    DBuf pj_, partial_, status_;
};

}  // namespace

std::unique_ptr<Engine> make_direct_engine(bool fp64_reference_order)
{
    return std::unique_ptr<Engine>(new DirectEngine(fp64_reference_order));
}

// ---- direct sum over selected rows ----------------------------------------
// Sources packed relative to frame[0..2] (a device FP64 centre).
__global__ void k_pack_frame(const double *__restrict__ x, const double *__restrict__ m, int n,
                             int n_pad, const double *__restrict__ frame, float4 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    float4 p;
    if (i < n) {
        p.x = (float)(x[3 * i + 0] - frame[0]);
        p.y = (float)(x[3 * i + 1] - frame[1]);
        p.z = (float)(x[3 * i + 2] - frame[2]);
        p.w = (float)m[i];
    } else {
        p = make_float4(kPadPos, kPadPos, kPadPos, 0.0f);
    }
    out[i] = p;
}

__global__ void k_gather_rows(const float4 *__restrict__ pj, const int *__restrict__ rows,
                              int nrows, int nrows_pad, float4 *__restrict__ pi)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows_pad) return;
    pi[r] = r < nrows ? pj[rows[r]] : make_float4(kPadPos, kPadPos, kPadPos, 0.0f);
}

ErrorStatus DirectRows::setup(int nj, int max_rows)
{
    const DeviceInfo *dev = nullptr;
    GS_TRY(device_info(&dev));
    nj_ = nj;
    nj_pad_ = ((nj + DS_JTILE - 1) / DS_JTILE) * DS_JTILE;
    jt_total_ = nj_pad_ / DS_JTILE;
    ni_pad_ = ((max_rows + DS_ITILE - 1) / DS_ITILE) * DS_ITILE;
    int per_sm = 1;
    GS_TRY(resident_ctas(k_direct_rows<false>, &per_sm));
    GS_TRY(resident_ctas(k_direct_rows<true>, &per_sm));
    slots_ = (long)dev->sm_count * per_sm;
    // Partial sums sized for the largest launch and for a launch of a single
    // row tile, which splits the j range most finely.
    const int i_tiles = ni_pad_ / DS_ITILE;
    int sp = 1, ch = 1;
    choose_tiles(i_tiles, jt_total_, slots_, 128, &sp, &ch);
    partial_rows_ = (size_t)sp * ni_pad_;
    choose_tiles(1, jt_total_, slots_, 128, &sp, &ch);
    partial_rows_ = std::max(partial_rows_, (size_t)sp * DS_ITILE);
    GS_TRY(pj_.reserve((size_t)nj_pad_ * sizeof(float4)));
    GS_TRY(pi_.reserve((size_t)ni_pad_ * sizeof(float4)));
    GS_TRY(partial_.reserve(partial_rows_ * 3 * sizeof(float2)));
    GS_TRY(status_.reserve(sizeof(unsigned)));
    GS_CUDA(cudaMemset(status_.p, 0, sizeof(unsigned)));
    return ok();
}

ErrorStatus DirectRows::compute(const double *d_x, const double *d_m, const double *d_frame,
                                const int *d_rows, int nrows, double G, double eps, double *d_a_rows,
                                cudaStream_t s, ForceTimer *timer)
{
    if (nrows <= 0) return ok();
    if (((nrows + DS_ITILE - 1) / DS_ITILE) * DS_ITILE > ni_pad_)
        return GS_RAISE(GRAV_VALUE_ERROR, "direct rows: %d rows exceed the prepared %d", nrows, ni_pad_);
    k_pack_frame<<<(nj_pad_ + 255) / 256, 256, 0, s>>>(d_x, d_m, nj_, nj_pad_, d_frame,
                                                       pj_.as<float4>());
    const int nr_pad = ((nrows + DS_ITILE - 1) / DS_ITILE) * DS_ITILE;
    k_gather_rows<<<(nr_pad + 255) / 256, 256, 0, s>>>(pj_.as<float4>(), d_rows, nrows, nr_pad,
                                                       pi_.as<float4>());
    const float eps2 = (float)(eps * eps);
    const int i_tiles = nr_pad / DS_ITILE;
    // the split is chosen for this launch's row count (few rows: many
    // j-chunks, so that the launch still fills every SM)
    int splits = 1, chunk = jt_total_;
    choose_tiles(i_tiles, jt_total_, slots_, (int)std::min<size_t>(128, partial_rows_ / nr_pad),
                 &splits, &chunk);
    auto kernel = eps2 > 0.0f ? k_direct_rows<true> : k_direct_rows<false>;
    if (timer) GS_TRY(timer->begin(s));
    kernel<<<i_tiles * splits, DS_THREADS, DS_SMEM, s>>>(
        pi_.as<float4>(), nr_pad, pj_.as<float4>(), i_tiles, chunk * DS_TILE_GRANULES,
        jt_total_ * DS_TILE_GRANULES, eps2, partial_.as<float2>(), status_.as<unsigned>());
    GS_CUDA(cudaGetLastError());
    if (timer) GS_TRY(timer->end(s));
    k_reduce_splits<<<dim3((nrows + 255) / 256, 3), 256, 0, s>>>(partial_.as<float2>(), splits,
                                                                 nrows, nr_pad, G, d_a_rows,
                                                                 Kick{nullptr, nullptr, 0.0});
    GS_CUDA(cudaGetLastError());
    return ok();
}

ErrorStatus DirectRows::check(cudaStream_t s)
{
    unsigned h = 0;
    GS_CUDA(cudaMemcpyAsync(&h, status_.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    GS_CUDA(cudaStreamSynchronize(s));
    if (h) {
        GS_CUDA(cudaMemsetAsync(status_.p, 0, sizeof(unsigned), s));
        if (h & ST_WAIT_TIMEOUT)
            return GS_RAISE(GRAV_FAILURE, "direct-sum rows kernel: shared-memory tile wait timed out");
    }
    return ok();
}

// ------------------------------------------------------------------------
// Allocation-free compensated-FP32 direct sum.
//
// For callers that cannot allocate device memory while they run: code that
// records or replays a fixed plan of work and may not call cudaMalloc
// (which can synchronise the device) in the middle of it, embedders whose
// allocator is a pool they own, and real-time loops that must not touch the
// allocator at all.  This entry point computes the accelerations of
// acceleration() with GRAV_GPU_PAIRWISE, from device arrays the caller
// owns, to the same accuracy: the pair terms are the same, but the work is
// always k_direct_sum's, in at most NOALLOC_MAX_SPLITS units of whole tiles per
// row, so the compensated partial sums are grouped otherwise and last bits
// differ, and small systems take longer.  Its scratch (the packed float4 particles,
// the per-split partial sums, the status word and the frame centre) lives
// in one file-scope device array instead of memory the library allocates.
// That array is part of the library image: every GPU that loads the library
// holds its NOALLOC_BYTES (about 6.5 MiB) until the process exits.
//
// Like acceleration(), it takes positions relative to the centre of their
// bounding box before rounding them to FP32; here that centre is reduced on
// the device (k_noalloc_frame) into the scratch array, so that systems far
// from the origin keep their accuracy.  A bulk-copy wait that runs out in
// k_direct_sum sets the status word, and the reduction then writes NaN into
// every output row instead of partial sums.
constexpr int NOALLOC_MAX_N = 32768;      // largest particle count accepted
constexpr int NOALLOC_MAX_SPLITS = 8;
constexpr size_t NOALLOC_PJ_BYTES = (size_t)NOALLOC_MAX_N * sizeof(float4);
constexpr size_t NOALLOC_PARTIAL_BYTES =
    (size_t)NOALLOC_MAX_SPLITS * 3 * NOALLOC_MAX_N * sizeof(float2);
constexpr size_t NOALLOC_BYTES = NOALLOC_PJ_BYTES + NOALLOC_PARTIAL_BYTES + 256;
static_assert(NOALLOC_MAX_N % DS_JTILE == 0, "capacity must be whole tiles");
// The last 256 bytes: the status word at offset 0, the FP64 frame centre at 64.
constexpr size_t NOALLOC_STATUS_OFF = NOALLOC_PJ_BYTES + NOALLOC_PARTIAL_BYTES;
constexpr size_t NOALLOC_FRAME_OFF = NOALLOC_STATUS_OFF + 64;
static_assert(NOALLOC_FRAME_OFF + 3 * sizeof(double) <= NOALLOC_BYTES, "tail holds the frame");

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

// Centre of the bounding box of x [n] (one CTA), formed as acceleration()
// forms it on the host: per axis the exact minimum and maximum, then
// 0.5 (lo + hi).
constexpr int NA_FRAME_THREADS = 1024;
__global__ void __launch_bounds__(NA_FRAME_THREADS)
k_noalloc_frame(const double *__restrict__ x, int n, double *__restrict__ frame)
{
    __shared__ double lo_s[3][NA_FRAME_THREADS / 32], hi_s[3][NA_FRAME_THREADS / 32];
    double lo[3] = {x[0], x[1], x[2]}, hi[3] = {x[0], x[1], x[2]};
    for (int i = threadIdx.x; i < n; i += NA_FRAME_THREADS)
        for (int k = 0; k < 3; ++k) {
            const double q = x[3 * i + k];
            lo[k] = q < lo[k] ? q : lo[k];
            hi[k] = q > hi[k] ? q : hi[k];
        }
    for (int k = 0; k < 3; ++k)
        for (int o = 16; o > 0; o >>= 1) {
            const double l = __shfl_xor_sync(0xffffffffu, lo[k], o);
            const double h = __shfl_xor_sync(0xffffffffu, hi[k], o);
            lo[k] = l < lo[k] ? l : lo[k];
            hi[k] = h > hi[k] ? h : hi[k];
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; ++k) {
            lo_s[k][w] = lo[k];
            hi_s[k][w] = hi[k];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        double l = lo_s[k][0], h = hi_s[k][0];
        for (int v = 1; v < NA_FRAME_THREADS / 32; ++v) {
            l = lo_s[k][v] < l ? lo_s[k][v] : l;
            h = hi_s[k][v] > h ? hi_s[k][v] : h;
        }
        frame[k] = 0.5 * (l + h);
    }
}

// k_reduce_splits for this entry point: when a tile wait of k_direct_sum
// ran out (status bit ST_WAIT_TIMEOUT), some partial sums were never
// written, and every row gets NaN instead of a wrong finite value.
__global__ void k_noalloc_reduce(const float2 *__restrict__ partial, int splits, int n, int n_pad,
                                 double G, const unsigned *__restrict__ status,
                                 double *__restrict__ a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (i >= n) return;
    a[3 * i + k] = (*status & ST_WAIT_TIMEOUT) ? __longlong_as_double(0x7ff8000000000000LL)
                                               : G * reduce_row(partial, splits, n_pad, k, i);
}

namespace {

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// Device address of the scratch array on the current device.  On a host
// `g_noalloc_scratch` only names a host-side stand-in for the symbol, so
// its address is looked up once per device (with that device current) by
// cudaGetSymbolAddress, which allocates nothing.
cudaError_t noalloc_scratch(void **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return cudaSuccess;
}

}  // namespace

}  // namespace gs

extern "C" int gsgpu_pairwise_acceleration_noalloc(const double *d_x, const double *d_m,
                                                   int num_particles, double G,
                                                   double softening_length, double *d_a,
                                                   void *stream)
{
    using namespace gs;
    if (!d_x || !d_m || !d_a) {
        std::fprintf(stderr, "gsgpu_pairwise_acceleration_noalloc: NULL array argument\n");
        return GRAV_POINTER_ERROR;
    }
    if (num_particles < 1 || num_particles > NOALLOC_MAX_N) {
        std::fprintf(stderr,
                     "gsgpu_pairwise_acceleration_noalloc: num_particles must be in [1, %d] "
                     "(the fixed scratch capacity). Got: %d\n",
                     NOALLOC_MAX_N, num_particles);
        return GRAV_VALUE_ERROR;
    }
    if (!(softening_length >= 0.0)) {
        std::fprintf(stderr, "gsgpu_pairwise_acceleration_noalloc: Softening length is "
                             "negative. Got: %.3g\n", softening_length);
        return GRAV_VALUE_ERROR;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    void *base = nullptr;
    cudaError_t e = noalloc_scratch(&base);
    int dev = 0, sms = 0, per_sm = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const float eps2 = (float)(softening_length * softening_length);
    auto kernel = eps2 > 0.0f ? k_direct_sum<true> : k_direct_sum<false>;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, DS_THREADS, DS_SMEM);
    if (e != cudaSuccess) {
        std::fprintf(stderr, "gsgpu_pairwise_acceleration_noalloc: %s\n", cudaGetErrorString(e));
        return GRAV_FAILURE;
    }
    unsigned char *scratch = static_cast<unsigned char *>(base);
    float4 *pj = reinterpret_cast<float4 *>(scratch);
    float2 *partial = reinterpret_cast<float2 *>(scratch + NOALLOC_PJ_BYTES);
    unsigned *status = reinterpret_cast<unsigned *>(scratch + NOALLOC_STATUS_OFF);
    double *frame = reinterpret_cast<double *>(scratch + NOALLOC_FRAME_OFF);

    // Units of whole source tiles, at most NOALLOC_MAX_SPLITS of them per row.
    const int n_pad = ((num_particles + DS_JTILE - 1) / DS_JTILE) * DS_JTILE;
    const int i_tiles = n_pad / DS_ITILE;
    const int jt_total = n_pad / DS_JTILE;
    const long slots = (long)sms * (per_sm > 0 ? per_sm : 1);
    int splits = 1, chunk = jt_total;
    choose_tiles(i_tiles, jt_total, slots, NOALLOC_MAX_SPLITS, &splits, &chunk);

    // The status word must start at zero; the frame centre, the packed array
    // and the partial sums are fully rewritten by every call.
    e = cudaMemsetAsync(status, 0, sizeof(unsigned), s);
    if (e == cudaSuccess) {
        k_noalloc_frame<<<1, NA_FRAME_THREADS, 0, s>>>(d_x, num_particles, frame);
        k_pack_frame<<<(n_pad + 255) / 256, 256, 0, s>>>(d_x, d_m, num_particles, n_pad, frame,
                                                         pj);
        kernel<<<i_tiles * splits, DS_THREADS, DS_SMEM, s>>>(
            pj, n_pad, i_tiles, chunk * DS_TILE_GRANULES, jt_total * DS_TILE_GRANULES, eps2,
            partial, status);
        k_noalloc_reduce<<<dim3((num_particles + 255) / 256, 3), 256, 0, s>>>(
            partial, splits, num_particles, n_pad, G, status, d_a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        std::fprintf(stderr, "gsgpu_pairwise_acceleration_noalloc: %s\n", cudaGetErrorString(e));
        return GRAV_FAILURE;
    }
    return GRAV_SUCCESS;
}
