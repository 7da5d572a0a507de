// k_walk_group.cu -- group Barnes-Hut walk with interaction lists
// (GRAV_GPU_BARNES_HUT_GROUP).
//
// The per-particle walk of k_walk.cu reproduces the reference's decisions
// (src/acceleration_barnes_hut.c:78-248) one child at a time, which costs
// about 200 instructions per accepted cell.  This walk trades identical
// decisions for throughput:
//   * groups come from the tree: in a cell with more than 32 particles,
//     each run of consecutive children of at most 32 particles is cut into
//     pieces of 32 sorted particles (a leaf with more is cut the same way),
//     so a group lies in one cell and its box stays compact where the
//     Morton curve jumps, and groups fill the lanes;
//     the one group that does not fit its cell (the particles whose Morton
//     coordinate wraps at the box maximum) is walked particle by particle;
//   * a persistent warp (or, with few groups, a CTA) takes groups from a work
//     queue and walks the tree once per group with the group opening criterion
//         accept node  <=>  the node holds none of the group's particles
//                           (sorted ranges disjoint) and
//                           side^2 < theta^2 * dist(com, group box)^2,
//     which implies the per-particle criterion side^2 < theta^2 |com - x|^2
//     of the reference for every particle of the group, so the accepted
//     cells are at least as well separated as the reference's.  The stack
//     holds opened nodes, and a warp's step tests the children of four of
//     them, eight lanes for each (7.4 of 8 have a node): a push is one store;
//   * accepted cells (centre of mass, mass, traceless quadrupole) and the
//     particles of opened leaves go to interaction lists in shared memory
//     (structure of arrays); when a list is full the group's particles are
//     evaluated against it, two entries at a time through paired FP32
//     operations on float2.  A lane holds two of the particles and takes every
//     second pair of entries, so that a shared load serves two particles (a
//     broadcast 16-byte load costs the shared-memory pipe four cycles, and five
//     of them per pair and particle are 1.25 times the pair's FP32 cycles) and
//     a group of at most 16 does no work for the empty row.  The partial sums
//     go to Kahan-compensated accumulators;
//   * coordinates are FP32 offsets from the group's first particle, formed
//     from the frame-centred double-float (hi, lo) copies of the tree, so
//     near-field differences keep FP32 relative accuracy.
// Bound: the FP32 pipe (31 paired operations per pair of quadrupole cells).  One
// walk of the galaxy pair, theta = 0.5, before and after two particles a lane,
// the stack of opened nodes and the team of warps: 1,048,576 particles 3.91 and
// 3.55 ms (FP32 pipe 58 and 62 % busy: four warps per scheduler alternate
// between lists and traversal, whose chains of dependent instructions fill the
// rest); 60,000 particles 341 and 255 us.
// Waits are __syncwarp and __syncthreads with team-uniform conditions only; a
// traversal stack that would overflow sets ST_STACK_OVERFLOW and ends the
// group's walk (no spin, no trap).
#include "gs_octree.h"
#include "gs_ptx.cuh"

#include <atomic>

namespace gs {

constexpr int GW_WARPS = 4;        // warps per CTA
// CTAs per SM.  Four hold 117 registers a thread without spills; with five (96
// registers) a step of 1,048,576 particles took the same time and one of 60,000
// 7 % more.
constexpr int GW_CTAS = 4;
constexpr int GW_STACK = 384;      // traversal stack entries per warp
constexpr int GW_CELLS = 128;      // cell list capacity per warp (64: 2 % slower)
constexpr int GW_PARTS = 128;      // particle list entries evaluated at a time
constexpr int GW_UNROLL = 2;       // turns of an evaluation loop in flight
// Below this many groups per warp of the grid a CTA walks each group together:
// with few groups the time is that of the slowest one.  Step of a galaxy pair,
// a warp and a CTA per group: 5,000 particles 412 and 332 us, 20,000 517 and
// 407, 60,000 (1.0 groups per warp) 574 and 552, 100,000 (1.7) 703 and 705,
// 150,000 887 and 939, 1,048,576 4182 and 5062 (the barriers of a step).
constexpr double GW_TEAM = 1.5;
constexpr int GW_ROWS = 2;         // particles per lane
constexpr int GW_COLS = 32 / GW_ROWS;
// Stack entries kept free for a depth-first descent: popping one node's
// children and pushing those (at most 8) that are opened grows the stack by 7
// per level, over at most OCT_MAX_LEVEL + 1 levels.  Pops shrink so that the
// stack never passes GW_STACK - GW_RESERVE before such a descent starts, hence
// never overflows.
constexpr int GW_RESERVE = 8 * (OCT_MAX_LEVEL + 1);

constexpr int GW_GROUP = 32;       // particles per group at most

// Whether the particles of [first, first + count) lie within the side of a
// depth-`depth` cell, from their positions.
__device__ bool group_extent_fits(int first, int count, int depth, const float4 *__restrict__ pa,
                                  const float4 *__restrict__ pb, double box_length)
{
    const float4 oh = pa[first], ol = pb[first];
    float lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
#pragma unroll 8
    for (int p = first + 1; p < first + count; ++p) {
        const float4 ph = pa[p], pl = pb[p];
        const float r[3] = {(ph.x - oh.x) + (pl.x - ol.x), (ph.y - oh.y) + (pl.y - ol.y),
                            (ph.z - oh.z) + (pl.z - ol.z)};
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], r[k]);
            hi[k] = fmaxf(hi[k], r[k]);
        }
    }
    const float ext = fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
    const double side = box_length / (double)(2 << min(depth, OCT_MAX_LEVEL + 1));
    return (double)ext * (double)ext <= 1.0001 * side * side;
}

// Group list: one thread per internal node.  A cell with more than GW_GROUP
// particles cuts each run of consecutive children of at most GW_GROUP
// particles into pieces of GW_GROUP (a leaf with more is cut the same way);
// the root is one group when it is small enough.  Entry: (first sorted particle,
// count).  A group whose particles do not fit within the side of its cell (the
// particles whose Morton coordinate wraps at the box maximum sit in a cell
// on the far side) goes to the list as single particles, so that no warp
// walks a box-wide group and its walks spread over the warps.
//
// A group's particles lie in one key cell, so it fits the cell's side unless
// it holds a particle whose key cell is not where it is (misplaced).  With at
// most kMisplacedCap of those (their sorted positions in mlist), only a group
// that holds one has its extent measured; the others fit without reading
// their particles.  With more, every group is measured.
//
// Internal nodes come in depth-first pre-order and a block's groups go to the
// list together, in that order, with one atomic operation per block: groups that
// are walked at the same time read the same nodes (one atomic per group took 139 us
// at 2,097,152 particles).
struct GroupListArgs {
    const int *ctr;
    const int4 *nc;       // (first child, children, first particle, particles)
    const int4 *in_rec;   // internal nodes in pre-order: (.., .., .., id)
    const int *depth;
    const float4 *pa, *pb;
    const double *frame;
    const int *mlist;
    int2 *groups;
    int *gctr;
};

// The groups of one cell: pieces (first particle, count), the count negative
// for particles that go to the list one by one.  A cell of more than GL_PIECES
// pieces (oversized leaves) is cut again when they are written.
constexpr int GL_PIECES = 16;
struct CellGroups {
    int pieces = 0, entries = 0;
    int2 piece[GL_PIECES];
};

// Cuts particles [first, first + count) into pieces; writes them from
// groups[at] on when at >= 0.
__device__ __noinline__ void put_groups(const GroupListArgs &A, int first, int count, int depth, int at,
                                        CellGroups &g)
{
    const int nmis = A.mlist[0];
    for (int b = 0; b < count; b += GW_GROUP) {
        const int f = first + b, c = min(GW_GROUP, count - b);
        bool measure = nmis > kMisplacedCap;
        for (int k = 0; k < nmis && !measure; ++k) {
            const int q = A.mlist[1 + k];
            measure = q >= f && q < f + c;
        }
        const bool fits = !measure || group_extent_fits(f, c, depth, A.pa, A.pb, A.frame[4]);
        if (at >= 0) {
            if (fits)
                A.groups[at + g.entries] = make_int2(f, c);
            else
                for (int q = 0; q < c; ++q) A.groups[at + g.entries + q] = make_int2(f + q, 1);
        } else if (g.pieces < GL_PIECES) {
            g.piece[g.pieces] = make_int2(f, fits ? c : -c);
        }
        ++g.pieces;
        g.entries += fits ? 1 : c;
    }
}

// The groups of one cell, written from groups[at] on when at >= 0.
__device__ void cell_groups(const GroupListArgs &A, int cell, int at, CellGroups &g)
{
    g.pieces = g.entries = 0;
    const int4 ci = A.nc[cell];
    // a smaller cell is grouped by its parent; a leaf (the root) is cut
    if (ci.w <= GW_GROUP || ci.y <= 0) {
        if (cell == 0 && ci.w > 0) put_groups(A, ci.z, ci.w, A.depth[cell], at, g);
        return;
    }
    int4 child[8];   // all in flight together
#pragma unroll
    for (int k = 0; k < 8; ++k)
        child[k] = k < ci.y ? A.nc[ci.x + k] : make_int4(0, 1, 0, GW_GROUP + 1);
    // Runs of consecutive children of at most GW_GROUP particles each are
    // contiguous in sorted order and lie in this cell: each run is cut into
    // pieces of GW_GROUP particles (the last one shorter), so that groups
    // fill the warp's lanes (children of 20, 20 and 20 particles make groups
    // of 32 and 28, not three of 20).
    int first = 0, count = 0;
#pragma unroll
    for (int k = 0; k <= 8; ++k) {
        const int4 ch = k < 8 ? child[k] : make_int4(0, 1, 0, GW_GROUP + 1);
        if (ch.w > GW_GROUP) {   // a child walked as its own cell, or the end
            if (count > 0) put_groups(A, first, count, A.depth[cell], at, g);
            if (ch.y <= 0)       // an oversized leaf (depth limit)
                put_groups(A, ch.z, ch.w, A.depth[ci.x + k], at, g);
            count = 0;
            continue;
        }
        if (ch.w <= 0) continue;
        if (count == 0) first = ch.z;
        count += ch.w;
    }
}

constexpr int GL_THREADS = 256;

__global__ void __launch_bounds__(GL_THREADS) k_group_list(GroupListArgs A)
{
    __shared__ int s_warp[GL_THREADS / 32], s_base;
    if (tree_nodes(A.ctr) <= 0) return;   // none in an overflowed build
    const int internal = A.ctr[CTR_SAFE_INTERNAL];
    const int cells = max(internal, 1);   // a root that is a leaf is a cell, too
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b = blockIdx.x * GL_THREADS; b < cells; b += gridDim.x * GL_THREADS) {   // block-uniform
        const int i = b + threadIdx.x;
        const int cell = i < internal ? A.in_rec[i].w : i == 0 ? 0 : -1;
        CellGroups g;
        if (cell >= 0) cell_groups(A, cell, -1, g);
        const int entries = g.entries;
        int incl = entries;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = 0, total = 0;
        for (int w = 0; w < GL_THREADS / 32; ++w) {
            if (w < warp) before += s_warp[w];
            total += s_warp[w];
        }
        if (threadIdx.x == 0) s_base = total > 0 ? atomicAdd(&A.gctr[0], total) : 0;
        __syncthreads();
        int at = s_base + before + incl - entries;
        if (g.pieces > GL_PIECES) {
            cell_groups(A, cell, at, g);
        } else {
            for (int k = 0; k < g.pieces; ++k) {
                const int2 v = g.piece[k];
                if (v.y > 0) A.groups[at++] = v;
                for (int q = 0; q < -v.y; ++q) A.groups[at++] = make_int2(v.x + q, 1);
            }
        }
        __syncthreads();   // s_warp and s_base are read
    }
}

struct GroupWalkArgs {
    const float4 *na;       // (com_hi, mass)
    const float4 *nb;       // (com_lo, (cell side)^2)
    const float4 *nq;       // 2 per node: (xx, xy, xz, yy), (yz, zz, -, -)
    const int4 *nc;         // (first child, children, first particle, particles)
    const float4 *pa;       // sorted particles (x_hi, m)
    const float4 *pb;       // (x_lo, 0)
    const int *sidx;
    const double *frame;    // cx, cy, cz, width, box_length
    float eps2;
    float theta2;
    double G;
    double *a;
    unsigned long long *counters;
    unsigned *status;
    const int *gate;        // when set, the launch runs only if *gate != 0
    const int2 *groups;     // (first sorted particle, count)
    int *gctr;              // [0] groups, [1] work-queue head
};

// One warp's lists and state.  Lists hold their entries in pairs: pair k is
// entries (2k, 2k+1), and each float4 carries two fields of both entries side
// by side, so that one 16-byte shared load gives two fields of the pair in the
// register pairs the paired FP32 operations read (half the loads of one float2
// per field).
struct GroupShared {
    float4 cA[GW_CELLS / 2];   // (x, x', y, y')        accepted cells:
    float4 cB[GW_CELLS / 2];   // (z, z', m, m')        centre of mass and mass
    float4 qA[GW_CELLS / 2];   // (xx, xx', xy, xy')    negated quadrupole
    float4 qB[GW_CELLS / 2];   // (xz, xz', yy, yy')
    float4 qC[GW_CELLS / 2];   // (yz, yz', zz, zz')
    float4 pA[16], pB[16];     // a tile of leaf particles, in the same way
    float4 oh, ol;             // origin: the group's first particle (double-float);
                               // oh.w: -unit^2, ol.w: 1 / unit
    float4 nol;                // ol times -unit
    float4 lo, hi;             // the group's box from it, times unit (length_unit); lo.w: unit,
                               // hi.w: theta^2 / unit^2
    float sum[6 * GW_ROWS][32];   // (sum, error) of x, y, z of every lane's particles
    int parts[GW_PARTS + 32];  // particles of opened leaves (sorted positions)
};
static_assert(GW_CELLS % 32 == 0 && GW_PARTS % 32 == 0, "lists hold whole tiles");

// Field f (0: the float4's first two lanes, 1: its last two) of entry j.
__device__ __forceinline__ void put(float4 *arr, int j, int f, float v)
{
    reinterpret_cast<float *>(arr)[(j >> 1) * 4 + 2 * f + (j & 1)] = v;
}

__device__ __forceinline__ float get(const float4 *arr, int j, int f)
{
    return reinterpret_cast<const float *>(arr)[(j >> 1) * 4 + 2 * f + (j & 1)];
}

__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }

// A lane's particles.  Lane l holds the particles l % GW_COLS + k GW_COLS
// (k < GW_ROWS) of the group and takes the pairs of a list that are
// l / GW_COLS modulo GW_ROWS, so one shared load serves GW_ROWS particles.
struct LaneRows {   // times unit
    float rx[GW_ROWS], ry[GW_ROWS], rz[GW_ROWS];
};

// With quadrupoles the lengths of a group's walk are times this power of two, which
// makes the box about 2^10 long: accepted cells are then 2^-11 to 2^12 away at an
// angle of 1, and r^-5 stays in the middle of the FP32 range whatever the units of the
// positions (as they come it is infinite below 2e-8 and subnormal above 3e7).  The
// scaling is exact, and fused multiply-adds take it along without an instruction.
// Terms of particles, which go to shorter distances and have no power beyond r^-3,
// are in the units of the positions.
template <bool QUAD>
__device__ __forceinline__ float length_unit(double box_length)
{
    if (!QUAD) return 1.0f;
    const int e = ((__double2hiint(box_length) >> 20) & 0x7ff) - 1023;
    return __int_as_float((127 + max(-50, min(50, 10 - e))) << 23);
}

// Adds a list's partial sums, whose lengths were times unit, to the compensated sums.
template <int K>
__device__ __forceinline__ void add_sums(GroupShared &g, int lane, const float2 *ax, const float2 *ay,
                                         const float2 *az, float unit2)
{
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float2 v[3] = {ax[k], ay[k], az[k]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float s = g.sum[6 * k + 2 * d][lane], c = g.sum[6 * k + 2 * d + 1][lane];
            kahan_add(s, c, (v[d].x + v[d].y) * unit2);
            g.sum[6 * k + 2 * d][lane] = s;
            g.sum[6 * k + 2 * d + 1][lane] = c;
        }
    }
}

// Evaluates the accepted cells for the first K particles of every lane.  The
// list is filled up to whole turns of the lanes with copies of its last cell
// without mass or quadrupole, which add zero.  With P = -Q and d = com - x:
//     a = d [m / r^3 - 2.5 ((d.P.d) / r^2) / r^5] + P d / r^5
// (the monopole plus G [-Q d / r^5 + 2.5 (d.Q.d) d / r^7], G applied last; r^-7 by
// itself would leave the FP32 range).
template <bool QUAD, int K>
__device__ __forceinline__ void eval_cells(GroupShared &g, int count, int lane, float eps2,
                                           const LaneRows &L)
{
    const float unit2 = -g.oh.w;
    const float2 e2 = splat(eps2 * unit2);
    float2 ax[K], ay[K], az[K];
#pragma unroll
    for (int k = 0; k < K; ++k) ax[k] = ay[k] = az[k] = splat(0.f);
    const int end = (count + 1) >> 1;
#pragma unroll GW_UNROLL
    for (int b = 0, j = lane / GW_COLS; b < end; b += GW_ROWS, j += GW_ROWS) {
        const float4 va = g.cA[j], vb = g.cB[j];
        float4 qa, qb, qc;
        if (QUAD) {
            qa = g.qA[j];
            qb = g.qB[j];
            qc = g.qC[j];
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float2 dx = __fadd2_rn(lo2(va), splat(-L.rx[k]));
            const float2 dy = __fadd2_rn(hi2(va), splat(-L.ry[k]));
            const float2 dz = __fadd2_rn(lo2(vb), splat(-L.rz[k]));
            const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
            const float2 ri = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
            const float2 ri2 = __fmul2_rn(ri, ri);
            const float2 ri3 = __fmul2_rn(ri2, ri);
            float2 sc = __fmul2_rn(hi2(vb), ri3);
            if (QUAD) {
                const float2 xx = lo2(qa), xy = hi2(qa), xz = lo2(qb);
                const float2 yy = hi2(qb), yz = lo2(qc), zz = hi2(qc);
                const float2 px = __ffma2_rn(xx, dx, __ffma2_rn(xy, dy, __fmul2_rn(xz, dz)));
                const float2 py = __ffma2_rn(xy, dx, __ffma2_rn(yy, dy, __fmul2_rn(yz, dz)));
                const float2 pz = __ffma2_rn(xz, dx, __ffma2_rn(yz, dy, __fmul2_rn(zz, dz)));
                const float2 dpd = __ffma2_rn(dx, px, __ffma2_rn(dy, py, __fmul2_rn(dz, pz)));
                const float2 ri5 = __fmul2_rn(ri3, ri2);
                sc = __ffma2_rn(splat(-2.5f), __fmul2_rn(__fmul2_rn(dpd, ri2), ri5), sc);
                ax[k] = __ffma2_rn(dx, sc, __ffma2_rn(px, ri5, ax[k]));
                ay[k] = __ffma2_rn(dy, sc, __ffma2_rn(py, ri5, ay[k]));
                az[k] = __ffma2_rn(dz, sc, __ffma2_rn(pz, ri5, az[k]));
            } else {
                ax[k] = __ffma2_rn(dx, sc, ax[k]);
                ay[k] = __ffma2_rn(dy, sc, ay[k]);
                az[k] = __ffma2_rn(dz, sc, az[k]);
            }
        }
    }
    add_sums<K>(g, lane, ax, ay, az, unit2);
}

// Evaluates the first `count` leaf particles (count > 0).  They are gathered 32
// at a time, one per lane, the next tile's loads in flight while one is
// evaluated; a short tile is filled with copies of its last particle without
// mass.  With softening every r^2 >= eps^2 > 0 and the particle's own term is 0
// by its zero offset; without it the own term (r^2 = 0) is skipped explicitly.
template <bool SOFT, int K>
__device__ __forceinline__ void eval_parts(const GroupWalkArgs &A, GroupShared &g, int count, int lane,
                                           const LaneRows &L)
{
    const float2 e2 = splat(A.eps2);
    const float back = g.ol.w;
    float2 ax[K], ay[K], az[K];
    float mx[K], my[K], mz[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        ax[k] = ay[k] = az[k] = splat(0.f);
        mx[k] = -L.rx[k] * back;
        my[k] = -L.ry[k] * back;
        mz[k] = -L.rz[k] * back;
    }
    const float4 oh = g.oh, ol = g.ol;
    int p = g.parts[min(lane, count - 1)];
    float4 ph = A.pa[p], pl = A.pb[p];
    for (int base = 0; base < count; base += 32) {
        __syncwarp();   // the last tile is read
        put(g.pA, lane, 0, (ph.x - oh.x) + (pl.x - ol.x));
        put(g.pA, lane, 1, (ph.y - oh.y) + (pl.y - ol.y));
        put(g.pB, lane, 0, (ph.z - oh.z) + (pl.z - ol.z));
        put(g.pB, lane, 1, base + lane < count ? ph.w : 0.f);
        if (base + 32 < count) {
            p = g.parts[min(base + 32 + lane, count - 1)];
            ph = A.pa[p];
            pl = A.pb[p];
        }
        __syncwarp();
        const int end = min(16, (count - base + 1) >> 1);
#pragma unroll GW_UNROLL
        for (int b = 0, j = lane / GW_COLS; b < end; b += GW_ROWS, j += GW_ROWS) {
            const float4 va = g.pA[j], vb = g.pB[j];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float2 dx = __fadd2_rn(lo2(va), splat(mx[k]));
                const float2 dy = __fadd2_rn(hi2(va), splat(my[k]));
                const float2 dz = __fadd2_rn(lo2(vb), splat(mz[k]));
                const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
                float2 ri = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                if (!SOFT) {   // own term without softening: r2 = 0 contributes nothing
                    ri.x = r2.x > 0.0f ? ri.x : 0.0f;
                    ri.y = r2.y > 0.0f ? ri.y : 0.0f;
                }
                const float2 sc = __fmul2_rn(hi2(vb), __fmul2_rn(__fmul2_rn(ri, ri), ri));
                ax[k] = __ffma2_rn(dx, sc, ax[k]);
                ay[k] = __ffma2_rn(dy, sc, ay[k]);
                az[k] = __ffma2_rn(dz, sc, az[k]);
            }
        }
    }
    add_sums<K>(g, lane, ax, ay, az, 1.0f);
}

// A group of at most GW_COLS particles leaves the second row empty and skips
// its work.
template <bool QUAD>
__device__ __forceinline__ void flush_cells(GroupShared &g, int count, int lane, float eps2, bool two,
                                            const LaneRows &L)
{
    const int at = count + lane;   // fill up to whole turns: 2 GW_ROWS entries
    if (lane < 2 * GW_ROWS && (at & ~(2 * GW_ROWS - 1)) < count) {
        put(g.cA, at, 0, get(g.cA, count - 1, 0));
        put(g.cA, at, 1, get(g.cA, count - 1, 1));
        put(g.cB, at, 0, get(g.cB, count - 1, 0));
        put(g.cB, at, 1, 0.f);
        if (QUAD) {
            put(g.qA, at, 0, 0.f);
            put(g.qA, at, 1, 0.f);
            put(g.qB, at, 0, 0.f);
            put(g.qB, at, 1, 0.f);
            put(g.qC, at, 0, 0.f);
            put(g.qC, at, 1, 0.f);
        }
    }
    __syncwarp();
    if (two)
        eval_cells<QUAD, 2>(g, count, lane, eps2, L);
    else
        eval_cells<QUAD, 1>(g, count, lane, eps2, L);
    __syncwarp();   // the list is read
}

template <bool SOFT>
__device__ __forceinline__ void flush_parts(const GroupWalkArgs &A, GroupShared &g, int count, int lane,
                                            bool two, const LaneRows &L)
{
    __syncwarp();
    if (two)
        eval_parts<SOFT, 2>(A, g, count, lane, L);
    else
        eval_parts<SOFT, 1>(A, g, count, lane, L);
}

// (s, c) += (s2, c2): both hold a sum s less its error c.
__device__ __forceinline__ void add_compensated(float &s, float &c, float s2, float c2)
{
    const float t = s + s2, b = t - s;
    c = (c + c2) - ((s - (t - b)) + (s2 - b));
    s = t;
}

// Barrier of a team: a warp or the whole CTA.
template <int TEAM>
__device__ __forceinline__ void team_sync()
{
    static_assert(TEAM == 1 || TEAM == GW_WARPS, "a team is a warp or a CTA");
    if (TEAM == 1)
        __syncwarp();
    else
        __syncthreads();
}

// Walk of one group, sorted particles [g0, gend), by warp `part` of a team of
// TEAM warps.  A team shares one stack: each step its warps take the next opened
// nodes from it together, test their children, put what is accepted on lists of
// their own and push what is opened at places that follow from the warps'
// counts.  They evaluate their lists in the same step, so that they stay in step.
// Lane l returns this warp's sums of particle l.
template <bool QUAD, bool SOFT, int TEAM>
__device__ __forceinline__ void walk_group(const GroupWalkArgs &A, GroupShared &g, int2 *stack,
                                           int2 *counts, int lane, int part, int g0, int gend,
                                           float *sum, float *err, unsigned &cells_total,
                                           unsigned &parts_total)
{
    constexpr int kStack = TEAM * GW_STACK;
    const int s = min(g0 + lane, gend - 1);   // lanes past the end repeat the last particle
    const bool two = gend - g0 > GW_COLS;
    LaneRows L;
    {
        float4 oh = A.pa[g0];
        const float4 ol = A.pb[g0];
        const float4 ph = A.pa[s], pl = A.pb[s];
        const float unit = length_unit<QUAD>(A.frame[4]);
        float lo[3] = {((ph.x - oh.x) + (pl.x - ol.x)) * unit, ((ph.y - oh.y) + (pl.y - ol.y)) * unit,
                       ((ph.z - oh.z) + (pl.z - ol.z)) * unit};
        float hi[3] = {lo[0], lo[1], lo[2]};
#pragma unroll
        for (int k = 0; k < GW_ROWS; ++k) {
            L.rx[k] = __shfl_sync(0xffffffffu, lo[0], k * GW_COLS + lane % GW_COLS);
            L.ry[k] = __shfl_sync(0xffffffffu, lo[1], k * GW_COLS + lane % GW_COLS);
            L.rz[k] = __shfl_sync(0xffffffffu, lo[2], k * GW_COLS + lane % GW_COLS);
        }
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
        if (lane == 0) {
            const float back = __int_as_float((254 << 23) - __float_as_int(unit));   // 1 / unit
            oh.w = -unit * unit;
            g.oh = oh;
            g.ol = make_float4(ol.x, ol.y, ol.z, back);
            g.nol = make_float4(-ol.x * unit, -ol.y * unit, -ol.z * unit, 0.f);
            g.lo = make_float4(lo[0], lo[1], lo[2], unit);
            g.hi = make_float4(hi[0], hi[1], hi[2], A.theta2 * back * back);
            if (part == 0) stack[0] = make_int2(0, 1);   // root
        }
#pragma unroll
        for (int i = 0; i < 6 * GW_ROWS; ++i) g.sum[i][lane] = 0.f;
    }
    const unsigned below = (1u << lane) - 1u;
    int top = 1, ncell = 0, npart = 0;
    unsigned tc = 0, tp = 0;
    team_sync<TEAM>();
    while (top > 0) {
        // take the children of up to four opened nodes a warp, eight lanes for
        // each, leaving room for as many opened nodes
        const int k = min(min(4 * TEAM, top), max(1, (kStack - GW_RESERVE - top) / 7));
        const int mine = 4 * part + (lane >> 3);
        top -= k;
        bool accept = false, leaf = false, open = false;
        int4 ci = make_int4(0, 0, 0, 0);
        float nx = 0.f, ny = 0.f, nz = 0.f, nm = 0.f;
        // the quadrupole comes with the node (used if accepted, as four nodes in
        // five are), so that its latency does not follow the decision
        float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
        const int2 from = mine < k ? stack[top + mine] : make_int2(0, 0);
        if ((lane & 7) < from.y) {
            const int node = from.x + (lane & 7);
            const float4 ca = A.na[node], cb = A.nb[node];
            ci = A.nc[node];
            if (QUAD) {
                q0 = A.nq[2 * node];
                q1 = A.nq[2 * node + 1];
            }
            const float4 oh = g.oh, nol = g.nol, lo = g.lo, hi = g.hi;
            // ((com_hi - origin_hi) + (com_lo - origin_lo)) unit
            nx = fmaf(ca.x - oh.x, lo.w, fmaf(cb.x, lo.w, nol.x));
            ny = fmaf(ca.y - oh.y, lo.w, fmaf(cb.y, lo.w, nol.y));
            nz = fmaf(ca.z - oh.z, lo.w, fmaf(cb.z, lo.w, nol.z));
            nm = ca.w;
            const float ex = fmaxf(fmaxf(lo.x - nx, nx - hi.x), 0.f);
            const float ey = fmaxf(fmaxf(lo.y - ny, ny - hi.y), 0.f);
            const float ez = fmaxf(fmaxf(lo.z - nz, nz - hi.z), 0.f);
            const float d2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
            // cb.w: (cell side)^2 of the node's depth
            const bool far = !(ci.z < gend && ci.z + ci.w > g0) && cb.w < hi.w * d2;
            accept = far && nm > 0.f;   // a far cell without mass adds nothing
            open = !far && ci.y > 0;
            leaf = !far && ci.y <= 0 && ci.w > 0;
        }
        const unsigned accepted = __ballot_sync(0xffffffffu, accept);
        const unsigned opened = __ballot_sync(0xffffffffu, open);
        unsigned leaves = __ballot_sync(0xffffffffu, leaf);
        int before = 0, pushes = __popc(opened);
        bool full = ncell + __popc(accepted) > GW_CELLS;
        if (TEAM > 1) {
            if (lane == 0) counts[part] = make_int2(pushes, full);
            __syncthreads();   // the popped entries and every warp's counts are read
            pushes = 0;
#pragma unroll
            for (int w = 0; w < TEAM; ++w) {
                const int2 c = counts[w];
                if (w < part) before += c.x;
                pushes += c.x;
                full |= c.y != 0;
            }
        }
        if (top + pushes > kStack) {   // team-uniform
            if (lane == 0) atomicOr(A.status, ST_STACK_OVERFLOW);
            break;
        }
        if (open) stack[top + before + __popc(opened & below)] = make_int2(ci.x, ci.y);
        top += pushes;
        if (accepted || full) {
            if (full && ncell > 0) {
                flush_cells<QUAD>(g, ncell, lane, A.eps2, two, L);
                tc += ncell;
                ncell = 0;
            }
            if (accept) {
                const int at = ncell + __popc(accepted & below);
                put(g.cA, at, 0, nx);
                put(g.cA, at, 1, ny);
                put(g.cB, at, 0, nz);
                put(g.cB, at, 1, nm);
                if (QUAD) {   // negated, as the evaluation expects
                    const float nu2 = g.oh.w;
                    put(g.qA, at, 0, q0.x * nu2);
                    put(g.qA, at, 1, q0.y * nu2);
                    put(g.qB, at, 0, q0.z * nu2);
                    put(g.qB, at, 1, q0.w * nu2);
                    put(g.qC, at, 0, q1.x * nu2);
                    put(g.qC, at, 1, q1.y * nu2);
                }
            }
            ncell += __popc(accepted);
        }
        // particles of leaves that are not accepted, a lane's leaf at a time
        while (leaves) {
            const int src = __ffs(leaves) - 1;
            leaves &= leaves - 1;
            const int first = __shfl_sync(0xffffffffu, ci.z, src);
            const int num = __shfl_sync(0xffffffffu, ci.w, src);
            for (int b = 0; b < num; b += 32) {
                if (b + lane < num) g.parts[npart + lane] = first + b + lane;
                npart += min(32, num - b);
                if (npart >= GW_PARTS) {   // whole tiles; the rest moves to the front
                    flush_parts<SOFT>(A, g, GW_PARTS, lane, two, L);
                    tp += GW_PARTS;
                    npart -= GW_PARTS;
                    int v = 0;
                    if (lane < npart) v = g.parts[GW_PARTS + lane];
                    __syncwarp();
                    if (lane < npart) g.parts[lane] = v;
                }
            }
        }
        team_sync<TEAM>();
    }
    if (ncell > 0) flush_cells<QUAD>(g, ncell, lane, A.eps2, two, L);
    if (npart > 0) flush_parts<SOFT>(A, g, npart, lane, two, L);
    // the lanes of a column hold parts of the same particles' sums; lane l keeps
    // particle l
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int k = 0; k < GW_ROWS; ++k) {
            float sm = g.sum[6 * k + 2 * d][lane], er = g.sum[6 * k + 2 * d + 1][lane];
#pragma unroll
            for (int o = GW_COLS; o < 32; o <<= 1)
                add_compensated(sm, er, __shfl_xor_sync(0xffffffffu, sm, o),
                                __shfl_xor_sync(0xffffffffu, er, o));
            if (k == 0 || lane / GW_COLS == k) {
                sum[d] = sm;
                err[d] = er;
            }
        }
    }
    cells_total = tc + ncell;
    parts_total = tp + npart;
    __syncwarp();   // every lane is done with the lists
}

template <bool QUAD, bool SOFT, int TEAM>
__device__ __forceinline__ void walk_queue(const GroupWalkArgs &A, int ngroups, GroupShared *gw,
                                           int2 *stacks)
{
    __shared__ int s_group[GW_WARPS];
    __shared__ int2 s_counts[GW_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = TEAM == 1 ? 0 : warp, lead = warp - part;
    unsigned long long n_cell = 0, n_pp = 0;
    for (;;) {
        if (part == 0 && lane == 0) s_group[lead] = atomicAdd(&A.gctr[1], 1);
        team_sync<TEAM>();
        const int gi = s_group[lead];
        if (gi >= ngroups) break;   // team-uniform
        const int2 grp = A.groups[gi];
        const int cnt = grp.y;
        float sum[3], err[3];
        unsigned tc, tp;
        walk_group<QUAD, SOFT, TEAM>(A, gw[warp], stacks + lead * GW_STACK, s_counts, lane, part,
                                     grp.x, grp.x + cnt, sum, err, tc, tp);
        double a[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) a[d] = (double)sum[d] - (double)err[d];
        if (TEAM > 1) {   // the other warps' sums, in their order
            if (part > 0) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    gw[warp].sum[2 * d][lane] = sum[d];
                    gw[warp].sum[2 * d + 1][lane] = err[d];
                }
            }
            if (lane == 0) s_counts[part] = make_int2(tc, tp);
            __syncthreads();
            if (part > 0) continue;   // the next group's first barrier ends the reads below
            for (int w = 1; w < TEAM; ++w) {
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    a[d] += (double)gw[w].sum[2 * d][lane] - (double)gw[w].sum[2 * d + 1][lane];
                tc += s_counts[w].x;
                tp += s_counts[w].y;
            }
        }
        if (lane < cnt) {
            const int id = A.sidx[grp.x + lane];
#pragma unroll
            for (int d = 0; d < 3; ++d) A.a[3 * id + d] = A.G * a[d];
        }
        n_cell += (unsigned long long)tc * cnt;
        n_pp += (unsigned long long)(tp - 1) * cnt;   // every particle meets itself in its own leaf
    }
    if (part == 0 && lane == 0 && n_cell + n_pp > 0) {
        atomicAdd(&A.counters[0], n_cell);
        atomicAdd(&A.counters[1], n_pp);
    }
}

template <bool QUAD, bool SOFT>
__global__ void __launch_bounds__(32 * GW_WARPS, GW_CTAS)
k_bh_group(GroupWalkArgs A)
{
    extern __shared__ __align__(16) unsigned char gw_smem[];
    if (A.gate && *A.gate == 0) return;          // block-uniform
    GroupShared *gw = reinterpret_cast<GroupShared *>(gw_smem);
    int2 *stacks = reinterpret_cast<int2 *>(gw + GW_WARPS);
    const int ngroups = A.gctr[0];
    if (ngroups < (int)(GW_TEAM * GW_WARPS * gridDim.x))   // grid-uniform
        walk_queue<QUAD, SOFT, GW_WARPS>(A, ngroups, gw, stacks);
    else
        walk_queue<QUAD, SOFT, 1>(A, ngroups, gw, stacks);
}

ErrorStatus launch_bh_group_walk(const OctreeDevice &t, double theta, double eps, double G,
                                 double *d_a, unsigned long long *counters, cudaStream_t s,
                                 const int *gate, bool reuse_groups)
{
    const bool soft = eps > 0.0 && (float)(eps * eps) > 0.0f;
    auto kernel = t.quad ? (soft ? k_bh_group<true, true> : k_bh_group<true, false>)
                         : (soft ? k_bh_group<false, true> : k_bh_group<false, false>);
    // The attribute belongs to the current device: set on every call (cheap,
    // host-side only, allowed during stream capture).
    const size_t smem = (sizeof(GroupShared) + GW_STACK * sizeof(int2)) * GW_WARPS;
    GS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    GroupWalkArgs w;
    w.na = t.w_na.as<float4>();
    w.nb = t.w_nb.as<float4>();
    w.nq = t.quad ? t.w_nq.as<float4>() : nullptr;
    w.nc = t.w_nc.as<int4>();
    w.pa = t.w_pa.as<float4>();
    w.pb = t.w_pb.as<float4>();
    w.sidx = t.sidx.as<int>();
    w.frame = t.frame.as<double>();
    w.eps2 = (float)(eps * eps);
    w.theta2 = (float)(theta * theta);
    w.G = G;
    w.a = d_a;
    w.counters = counters;
    w.status = reinterpret_cast<unsigned *>(t.ctr.as<int>() + CTR_STATUS);
    w.gate = gate;
    w.groups = t.g_list.as<int2>();
    w.gctr = t.g_ctr.as<int>();
    const DeviceInfo *dev = nullptr;
    GS_TRY(device_info(&dev));
    if (reuse_groups) {
        // the list and its count stay; only the work-queue head restarts
        GS_CUDA(cudaMemsetAsync(w.gctr + 1, 0, sizeof(int), s));
    } else {
        GS_CUDA(cudaMemsetAsync(t.g_ctr.p, 0, 2 * sizeof(int), s));
        const GroupListArgs l = {t.ctr.as<int>(), w.nc, t.in_rec.as<int4>(), t.t_depth.as<int>(),
                                 w.pa, w.pb, t.frame.as<double>(), t.mlist.as<int>(),
                                 t.g_list.as<int2>(), w.gctr};
        k_group_list<<<dev->sm_count * 8, GL_THREADS, 0, s>>>(l);
    }
    // persistent: every SM filled once (computed once per device)
    static std::atomic<int> grid_cache[kMaxDevices];
    int grid = grid_cache[dev->id].load(std::memory_order_acquire);
    if (grid == 0) {
        int per_sm = 0;
        GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bh_group<true, true>,
                                                              32 * GW_WARPS, smem));
        grid = dev->sm_count * (per_sm > 0 ? per_sm : 1);
        grid_cache[dev->id].store(grid, std::memory_order_release);
    }
    kernel<<<grid, 32 * GW_WARPS, smem, s>>>(w);
    GS_CUDA(cudaGetLastError());
    return ok();
}

}  // namespace gs
