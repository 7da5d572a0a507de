// k_walk.cu -- Barnes-Hut tree walk and the Barnes-Hut engine.
//
// Replaces helper_compute_acceleration (src/acceleration_barnes_hut.c:78-248)
// and acceleration_barnes_hut (:33-76).
//
// Warp-cooperative walk.  A warp (with few particles, a CTA) owns 32 consecutive
// particles in Morton order and walks the union of their traversals, each
// particle making the reference's own decision --
//   cell-membership test (compat: the reference's Morton prefixes with its
//   sorted-keys-by-particle-id read, src/acceleration_barnes_hut.c:120/:145;
//   otherwise the sorted index in the cell's range, which is the same test on the
//   particle's own key), then the opening test
//   (w_level)^2 < theta^2 |R|^2 (:157-162) -> monopole (:164-174),
//   else leaf -> particle terms skipping itself (:181-214), else descend.
// A shared stack holds opened nodes with the mask of the lanes that opened them.
// A step takes four of them, eight lanes for each, one child per lane:
//   * a lane first decides for all 32 particles at once, from their box, with
//     margins that make the answer every particle's own (72 % of the nodes at
//     N = 150,000, theta 0.5: 67 % accepted, 5 % opened by all);
//   * the other nodes go through shared memory, all lanes testing each;
//   * accepted cells and the particles of opened leaves go to a list with the
//     lanes they act on, evaluated 64 entries at a time, two particles and two
//     entries per lane through paired FP32 operations.
// Each particle sees exactly the nodes of the reference's depth-first walk, in
// another order.
//
// What bounds it is instruction issue.  Walking one child at a time cost about
// 220 instructions per node and warp; testing and evaluating every node with all
// lanes about 50; now 17 per list entry and row and 25 per tested node.  Step of
// the galaxy pair, theta 0.5, before and after the last change: N = 8,000 505 and
// 283 us, 40,000 1010 and 500, 150,000 1480 and 1174 (walk 1.08 and 0.86 ms); with
// the compat tests 2941 and 2292 at 150,000.
//
// Precision: positions and centres of mass are double-float pairs (hi, lo)
// relative to the bounding-box centre, so R = (c_hi - x_hi) + (c_lo - x_lo)
// keeps FP32 relative accuracy for close pairs; pair terms are FP32 with
// rsqrt; each term is added to a Kahan-compensated FP32
// accumulator.  The opening test is made in FP32 unless |w^2 - theta^2|R|^2|
// is within 1e-5 of w^2, in which case it is recomputed in FP64 exactly as
// the reference does, so every decision equals the reference's.
#include "gs_octree.h"
#include "gs_ptx.cuh"

#include <cstdlib>
#include <cstring>

namespace gs {

constexpr int WK_THREADS = 128;
constexpr int WK_WARPS = WK_THREADS / 32;
// CTAs per SM: 124 registers a thread without spills.  Five (95 registers) took
// 5 % longer at N = 150,000 and 1 % less at 600,000, six 28 and 14 % longer.
constexpr int WK_CTAS = 4;
// Below this many warps of particles per resident warp a CTA walks each 32
// particles together: with few of them the time is that of the slowest walk.
// Step of a galaxy pair, a warp and a CTA per 32 particles: N = 8,000 445 and
// 286 us, 20,000 490 and 334, 40,000 (0.5) 567 and 495, 80,000 (1.03) 749 and 772,
// 150,000 1183 and 1284.
constexpr double WK_TEAM = 0.8;
constexpr int WK_STACK = 384;    // stack entries (opened nodes) per warp
constexpr int WK_LIST = 64;      // list entries per warp
constexpr int WK_COLS = 16;      // lanes per row of a warp's particles
// Entries kept free for a depth-first descent: popping one opened node and pushing
// those of its (at most 8) children that are opened grows the stack by 7 per
// level.  Pops shrink so that the stack never passes WK_STACK - WK_RESERVE before
// such a descent starts.
constexpr int WK_RESERVE = 8 * (OCT_MAX_LEVEL + 1);

struct WalkArgs {
    const float4 *na;
    const float4 *nb;
    const float4 *nq;       // quadrupoles (2 float4 per node) or null
    const int4 *nc;
    const uint64_t *nkey;
    const double *ncom;     // FP64 centre of mass [3*nodes] (exact opening test)
    const int *depth;
    const float4 *pa;
    const float4 *pb;
    const int *sidx;
    const uint64_t *skeys;  // sorted keys
    const double *x;        // FP64 positions by particle id
    const double *frame;    // cx, cy, cz, width, box_length
    int n;
    float eps2;
    double theta2;
    double G;
    double *a;
    unsigned long long *counters;   // [0] accepted cells, [1] leaf pair terms
    unsigned *status;
};

// One warp's state.  List entries (accepted cells and particles of opened
// leaves, each with the lanes it acts on) are kept in pairs: pair k is entries
// (2k, 2k+1), and each float4 carries two fields of both side by side, the
// register pairs of the paired FP32 operations.
template <bool QUAD, bool COMPAT>
struct WalkShared {
    float4 sA[WK_LIST / 2];      // (x, x', y, y')    hi
    float4 sB[WK_LIST / 2];      // (z, z', m, m')
    float4 sC[WK_LIST / 2];      // (x, x', y, y')    lo
    float2 sZ[WK_LIST / 2];      // (z, z')
    uint2 sM[WK_LIST / 2];       // lanes
    // negated quadrupole (xx, xx', xy, xy'), (xz, xz', yy, yy'), (yz, yz', zz, zz'); 0 for a particle
    float4 qA[QUAD ? WK_LIST / 2 : 1], qB[QUAD ? WK_LIST / 2 : 1], qC[QUAD ? WK_LIST / 2 : 1];
    float4 a[32], b[32];         // nodes to test lane by lane: com (hi, mass), (lo, cell side^2)
    int4 c[32];                  // (node, -, first particle, particles)
    unsigned mask[32];           // lanes that reach it; after the test, that open it
    uint64_t key[COMPAT ? 32 : 1];
    int level[COMPAT ? 32 : 1];
    uint64_t own[COMPAT ? 32 : 1];   // the particles' keys in order
    int2 part[64];               // particles of opened leaves, lanes
    float pos[6][32];            // negated particle positions: hi x y z, lo x y z
    float4 oh, ol, lo, hi;       // origin (the first particle) and the particles' box from it
    unsigned poison;             // lanes that a term that is not finite acts on
};

// Compensated sums of a lane's two particles, the even and the odd list entries
// apart; n holds the negated compensations.
struct Acc {
    float2 s[2][3], n[2][3];
};

__device__ __forceinline__ void put(float4 *arr, int j, int f, float v)
{
    reinterpret_cast<float *>(arr)[(j >> 1) * 4 + 2 * f + (j & 1)] = v;
}

__device__ __forceinline__ float2 wk_lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 wk_hi2(const float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 wk_splat(float v) { return make_float2(v, v); }

template <bool QUAD, bool COMPAT>
__device__ __forceinline__ void put_entry(WalkShared<QUAD, COMPAT> &w, int at, const float4 h,
                                          const float4 l, unsigned lanes, const float4 q0, const float4 q1)
{
    put(w.sA, at, 0, h.x);
    put(w.sA, at, 1, h.y);
    put(w.sB, at, 0, h.z);
    put(w.sB, at, 1, h.w);
    put(w.sC, at, 0, l.x);
    put(w.sC, at, 1, l.y);
    reinterpret_cast<float *>(w.sZ)[at] = l.z;
    reinterpret_cast<unsigned *>(w.sM)[at] = lanes;
    if (QUAD) {   // negated, as the evaluation expects
        put(w.qA, at, 0, -q0.x);
        put(w.qA, at, 1, -q0.y);
        put(w.qB, at, 0, -q0.z);
        put(w.qB, at, 1, -q0.w);
        put(w.qC, at, 0, -q1.x);
        put(w.qC, at, 1, -q1.y);
    }
}

// Evaluates the list.  Lane l holds particles l % 16 and l % 16 + 16 of the warp
// and takes every second pair of entries, so that one shared load serves two
// particles (a broadcast 16-byte load costs the shared-memory pipe four cycles).
// Lanes an entry does not act on add zeros.
template <bool QUAD, bool COMPAT>
__device__ __forceinline__ void eval_list(WalkShared<QUAD, COMPAT> &w, int count, int lane, float eps2,
                                          Acc &acc)
{
    const int fill = count + lane;   // up to whole turns of four entries, on no lane
    if (lane < 4 && (fill & ~3) < count) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        put_entry<QUAD, COMPAT>(w, fill, zero, zero, 0u, zero, zero);
    }
    __syncwarp();
    const int col = lane % WK_COLS;
    const unsigned bit[2] = {1u << col, 1u << (col + WK_COLS)};
    float2 nh[2][3], nl[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            nh[k][d] = wk_splat(w.pos[d][col + k * WK_COLS]);
            nl[k][d] = wk_splat(w.pos[3 + d][col + k * WK_COLS]);
        }
    const float2 e2 = wk_splat(eps2), minus = wk_splat(-1.0f);
    const int end = (count + 1) >> 1;
#pragma unroll 1
    for (int b = 0, j = lane / WK_COLS; b < end; b += 2, j += 2) {
        const float4 vA = w.sA[j], vB = w.sB[j], vC = w.sC[j];
        const float2 vZ = w.sZ[j];
        const uint2 lanes = w.sM[j];
        float4 qa, qb, qc;
        if (QUAD) {
            qa = w.qA[j];
            qb = w.qB[j];
            qc = w.qC[j];
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float2 dx = __fadd2_rn(__fadd2_rn(wk_lo2(vA), nh[k][0]), __fadd2_rn(wk_lo2(vC), nl[k][0]));
            const float2 dy = __fadd2_rn(__fadd2_rn(wk_hi2(vA), nh[k][1]), __fadd2_rn(wk_hi2(vC), nl[k][1]));
            const float2 dz = __fadd2_rn(__fadd2_rn(wk_lo2(vB), nh[k][2]), __fadd2_rn(vZ, nl[k][2]));
            const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
            const float2 ri = make_float2(lanes.x & bit[k] ? rsqrt_approx(r2.x) : 0.0f,
                                          lanes.y & bit[k] ? rsqrt_approx(r2.y) : 0.0f);
            const float2 ri2 = __fmul2_rn(ri, ri);
            const float2 ri3 = __fmul2_rn(ri2, ri);
            float2 sc, p[3];
            if (QUAD) {
                // d = com - x = -R, P = -Q:  G [m d / r^3 + P d / r^5 - 2.5 (d.P.d) d / r^7], as
                // r^-3 [d (m - 2.5 (d.t) r^-2) + t] with t = P d / r^2.  t is at most m s^2 / r
                // for a cell of extent s, so no term leaves the range before m r^-3 does (r^-7
                // is infinite below 3e-6, r^-5 below 2e-8, and a particle's P = 0 then gives
                // NaN; above 3e6 r^-7 is 0).  The same number of operations.
                const float2 xx = wk_lo2(qa), xy = wk_hi2(qa), xz = wk_lo2(qb);
                const float2 yy = wk_hi2(qb), yz = wk_lo2(qc), zz = wk_hi2(qc);
                const float2 tx = __fmul2_rn(__ffma2_rn(xx, dx, __ffma2_rn(xy, dy, __fmul2_rn(xz, dz))), ri2);
                const float2 ty = __fmul2_rn(__ffma2_rn(xy, dx, __ffma2_rn(yy, dy, __fmul2_rn(yz, dz))), ri2);
                const float2 tz = __fmul2_rn(__ffma2_rn(xz, dx, __ffma2_rn(yz, dy, __fmul2_rn(zz, dz))), ri2);
                const float2 dt = __ffma2_rn(dx, tx, __ffma2_rn(dy, ty, __fmul2_rn(dz, tz)));
                sc = __fmul2_rn(__ffma2_rn(wk_splat(-2.5f), __fmul2_rn(dt, ri2), wk_hi2(vB)), ri3);
                p[0] = __ffma2_rn(tx, ri3, __fmul2_rn(dx, sc));
                p[1] = __ffma2_rn(ty, ri3, __fmul2_rn(dy, sc));
                p[2] = __ffma2_rn(tz, ri3, __fmul2_rn(dz, sc));
            } else {
                sc = __fmul2_rn(wk_hi2(vB), ri3);
                p[0] = __fmul2_rn(dx, sc);
                p[1] = __fmul2_rn(dy, sc);
                p[2] = __fmul2_rn(dz, sc);
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float2 y = __fadd2_rn(p[d], acc.n[k][d]);
                const float2 t = __fadd2_rn(acc.s[k][d], y);
                acc.n[k][d] = __ffma2_rn(__ffma2_rn(acc.s[k][d], minus, t), minus, y);   // y - (t - s)
                acc.s[k][d] = t;
            }
        }
    }
    __syncwarp();   // the list is read
}

__device__ __forceinline__ bool all_finite(const float4 v)
{
    return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, v.w * 0.f))) == 0.f;
}

// The particles w.part[0 .. count) (at most 32) of opened leaves become list entries
// from `at` on; returns the lanes that this lane's one acts on (not the particle
// itself).  Lanes an entry does not act on add its terms times zero, so a particle
// with a coordinate or mass that is not finite acts on no lane: the sums of those it
// should act on become NaN at the end (w.poison).
template <bool QUAD, bool COMPAT>
__device__ __forceinline__ unsigned put_parts(const WalkArgs &A, WalkShared<QUAD, COMPAT> &w, int at,
                                              int count, int s0, int lane)
{
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane >= count) return 0u;
    const int2 e = w.part[lane];
    const int own = e.x - s0;
    const unsigned lanes = (unsigned)e.y & ~((unsigned)own < 32u ? 1u << own : 0u);
    float4 h = A.pa[e.x], l = A.pb[e.x];
    unsigned on = lanes;
    if (!all_finite(h)) {
        atomicOr(&w.poison, lanes);
        h = l = zero;
        on = 0;
    }
    put_entry<QUAD, COMPAT>(w, at + lane, h, l, on, zero, zero);
    return lanes;
}

template <int TEAM>
__device__ __forceinline__ void walk_sync()
{
    if (TEAM == 1)
        __syncwarp();
    else
        __syncthreads();
}

// A warp (TEAM = 1) or a CTA (TEAM = WK_WARPS) per 32 particles.  A team shares
// one stack: its warps take the next opened nodes from it together, keep lists of
// their own and push what their lanes open at places that follow from the warps'
// counts.
template <bool QUAD, bool COMPAT, int TEAM>
__global__ void __launch_bounds__(WK_THREADS, WK_CTAS)
k_bh_walk(WalkArgs A)
{
    using Shared = WalkShared<QUAD, COMPAT>;
    constexpr int kStack = TEAM * WK_STACK;
    __shared__ Shared shared_all[WK_WARPS];
    __shared__ int2 stack_all[WK_WARPS * WK_STACK];                // (first child, lanes)
    __shared__ unsigned char children_all[WK_WARPS * WK_STACK];    // children
    __shared__ int counts[WK_WARPS];

    if (*A.status & ST_TREE_OVERFLOW) return;   // the build overflowed: no tree to walk
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int part = TEAM == 1 ? 0 : warp;
    Shared &w = shared_all[warp];
    int2 *stack = stack_all + (warp - part) * WK_STACK;
    unsigned char *children = children_all + (warp - part) * WK_STACK;
    const unsigned lt = (1u << lane) - 1u;

    const int s0 = (TEAM == 1 ? blockIdx.x * WK_WARPS + warp : blockIdx.x) * 32;
    if (s0 >= A.n) return;   // team-uniform
    const int held = min(32, A.n - s0);
    const int s = s0 + lane;
    const bool valid = lane < held;
    const int id = valid ? A.sidx[s] : -1;
    uint64_t key_i = 0;
    // negated particle position; lanes past the end repeat the last particle
    float nh[3], nl[3];
    {
        if (COMPAT && valid) key_i = A.skeys[id];
        const float4 oh = A.pa[s0], ol = A.pb[s0];
        const float4 ph = A.pa[min(s, A.n - 1)], pl = A.pb[min(s, A.n - 1)];
        nh[0] = -ph.x, nh[1] = -ph.y, nh[2] = -ph.z;
        nl[0] = -pl.x, nl[1] = -pl.y, nl[2] = -pl.z;
        float lo[3] = {(ph.x - oh.x) + (pl.x - ol.x), (ph.y - oh.y) + (pl.y - ol.y),
                       (ph.z - oh.z) + (pl.z - ol.z)};
        float hi[3] = {lo[0], lo[1], lo[2]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            w.pos[d][lane] = nh[d];
            w.pos[3 + d][lane] = nl[d];
            for (int o = 16; o > 0; o >>= 1) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
        }
        if (lane == 0) {
            w.oh = oh;
            w.ol = ol;
            w.lo = make_float4(lo[0], lo[1], lo[2], 0.f);
            w.hi = make_float4(hi[0], hi[1], hi[2], 0.f);
            w.poison = 0;
        }
    }
    if (COMPAT) {   // each key goes to its rank; lanes past the end behind all keys
        if (!valid) key_i = ~0ull;
        int rank = 0;
        for (int q = 0; q < 32; ++q) {
            const uint64_t other = __shfl_sync(0xffffffffu, key_i, q);
            rank += other < key_i || (other == key_i && q < lane);
        }
        w.own[rank] = key_i;
    }
    const float th2f = (float)A.theta2;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    Acc acc = {};
    unsigned n_cell = 0, n_pp = 0;   // of the lane's nodes and leaf particles
    int nlist = 0, npart = 0;

    // the root is opened by every lane without a test: its children start the walk
    const unsigned all = held == 32 ? 0xffffffffu : (1u << held) - 1u;
    const int4 root = A.nc[0];
    int top = root.y > 0 ? 1 : 0;
    if (lane == 0 && part == 0) {
        stack[0] = make_int2(root.x, (int)all);
        children[0] = (unsigned char)root.y;
    }
    walk_sync<TEAM>();
    while (top > 0) {
        // the children of up to four opened nodes a warp, eight lanes for each
        const int k = min(min(4 * TEAM, top), max(1, (kStack - WK_RESERVE - top) / 7));
        const int mine = 4 * part + (lane >> 3);
        top -= k;
        int4 ci = make_int4(0, 0, 0, 0);
        float4 ca = zero4, cb = zero4, q0 = zero4, q1 = zero4;
        unsigned reach = 0, opened = 0;   // lanes that reach this lane's node, that open it
        bool test = false;
        int node = 0, level = 0;
        uint64_t nkey = 0;
        if (mine < k && (lane & 7) < children[top + mine]) {
            const int2 from = stack[top + mine];
            node = from.x + (lane & 7);
            reach = (unsigned)from.y;
            ca = A.na[node];
            cb = A.nb[node];
            ci = A.nc[node];
            if (QUAD) {
                q0 = A.nq[2 * (size_t)node];
                q1 = A.nq[2 * (size_t)node + 1];
            }
            // Decisions that are the same for all 32 particles, from their box: with
            // a margin above the rounding of the offsets (4e-7 of them) and of the
            // squares and above the band of the exact test, so that every
            // particle's own test below would decide the same.
            const float4 oh = w.oh, ol = w.ol, lo = w.lo, hi = w.hi;
            const float n[3] = {(ca.x - oh.x) + (cb.x - ol.x), (ca.y - oh.y) + (cb.y - ol.y),
                                (ca.z - oh.z) + (cb.z - ol.z)};
            const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
            float near2 = 0.f, far2 = 0.f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float g = 4e-7f * (fabsf(n[d]) + fmaxf(fabsf(l[d]), fabsf(h[d])));
                const float nd = fmaxf(fmaxf(l[d] - n[d], n[d] - h[d]) - g, 0.f);
                const float fd = fmaxf(n[d] - l[d], h[d] - n[d]) + g;
                near2 = fmaf(nd, nd, near2);
                far2 = fmaf(fd, fd, far2);
            }
            // no particle is inside the cell
            bool away = ci.z >= s0 + held || ci.z + ci.w <= s0;
            if (COMPAT) {   // the first of the ordered keys at or after the cell's
                nkey = A.nkey[node];
                level = A.depth[node];
                const int sh = 3 * (OCT_MAX_LEVEL - level);
                const uint64_t cell = nkey >> sh;
                int at = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (w.own[at + step - 1] >> sh < cell) at += step;
                away = w.own[at] >> sh != cell;
            }
            const bool around = !COMPAT && ci.z <= s0 && ci.z + ci.w >= s0 + held;
            if (around || cb.w > 1.00002f * th2f * far2)
                opened = reach;
            else
                // (far2 is NaN where any coordinate of the centre is, near2 is not)
                test = !(away && 1.00002f * cb.w < th2f * fmaf(far2, 0.f, near2));
        }
        // the other nodes lane by lane
        const unsigned tests = __ballot_sync(0xffffffffu, test);
        if (test) {
            const int at = __popc(tests & lt);
            w.a[at] = ca;
            w.b[at] = cb;
            w.c[at] = make_int4(node, 0, ci.z, ci.w);
            w.mask[at] = reach;
            if (COMPAT) {
                w.key[at] = nkey;
                w.level[at] = level;
            }
        }
        __syncwarp();
        const int ntest = __popc(tests);
#pragma unroll 2
        for (int j = 0; j < ntest; ++j) {
            const float4 va = w.a[j], vb = w.b[j];
            const int4 vc = w.c[j];
            const bool act = (w.mask[j] >> lane) & 1u;
            const float dx = (va.x + nh[0]) + (vb.x + nl[0]);
            const float dy = (va.y + nh[1]) + (vb.y + nl[1]);
            const float dz = (va.z + nh[2]) + (vb.z + nl[2]);
            const float t = th2f * fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            bool accept = vb.w < t;
            bool inside;
            if (COMPAT) {
                const int sh = 3 * (OCT_MAX_LEVEL - w.level[j]);
                inside = (key_i >> sh) == (w.key[j] >> sh);
            } else {
                inside = (unsigned)(s - vc.z) < (unsigned)vc.w;
            }
            if (act && !inside && fabsf(vb.w - t) <= 1e-5f * vb.w) {
                // exact FP64 test, reference operation order
                const int c = vc.x;
                const double r0 = __dsub_rn(A.x[3 * (size_t)id + 0], A.ncom[3 * (size_t)c + 0]);
                const double r1 = __dsub_rn(A.x[3 * (size_t)id + 1], A.ncom[3 * (size_t)c + 1]);
                const double r2 = __dsub_rn(A.x[3 * (size_t)id + 2], A.ncom[3 * (size_t)c + 2]);
                const double nsd = __dadd_rn(__dadd_rn(__dmul_rn(r0, r0), __dmul_rn(r1, r1)),
                                             __dmul_rn(r2, r2));
                // box_length / (2 << level)  (src/acceleration_barnes_hut.c:157)
                const double wd = __ddiv_rn(A.frame[4], (double)(2 << A.depth[c]));
                accept = __dmul_rn(wd, wd) < __dmul_rn(A.theta2, nsd);
            }
            const unsigned om = __ballot_sync(0xffffffffu, act && (inside || !accept));
            if (lane == 0) w.mask[j] = om;
        }
        __syncwarp();
        if (test) opened = w.mask[__popc(tests & lt)];
        // opened nodes
        const bool push = opened != 0 && ci.y > 0;
        const unsigned pushed = __ballot_sync(0xffffffffu, push);
        int before = 0, pushes = __popc(pushed);
        if (TEAM > 1) {
            if (lane == 0) counts[part] = pushes;
            __syncthreads();   // the popped entries and every warp's counts are read
            pushes = 0;
#pragma unroll
            for (int q = 0; q < TEAM; ++q) {
                if (q < part) before += counts[q];
                pushes += counts[q];
            }
        }
        if (top + pushes > kStack) {   // team-uniform
            if (lane == 0) atomicOr(A.status, ST_STACK_OVERFLOW);
            break;
        }
        if (push) {
            const int at = top + before + __popc(pushed & lt);
            stack[at] = make_int2(ci.x, (int)opened);
            children[at] = (unsigned char)ci.y;
        }
        top += pushes;
        // accepted cells
        const unsigned takers = reach & ~opened;
        const unsigned taken = __ballot_sync(0xffffffffu, takers != 0);
        if (nlist + __popc(taken) > WK_LIST) {
            eval_list<QUAD, COMPAT>(w, nlist, lane, A.eps2, acc);
            nlist = 0;
        }
        if (takers) {
            unsigned on = takers;
            if (!all_finite(ca) || (QUAD && !(all_finite(q0) && all_finite(q1)))) {
                atomicOr(&w.poison, takers);   // as in put_parts
                ca = cb = q0 = q1 = zero4;
                on = 0;
            }
            put_entry<QUAD, COMPAT>(w, nlist + __popc(taken & lt), ca, cb, on, q0, q1);
        }
        nlist += __popc(taken);
        n_cell += __popc(takers);
        // particles of opened leaves: leaves of one particle together, the others
        // in turn; 32 particles at a time become list entries
        const int num = opened != 0 && ci.y <= 0 ? ci.w : 0;
        const unsigned ones = __ballot_sync(0xffffffffu, num == 1);
        unsigned leaves = __ballot_sync(0xffffffffu, num > 1);
        if (num == 1) w.part[npart + __popc(ones & lt)] = make_int2(ci.z, (int)opened);
        npart += __popc(ones);
        int skip = 0;   // particles of the first remaining leaf already taken
        while (npart >= 32 || leaves) {
            if (npart >= 32) {
                __syncwarp();
                if (nlist + 32 > WK_LIST) {
                    eval_list<QUAD, COMPAT>(w, nlist, lane, A.eps2, acc);
                    nlist = 0;
                }
                n_pp += __popc(put_parts<QUAD, COMPAT>(A, w, nlist, 32, s0, lane));
                nlist += 32;
                npart -= 32;
                int2 rest = make_int2(0, 0);
                if (lane < npart) rest = w.part[32 + lane];
                __syncwarp();
                if (lane < npart) w.part[lane] = rest;
                continue;
            }
            const int src = __ffs(leaves) - 1;
            const int first = __shfl_sync(0xffffffffu, ci.z, src) + skip;
            const int left = __shfl_sync(0xffffffffu, num, src) - skip;
            const int om = __shfl_sync(0xffffffffu, (int)opened, src);
            const int take = min(left, 32);
            if (lane < take) w.part[npart + lane] = make_int2(first + lane, om);
            npart += take;
            skip += take;
            if (take == left) {
                leaves &= leaves - 1;
                skip = 0;
            }
        }
        walk_sync<TEAM>();
    }
    __syncwarp();
    if (npart > 0) {   // fewer than 32
        if (nlist + npart > WK_LIST) {
            eval_list<QUAD, COMPAT>(w, nlist, lane, A.eps2, acc);
            nlist = 0;
        }
        n_pp += __popc(put_parts<QUAD, COMPAT>(A, w, nlist, npart, s0, lane));
        nlist += npart;
    }
    if (nlist > 0) eval_list<QUAD, COMPAT>(w, nlist, lane, A.eps2, acc);
    // lanes l and l ^ 16 hold halves of the same two particles' sums: lane l keeps
    // particle l
    double a[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double row[2];
#pragma unroll
        for (int q = 0; q < 2; ++q)
            row[q] = ((double)acc.s[q][d].x + (double)acc.n[q][d].x) +
                     ((double)acc.s[q][d].y + (double)acc.n[q][d].y);
        const bool second = lane >= WK_COLS;
        a[d] = (second ? row[1] : row[0]) +
               __shfl_xor_sync(0xffffffffu, second ? row[0] : row[1], WK_COLS);
        if ((w.poison >> lane) & 1u) a[d] = __longlong_as_double(0x7ff8000000000000ll);
    }
    if (TEAM > 1) {   // the other warps' sums, in their order
        double *out = reinterpret_cast<double *>(w.sA);
        static_assert(sizeof(w.sA) + sizeof(w.sB) + sizeof(w.sC) >= 96 * sizeof(double), "sums fit");
        if (part > 0)
            for (int d = 0; d < 3; ++d) out[32 * d + lane] = a[d];
        __syncthreads();
        if (part == 0)
            for (int q = 1; q < TEAM; ++q) {
                const double *in = reinterpret_cast<const double *>(shared_all[q].sA);
                for (int d = 0; d < 3; ++d) a[d] += in[32 * d + lane];
            }
    }
    if (valid && part == 0)
        for (int d = 0; d < 3; ++d) A.a[3 * (size_t)id + d] = A.G * a[d];
    // interaction counts (warp sums, one atomic per warp)
    unsigned long long tc = n_cell, tp = n_pp;
    for (int o = 16; o > 0; o >>= 1) {
        tc += __shfl_down_sync(0xffffffffu, tc, o);
        tp += __shfl_down_sync(0xffffffffu, tp, o);
    }
    if (lane == 0) {
        atomicAdd(&A.counters[0], tc);
        atomicAdd(&A.counters[1], tp);
    }
}

template <int TEAM>
static void launch_walk_team(const WalkArgs &w, bool quad, bool compat, cudaStream_t s)
{
    const int warps = (w.n + 31) / 32, grid = TEAM == 1 ? (warps + WK_WARPS - 1) / WK_WARPS : warps;
    if (compat)
        k_bh_walk<false, true, TEAM><<<grid, WK_THREADS, 0, s>>>(w);
    else if (quad)
        k_bh_walk<true, false, TEAM><<<grid, WK_THREADS, 0, s>>>(w);
    else
        k_bh_walk<false, false, TEAM><<<grid, WK_THREADS, 0, s>>>(w);
}

static void launch_walk_kernel(const WalkArgs &w, bool quad, bool compat, int sm_count,
                               cudaStream_t s)
{
    if ((w.n + 31) / 32 < (int)(WK_TEAM * WK_CTAS * WK_WARPS * sm_count))
        launch_walk_team<WK_WARPS>(w, quad, compat, s);
    else
        launch_walk_team<1>(w, quad, compat, s);
}

// ------------------------------------------------------------------------
namespace {

class BarnesHutEngine final : public Engine {
  public:
    BarnesHutEngine(bool compat, bool quad, bool group)
        : compat_(compat), quad_(quad && !compat), group_(group && !compat)
    {
    }

    ErrorStatus setup(int n, double G, const AccelerationParam &p) override
    {
        n_ = n;
        G_ = G;
        eps_ = p.softening_length;
        theta_ = p.opening_angle;
        GS_TRY(tree_.setup(n, p.max_num_particles_per_leaf, compat_, quad_));
        GS_TRY(counters_.reserve(4 * sizeof(unsigned long long)));
        GS_CUDA(cudaMemset(counters_.p, 0, 4 * sizeof(unsigned long long)));
        return ok();
    }

    ErrorStatus compute(const double *d_x, const double *d_m, double *d_a, cudaStream_t s,
                        ForceTimer *timer) override
    {
        GS_TRY(tree_.build(d_x, d_m, s));
        WalkArgs w;
        w.na = tree_.w_na.as<float4>();
        w.nb = tree_.w_nb.as<float4>();
        w.nq = quad_ ? tree_.w_nq.as<float4>() : nullptr;
        w.nc = tree_.w_nc.as<int4>();
        w.nkey = tree_.w_nkey.as<uint64_t>();
        w.ncom = tree_.t_com.as<double>();
        w.depth = tree_.t_depth.as<int>();
        w.pa = tree_.w_pa.as<float4>();
        w.pb = tree_.w_pb.as<float4>();
        w.sidx = tree_.sidx.as<int>();
        w.skeys = tree_.keys.as<uint64_t>();
        w.x = d_x;
        w.frame = tree_.frame.as<double>();
        w.n = n_;
        w.eps2 = (float)(eps_ * eps_);
        w.theta2 = theta_ * theta_;
        w.G = G_;
        w.a = d_a;
        w.counters = counters_.as<unsigned long long>();
        w.status = reinterpret_cast<unsigned *>(tree_.ctr.as<int>() + CTR_STATUS);
        GS_CUDA(cudaMemsetAsync(counters_.p, 0, 2 * sizeof(unsigned long long), s));
        if (group_) {
            if (timer) GS_TRY(timer->begin(s));
            GS_TRY(launch_bh_group_walk(tree_, theta_, eps_, G_, d_a, w.counters, s));
            if (timer) GS_TRY(timer->end(s));
            return ok();
        }
        if (timer) GS_TRY(timer->begin(s));
        const DeviceInfo *dev = nullptr;
        GS_TRY(device_info(&dev));
        launch_walk_kernel(w, quad_, compat_, dev->sm_count, s);
        GS_CUDA(cudaGetLastError());
        if (timer) GS_TRY(timer->end(s));
        return ok();
    }

    // the group walk is two launches (group list, walk)
    int kernels_per_eval() const override { return tree_.launches_per_build() + (group_ ? 2 : 1); }

    ErrorStatus check_status(cudaStream_t s) override
    {
        int nodes = 0;
        unsigned st = 0;
        GS_TRY(tree_.read_counts(s, &nodes, &st));
        if (st) GS_TRY(tree_.clear_status(s));
        if (st & ST_TREE_OVERFLOW)
            return GS_RAISE(GRAV_MEMORY_ERROR, "octree node capacity (%d) exceeded", tree_.cap_nodes);
        if (st & ST_STACK_OVERFLOW)
            return GS_RAISE(GRAV_FAILURE, "tree walk deeper than the octree depth limit");
        if (st & ST_WAIT_TIMEOUT)
            return GS_RAISE(GRAV_FAILURE, "octree key sort: a look-back wait ran out");
        return ok();
    }

    void set_build_timers(ForceTimer *morton, ForceTimer *sort) override
    {
        tree_.tm_morton = morton;
        tree_.tm_sort = sort;
    }

    ErrorStatus interaction_counts(cudaStream_t s, long long out[2]) override
    {
        unsigned long long h[2] = {0, 0};
        GS_CUDA(cudaMemcpyAsync(h, counters_.p, sizeof(h), cudaMemcpyDeviceToHost, s));
        GS_CUDA(cudaStreamSynchronize(s));
        out[0] = (long long)h[0];
        out[1] = (long long)h[1];
        return ok();
    }

  private:
    bool compat_, quad_, group_;
    int n_ = 0;
    double G_ = 1.0, eps_ = 0.0, theta_ = 1.0;
    OctreeDevice tree_;
    DBuf counters_;
};

}  // namespace

std::unique_ptr<Engine> make_barnes_hut_engine(bool compat, bool quad, bool group)
{
    return std::unique_ptr<Engine>(new BarnesHutEngine(compat, quad, group));
}

ErrorStatus accel_host(double *a, const System *system, const AccelerationParam *param_in);

// construct_octree on the GPU, copied to host arrays the caller frees with
// free_linear_octree (src/linear_octree.c:825-976).
ErrorStatus octree_to_host(const AccelerationParam &p_in, const System *system,
                           const double *box_center, double box_width, LinearOctree *out)
{
    if (!out) return GS_RAISE(GRAV_POINTER_ERROR, "Octree pointer is NULL");
    if (!system) return GS_RAISE(GRAV_POINTER_ERROR, "System pointer is NULL");
    if (system->num_particles <= 0 || !system->x || !system->m)
        return GS_RAISE(GRAV_VALUE_ERROR, "System has no particles");
    const int n = system->num_particles;
    const bool compat = p_in.method == ACCELERATION_METHOD_BARNES_HUT ||
                        p_in.method == GRAV_GPU_BARNES_HUT_COMPAT;
    int leaf = p_in.max_num_particles_per_leaf;
    if (leaf == -1) leaf = 1;
    if (leaf < 1)
        return GS_RAISE(GRAV_VALUE_ERROR,
                        "Maximum number of particles per leaf must be positive. Got: %d", leaf);
    OctreeDevice t;
    GS_TRY(t.setup(n, leaf, compat));
    DBuf dx, dm;
    GS_TRY(dx.reserve((size_t)n * 3 * sizeof(double)));
    GS_TRY(dm.reserve((size_t)n * sizeof(double)));
    cudaStream_t s = nullptr;
    GS_CUDA(cudaMemcpy(dx.p, system->x, (size_t)n * 3 * sizeof(double), cudaMemcpyHostToDevice));
    GS_CUDA(cudaMemcpy(dm.p, system->m, (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    GS_TRY(t.build(dx.as<double>(), dm.as<double>(), s, box_center, box_width));
    int nodes = 0;
    unsigned st = 0;
    GS_TRY(t.read_counts(s, &nodes, &st));
    if (st & ST_TREE_OVERFLOW)
        return GS_RAISE(GRAV_MEMORY_ERROR, "octree node capacity (%d) exceeded", t.cap_nodes);
    if (st & ST_WAIT_TIMEOUT)
        return GS_RAISE(GRAV_FAILURE, "octree key sort: a look-back wait ran out");
    LinearOctree o;
    std::memset(&o, 0, sizeof(o));
    o.num_internal_nodes = nodes;
    o.particle_morton_indices_deepest_level = (int64_t *)std::malloc((size_t)n * sizeof(int64_t));
    o.sorted_indices = (int *)std::malloc((size_t)n * sizeof(int));
    o.tree_num_particles = (int *)std::malloc((size_t)nodes * sizeof(int));
    o.tree_num_internal_children = (int *)std::malloc((size_t)nodes * sizeof(int));
    o.tree_first_particle_sorted_idx = (int *)std::malloc((size_t)nodes * sizeof(int));
    o.tree_first_internal_children_idx = (int *)std::malloc((size_t)nodes * sizeof(int));
    o.tree_mass = (double *)std::malloc((size_t)nodes * sizeof(double));
    o.tree_center_of_mass_x = (double *)std::malloc((size_t)nodes * sizeof(double));
    o.tree_center_of_mass_y = (double *)std::malloc((size_t)nodes * sizeof(double));
    o.tree_center_of_mass_z = (double *)std::malloc((size_t)nodes * sizeof(double));
    double *com = (double *)std::malloc((size_t)nodes * 3 * sizeof(double));
    double frame[8];
    if (!o.particle_morton_indices_deepest_level || !o.sorted_indices || !o.tree_num_particles ||
        !o.tree_num_internal_children || !o.tree_first_particle_sorted_idx ||
        !o.tree_first_internal_children_idx || !o.tree_mass || !o.tree_center_of_mass_x ||
        !o.tree_center_of_mass_y || !o.tree_center_of_mass_z || !com) {
        std::free(com);
        free_linear_octree(&o);
        return GS_RAISE(GRAV_MEMORY_ERROR, "Failed to allocate memory for the octree arrays");
    }
    cudaError_t e = cudaSuccess;
    e = e ? e : cudaMemcpy(o.particle_morton_indices_deepest_level, t.keys.p, (size_t)n * 8, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.sorted_indices, t.sidx.p, (size_t)n * 4, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.tree_num_particles, t.t_np.p, (size_t)nodes * 4, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.tree_num_internal_children, t.t_nc.p, (size_t)nodes * 4, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.tree_first_particle_sorted_idx, t.t_fp.p, (size_t)nodes * 4, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.tree_first_internal_children_idx, t.t_fc.p, (size_t)nodes * 4, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(o.tree_mass, t.t_mass.p, (size_t)nodes * 8, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(com, t.t_com.p, (size_t)nodes * 24, cudaMemcpyDeviceToHost);
    e = e ? e : cudaMemcpy(frame, t.frame.p, sizeof(frame), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        std::free(com);
        free_linear_octree(&o);
        GS_CUDA(e);
    }
    for (int i = 0; i < nodes; ++i) {
        o.tree_center_of_mass_x[i] = com[3 * i + 0];
        o.tree_center_of_mass_y[i] = com[3 * i + 1];
        o.tree_center_of_mass_z[i] = com[3 * i + 2];
    }
    std::free(com);
    o.box_width = frame[3];
    *out = o;
    return ok();
}

}  // namespace gs

using namespace gs;

extern "C" {

ErrorStatus acceleration_barnes_hut(double *a, const System *system,
                                    const AccelerationParam *acceleration_param)
{
    if (!acceleration_param)
        return GS_RAISE(GRAV_POINTER_ERROR, "Acceleration parameter pointer is NULL");
    AccelerationParam p = *acceleration_param;
    if (p.method == ACCELERATION_METHOD_BARNES_HUT || p.method == GRAV_GPU_BARNES_HUT_COMPAT)
        p.method = GRAV_GPU_BARNES_HUT_COMPAT;
    else
        p.method = GRAV_GPU_BARNES_HUT;
    return gs::accel_host(a, system, &p);
}

LinearOctree get_new_linear_octree(void)
{
    LinearOctree t;
    std::memset(&t, 0, sizeof(t));
    return t;
}

ErrorStatus construct_octree(LinearOctree *octree, const System *system,
                             const AccelerationParam *acceleration_param, const double *box_center,
                             double box_width)
{
    if (!acceleration_param)
        return GS_RAISE(GRAV_POINTER_ERROR, "Acceleration parameter pointer is NULL");
    return gs::octree_to_host(*acceleration_param, system, box_center, box_width, octree);
}

void free_linear_octree(LinearOctree *octree)
{
    if (!octree) return;
    std::free(octree->particle_morton_indices_deepest_level);
    std::free(octree->sorted_indices);
    std::free(octree->tree_num_particles);
    std::free(octree->tree_num_internal_children);
    std::free(octree->tree_first_particle_sorted_idx);
    std::free(octree->tree_first_internal_children_idx);
    std::free(octree->tree_mass);
    std::free(octree->tree_center_of_mass_x);
    std::free(octree->tree_center_of_mass_y);
    std::free(octree->tree_center_of_mass_z);
    std::memset(octree, 0, sizeof(*octree));
}

}  // extern "C"
