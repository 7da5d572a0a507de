// k_octree.cu -- GPU construction of grav_sim's linear octree.
//
// Replaces construct_octree and its helpers (src/linear_octree.c:113-962).
// Results equal the reference's: bounding box, Morton keys, sorted order,
// node numbering and topology bit for bit; internal-node mass and centre of
// mass bit for bit (FP64, reference summation order, no FMA contraction).
//
//   bounding box   k_bbox_partial + k_bbox_final: exact FP64 min/max.
//   Morton keys    k_morton: (x - c)/w + 0.5 in FP64, truncation to int64,
//                  21-bit mask (a coordinate at the box maximum wraps to 0,
//                  as in the reference), bit interleave.
//   sort           RadixSorter (stable LSD, 8-bit digits, one sweep per digit) of (key, id).
//   topology       from the sorted keys alone: which internal nodes start at a
//                  particle follows from three keys (k_tree_count, k_tree_emit);
//                  a child is internal when it holds more than leaf_max particles
//                  and is above depth 21.  k_tree_children finds each node's
//                  octants by binary search.
//   numbering      the reference numbers nodes in creation order: all
//                  children of a node get consecutive ids when the node is
//                  expanded, and nodes are expanded in depth-first pre-order.
//                  Pre-order of internal nodes is the order of (first
//                  particle, depth), the order in which they are emitted, so an
//                  exclusive scan of their child counts gives each one's
//                  first-child id (k_tree_nodes).
//   multipoles     bottom-up in one launch (arrival counters): an internal
//                  node adds, child by child in octant order, the particles
//                  of leaf children (sorted order) and the running sums of
//                  internal children -- the reference's order (:652-735).
//                  Leaves keep mass 0 and centre of mass 0 in compat mode
//                  (the reference's behaviour); otherwise they get their own
//                  sums.  The same kernels write the walk's node records and,
//                  for the quadrupole walks, FP32 quadrupoles.
// Every count the kernels need is read from device memory, so a whole build
// is graph-capturable.  Node-capacity overflow sets ST_TREE_OVERFLOW, which
// stays set until the host reports it; the kernels after the expansion then do
// no work (tree_failed / tree_nodes).
#include "gs_fp64.cuh"
#include "gs_octree.h"
#include "gs_ptx.cuh"

#include <cstdio>

namespace gs {

constexpr int OT_THREADS = 256;
constexpr int BBOX_BLOCKS = 512;

__device__ __forceinline__ double dmin(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double dmax(double a, double b) { return fmax(a, b); }

__global__ void __launch_bounds__(OT_THREADS)
k_bbox_partial(const double *__restrict__ x, int n, double *__restrict__ part)
{
    __shared__ double s[6][OT_THREADS];
    double lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = x[k];
        hi[k] = x[k];
    }
    for (int i = blockIdx.x * OT_THREADS + threadIdx.x; i < n; i += gridDim.x * OT_THREADS) {
        for (int k = 0; k < 3; ++k) {
            const double q = x[3 * i + k];
            lo[k] = dmin(lo[k], q);
            hi[k] = dmax(hi[k], q);
        }
    }
    for (int k = 0; k < 3; ++k) {
        s[k][threadIdx.x] = lo[k];
        s[3 + k][threadIdx.x] = hi[k];
    }
    __syncthreads();
    for (int w = OT_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            for (int k = 0; k < 3; ++k) {
                s[k][threadIdx.x] = dmin(s[k][threadIdx.x], s[k][threadIdx.x + w]);
                s[3 + k][threadIdx.x] = dmax(s[3 + k][threadIdx.x], s[3 + k][threadIdx.x + w]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = s[threadIdx.x][0];
}

// src/linear_octree.c:138-145 (and :856-867 when a box is given)
// One CTA of OT_THREADS threads: min / max are exact in any order, so the
// block partials are reduced as a tree.
__global__ void __launch_bounds__(OT_THREADS)
k_bbox_final(const double *__restrict__ part, int blocks, double ocx, double ocy, double ocz,
             double owidth, double *__restrict__ frame)
{
    __shared__ double s[6][OT_THREADS];
    double lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = part[k];
        hi[k] = part[3 + k];
    }
    for (int b = threadIdx.x; b < blocks; b += OT_THREADS)
        for (int k = 0; k < 3; ++k) {
            lo[k] = dmin(lo[k], part[6 * b + k]);
            hi[k] = dmax(hi[k], part[6 * b + 3 + k]);
        }
    for (int k = 0; k < 3; ++k) {
        s[k][threadIdx.x] = lo[k];
        s[3 + k][threadIdx.x] = hi[k];
    }
    __syncthreads();
    for (int w2 = OT_THREADS / 2; w2 > 0; w2 >>= 1) {
        if (threadIdx.x < w2) {
            for (int k = 0; k < 3; ++k) {
                s[k][threadIdx.x] = dmin(s[k][threadIdx.x], s[k][threadIdx.x + w2]);
                s[3 + k][threadIdx.x] = dmax(s[3 + k][threadIdx.x], s[3 + k][threadIdx.x + w2]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    for (int k = 0; k < 3; ++k) {
        lo[k] = s[k][0];
        hi[k] = s[3 + k][0];
    }
    double c[3], w;
    if (owidth > 0.0) {
        c[0] = ocx;
        c[1] = ocy;
        c[2] = ocz;
        w = owidth;
    } else {
        for (int k = 0; k < 3; ++k) c[k] = __ddiv_rn(__dadd_rn(hi[k], lo[k]), 2.0);
        w = dmax(dmax(__dsub_rn(hi[0], lo[0]), __dsub_rn(hi[1], lo[1])), __dsub_rn(hi[2], lo[2]));
    }
    frame[0] = c[0];
    frame[1] = c[1];
    frame[2] = c[2];
    frame[3] = w;
    frame[4] = __dmul_rn(w, 2.0);
    // the width's double-word reciprocal for div_by_width: zh = RN(1/w) and
    // zl = RN(1/w - zh), where 1 - zh w is exact (zh is correctly rounded)
    const double zh = __ddiv_rn(1.0, w);
    frame[5] = zh;
    frame[6] = __ddiv_rn(__fma_rn(-zh, w, 1.0), w);
    const double aw = fabs(w);
    frame[7] = (aw >= 0x1p-100 && aw <= 0x1p+100) ? 1.0 : 0.0;
}

// RN(x / w) for the box width w = frame[3] without a division, from the
// double-word reciprocal (frame[5], frame[6]) that k_bbox_final stored:
// q = RN(x zh + RN(x zl)) is within an ulp of x / w (Brisebarre, Muller and
// Raina, IEEE Trans. Computers 53(8), 2004), and the exact remainder
// r = x - q w corrects it to RN(q + r zh) = RN(x / w) (Markstein, IBM J.
// Res. Dev. 34(1), 1990).  The remainder is exact while its last bit stays
// above the subnormal range: |w| in [2^-100, 2^100] (frame[7]) and |x| in
// [2^-900, 2^900), tested on its exponent bits (an FP64 comparison costs the FP64
// pipe as much as an add); other operands (zeros, subnormals, infinities, NaN)
// take the division itself.  Checked against __ddiv_rn bit for bit by
// gsgpu_width_division_selftest.
__device__ __forceinline__ double div_by_width(double x, const double *__restrict__ frame)
{
    if (is_zero(frame[7]) || !exponent_within(x, 900)) return __ddiv_rn(x, frame[3]);
    const double q = __fma_rn(x, frame[5], __dmul_rn(x, frame[6]));
    const double r = __fma_rn(-q, frame[3], x);
    return __fma_rn(r, frame[5], q);
}

// 21 low bits of v spread to every third bit (magic-number interleave).
__device__ __forceinline__ uint64_t spread3(uint64_t v)
{
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x001f00000000ffffull;
    v = (v | (v << 16)) & 0x001f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// src/linear_octree.c:159-202
__global__ void k_morton(const double *__restrict__ x, int n, const double *__restrict__ frame,
                         uint64_t *__restrict__ keys, int *__restrict__ sidx,
                         unsigned char *__restrict__ misplaced)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t k = 0;
    bool out = false;   // a coordinate outside [0, 2^21) is masked: the key cell is elsewhere
    for (int d = 0; d < 3; ++d) {
        const double u = __dadd_rn(div_by_width(__dsub_rn(x[3 * i + d], frame[d]), frame), 0.5);
        const long long q = __double2ll_rz(__dmul_rn(u, 2097152.0));
        out = out || q < 0 || q > 0x1fffffll;
        k |= spread3((uint64_t)q) << d;
    }
    keys[i] = k;
    sidx[i] = i;
    misplaced[i] = out ? 1 : 0;
}

// ---- topology ---------------------------------------------------------------
// A cell of depth d that starts at sorted particle i is internal when the keys
// i .. i + leaf_max share its prefix, so the internal nodes that start at i are
// the depths from (levels shared with key i - 1) + 1 to (levels shared with key
// i + leaf_max), and their number needs three keys.  Their order by (first
// particle, depth) is the reference's depth-first pre-order, so an exclusive
// scan of those numbers over the particles gives every internal node its index:
// no level-by-level expansion and no sort of the nodes.
constexpr int TC_ITEMS = 8;
constexpr int TC_TILE = OT_THREADS * TC_ITEMS;   // particles per scan tile
constexpr int TN_ROUND = OT_THREADS / 8;         // internal nodes a CTA works on at once
constexpr int TN_ROUNDS = 8;                     // rounds per scan tile at most
constexpr int TN_GRID = 4;                       // CTAs per SM of the kernels over nodes
constexpr int TN_MANY = 2;                       // tiles per CTA from which a tile takes more rounds

// Internal nodes per scan tile of a tree with ni of them, on a grid of `ctas`.  A
// round is a chain of dependent loads (the searches of the octants' ends), so a small
// tree takes one round per tile: eight rounds left 8 of 152 SMs with work at 60,000
// particles and 16 per leaf (38 us, now 11).  With more than TN_MANY tiles a CTA (eight
// an SM) tiles grow with the tree, so that their scan, by one CTA, stays short.
__device__ __forceinline__ int node_tile(int ni, int ctas)
{
    return TN_ROUND * min(TN_ROUNDS, 1 + ni / (TN_ROUND * TN_MANY * ctas));
}

// Levels (octant digits) shared by two 63-bit keys.
__device__ __forceinline__ int shared_levels(uint64_t a, uint64_t b)
{
    const uint64_t x = a ^ b;
    return x ? (62 - (63 - __clzll((long long)x))) / 3 : OCT_MAX_LEVEL;
}

// Depths [lo, hi] of the internal nodes that start at particle i (none when
// hi < lo).  The root is internal whatever its count.
__device__ __forceinline__ void internal_depths(const uint64_t *__restrict__ keys, int n,
                                                int leaf_max, int i, int &lo, int &hi)
{
    const uint64_t k = keys[i];
    lo = i == 0 ? 0 : shared_levels(keys[i - 1], k) + 1;
    hi = leaf_max < n - i ? min(OCT_MAX_LEVEL - 1, shared_levels(k, keys[i + leaf_max])) : -1;
    if (i == 0) hi = max(hi, 0);
}

// Exclusive prefix of v over the CTA's threads; every thread also gets the sum.
__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned &sum)
{
    __shared__ unsigned wsum[OT_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    unsigned before = 0;
    sum = 0;
    for (int q = 0; q < OT_THREADS / 32; ++q) {
        before += q < w ? wsum[q] : 0u;
        sum += wsum[q];
    }
    __syncthreads();
    return before + incl - v;
}

// The CTA that is the last of the grid to come here returns true in all its
// threads (and sees what the others wrote before); the counter is left at 0.
__device__ __forceinline__ bool last_block(int *counter)
{
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
        if (last) *counter = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// tile[0 .. tiles) -> its exclusive scan, by one CTA; returns the total.
__device__ unsigned long long scan_tiles_inplace(unsigned *tile, int tiles)
{
    unsigned long long run = 0;
    for (int b = 0; b < tiles; b += OT_THREADS) {
        const int t = b + (int)threadIdx.x;
        unsigned sum;
        const unsigned before = block_exclusive(t < tiles ? __ldcg(tile + t) : 0u, sum);
        if (t < tiles) tile[t] = (unsigned)run + before;   // meaningful while the total fits
        run += sum;
    }
    return run;
}

// Internal nodes per tile of particles, and their scan by the last CTA.
__global__ void __launch_bounds__(OT_THREADS)
k_tree_count(const uint64_t *__restrict__ keys, int n, int leaf_max, int cap,
             unsigned *__restrict__ tile_sum, int *__restrict__ ctr)
{
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < TC_ITEMS; ++k) {
        const int i = blockIdx.x * TC_TILE + k * OT_THREADS + threadIdx.x;
        if (i < n) {
            int lo, hi;
            internal_depths(keys, n, leaf_max, i, lo, hi);
            c += max(0, hi - lo + 1);
        }
    }
    unsigned sum;
    (void)block_exclusive(c, sum);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = sum;
    if (!last_block(&ctr[CTR_DONE])) return;
    const unsigned long long total = scan_tiles_inplace(tile_sum, gridDim.x);
    if (threadIdx.x == 0) {
        // every internal node but the root is a node, and has a child
        if (total >= (unsigned long long)cap)
            atomicOr((unsigned *)&ctr[CTR_STATUS], ST_TREE_OVERFLOW);
        const bool failed = tree_failed(ctr);
        ctr[CTR_INTERNAL] = failed ? 0 : (int)total;
        ctr[CTR_SAFE_INTERNAL] = failed ? 0 : (int)total;
    }
}

// Index of the first internal node at or after each particle (pre_of), and
// each internal node's (first particle, depth).
__global__ void __launch_bounds__(OT_THREADS)
k_tree_emit(const uint64_t *__restrict__ keys, int n, int leaf_max,
            const unsigned *__restrict__ tile_off, const int *__restrict__ ctr,
            int *__restrict__ pre_of, int2 *__restrict__ in_sd)
{
    if (tree_failed(ctr)) return;
    const int i0 = blockIdx.x * TC_TILE + threadIdx.x * TC_ITEMS;
    int lo[TC_ITEMS], cnt[TC_ITEMS];
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < TC_ITEMS; ++k) {
        lo[k] = cnt[k] = 0;
        if (i0 + k < n) {
            int hi;
            internal_depths(keys, n, leaf_max, i0 + k, lo[k], hi);
            cnt[k] = max(0, hi - lo[k] + 1);
        }
        c += cnt[k];
    }
    unsigned sum;
    int at = (int)(tile_off[blockIdx.x] + block_exclusive(c, sum));
#pragma unroll
    for (int k = 0; k < TC_ITEMS; ++k) {
        if (i0 + k >= n) break;
        pre_of[i0 + k] = at;
        for (int q = 0; q < cnt[k]; ++q) in_sd[at + q] = make_int2(i0 + k, lo[k] + q);
        at += cnt[k];
    }
}

// First index after s whose key, shifted, exceeds `limit`: steps of a factor
// of eight from s (most nodes hold few particles), then a binary search.
__device__ __forceinline__ int prefix_end(const uint64_t *__restrict__ keys, int s, int n,
                                          int shift, uint64_t limit)
{
    int lo = s, hi = n;   // the answer lies in [lo, hi]
    for (long long step = 8;; step *= 8) {
        const long long at = s + step;
        if (at >= n) break;
        if ((keys[at] >> shift) > limit) {
            hi = (int)at;
            break;
        }
        lo = (int)at + 1;
    }
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if ((keys[mid] >> shift) > limit)
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

// Children of every internal node (src/linear_octree.c:342-576): eight lanes
// per node, one per octant, each finds where its octant ends.  in_end[8 ii + o]
// receives the ends, in_nch[ii] the non-empty octants; the last CTA scans the
// children over the tiles of nodes, which gives the node total.
__global__ void __launch_bounds__(OT_THREADS)
k_tree_children(const uint64_t *__restrict__ keys, int n, int cap, const int2 *__restrict__ in_sd,
                int *__restrict__ in_end, int *__restrict__ in_nch,
                unsigned *__restrict__ tile_sum, int *__restrict__ ctr)
{
    const int ni = ctr[CTR_SAFE_INTERNAL];
    const int lane = threadIdx.x & 31, o = lane & 7, g0 = lane & ~7;
    const int size = node_tile(ni, gridDim.x), tiles = (ni + size - 1) / size;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        unsigned mine = 0;
        for (int q = 0; q < size; q += TN_ROUND) {
            const int ii = tile * size + q + (threadIdx.x >> 3);
            const bool act = ii < ni;
            int s = 0, end = 0;
            if (act) {
                const int2 sd = in_sd[ii];
                s = sd.x;
                const int shift = 3 * (OCT_MAX_LEVEL - 1 - sd.y);
                end = prefix_end(keys, s, n, shift, ((keys[s] >> shift) & ~7ull) | (uint64_t)o);
                in_end[8 * (size_t)ii + o] = end;
            }
            const int up = __shfl_up_sync(0xffffffffu, end, 1, 8);
            const bool has = act && end > (o == 0 ? s : up);
            const int nch = __popc((__ballot_sync(0xffffffffu, has) >> g0) & 0xffu);
            if (act && o == 0) {
                in_nch[ii] = nch;
                mine += nch;
            }
        }
        unsigned sum;
        (void)block_exclusive(mine, sum);
        if (threadIdx.x == 0) tile_sum[tile] = sum;
    }
    if (!last_block(&ctr[CTR_DONE])) return;
    const unsigned long long total = scan_tiles_inplace(tile_sum, tiles) + 1ull;
    if (threadIdx.x == 0) {
        if (total > (unsigned long long)cap) {
            atomicOr((unsigned *)&ctr[CTR_STATUS], ST_TREE_OVERFLOW);
            ctr[CTR_SAFE_INTERNAL] = 0;
        }
        ctr[CTR_NODES] = tree_failed(ctr) ? 1 : (int)total;
    }
}

// Node arrays by id: the children of internal node ii take the ids from
// first child = 1 + (children of the internal nodes before it), in octant
// order, which is the reference's creation order.  in_rec[ii] is (first child,
// children | internal ones' mask << 8, parent, id); a child's half of it is
// written by its parent.
__global__ void __launch_bounds__(OT_THREADS)
k_tree_nodes(int n, int leaf_max, const unsigned *__restrict__ tile_off,
             const int *__restrict__ ctr, const int2 *__restrict__ in_sd,
             const int *__restrict__ in_end, const int *__restrict__ in_nch,
             const int *__restrict__ pre_of, int4 *__restrict__ in_rec, int *__restrict__ in_arrive,
             int *__restrict__ t_np, int *__restrict__ t_fp, int *__restrict__ t_depth,
             int *__restrict__ t_int)
{
    __shared__ int s_fc[TN_ROUND * TN_ROUNDS];
    const int ni = ctr[CTR_SAFE_INTERNAL];
    const int lane = threadIdx.x & 31, o = lane & 7, g0 = lane & ~7;
    const int size = node_tile(ni, gridDim.x), tiles = (ni + size - 1) / size;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int mine = tile * size + (int)threadIdx.x;
        unsigned sum;
        const unsigned before = block_exclusive(
            (int)threadIdx.x < size && mine < ni ? (unsigned)in_nch[mine] : 0u, sum);
        s_fc[threadIdx.x] = 1 + (int)(tile_off[tile] + before);
        __syncthreads();
        for (int q = 0; q < size; q += TN_ROUND) {
            const int local = q + (int)(threadIdx.x >> 3);
            const int ii = tile * size + local;
            const bool act = ii < ni;
            int2 sd = make_int2(0, 0);
            int end = 0;
            if (act) {
                sd = in_sd[ii];
                end = in_end[8 * (size_t)ii + o];
            }
            const int up = __shfl_up_sync(0xffffffffu, end, 1, 8);
            const int start = o == 0 ? sd.x : up;
            const int cnt = act ? end - start : 0;
            const int cd = sd.y + 1;
            const bool inner = cnt > leaf_max && cd < OCT_MAX_LEVEL;
            const unsigned m8 = (__ballot_sync(0xffffffffu, cnt > 0) >> g0) & 0xffu;
            const int rank = __popc(m8 & ((1u << o) - 1u));
            unsigned imask = inner ? 1u << rank : 0u;
            for (int w = 1; w < 8; w <<= 1) imask |= __shfl_xor_sync(0xffffffffu, imask, w, 8);
            if (!act) continue;
            const int fc = s_fc[local];
            int2 *rec = reinterpret_cast<int2 *>(in_rec);
            if (o == 0) {
                rec[2 * (size_t)ii] = make_int2(fc, __popc(m8) | (int)(imask << 8));
                in_arrive[ii] = 0;
                if (ii == 0) {
                    rec[1] = make_int2(-1, 0);
                    t_np[0] = n;
                    t_fp[0] = 0;
                    t_depth[0] = 0;
                    t_int[0] = 0;
                }
            }
            if (cnt > 0) {
                const int id = fc + rank;
                // the child's own index: the next one when it starts where
                // this node does, else the first one of its first particle
                const int ci = start == sd.x ? ii + 1 : pre_of[start];
                t_np[id] = cnt;
                t_fp[id] = start;
                t_depth[id] = cd;
                t_int[id] = inner ? ci : -1;
                if (inner) rec[2 * (size_t)ci + 1] = make_int2(ii, id);
            }
        }
        __syncthreads();
    }
}

// Parent id of every node and the leaf of every sorted particle (used by
// the learned method's features).
__global__ void k_tree_links(const int *__restrict__ ctr, const int4 *__restrict__ in_rec,
                             const int *__restrict__ t_np, const int *__restrict__ t_fp,
                             const int *__restrict__ t_int, int *__restrict__ t_parent,
                             int *__restrict__ leaf_of)
{
    const int ni = ctr[CTR_SAFE_INTERNAL];
    for (int ii = blockIdx.x * blockDim.x + threadIdx.x; ii < ni; ii += gridDim.x * blockDim.x) {
        const int4 r = in_rec[ii];
        if (ii == 0) t_parent[0] = -1;
        for (int c = r.x; c < r.x + (r.y & 255); ++c) {
            t_parent[c] = r.w;
            if (t_int[c] < 0)
                for (int p = t_fp[c]; p < t_fp[c] + t_np[c]; ++p) leaf_of[p] = c;
        }
    }
}

// Mass and mass-weighted coordinate sums of sorted particles [first,
// first + count) in sorted order (reference :667-674), from the sorted
// (m, m x, m y, m z) records: four ordered additions per particle.  The products
// are the ones the reference forms inside the sum; formed once per particle when
// the records are written, they need not be formed again for the leaf and for
// its parent (7 and 2 FP64 instructions per particle before; k_leaf_multipoles
// 90 and 65 us at N = 1,048,576).
__device__ __forceinline__ void add_particles(const double *__restrict__ mx, int first, int count,
                                              double &M, double &S0, double &S1, double &S2)
{
#pragma unroll 4
    for (int p = first; p < first + count; ++p) {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(mx + 4 * (size_t)p));
        const double2 b = __ldg(reinterpret_cast<const double2 *>(mx + 4 * (size_t)p) + 1);
        M = __dadd_rn(M, a.x);
        S0 = __dadd_rn(S0, a.y);
        S1 = __dadd_rn(S1, b.x);
        S2 = __dadd_rn(S2, b.y);
    }
}

// acc plus the values q[4 p] of p in [p0, p1), in order; eight loads are in
// flight while eight values are added, so that the chain of additions waits for
// the first eight only.
__device__ __forceinline__ double add_run(double acc, const double *__restrict__ q, int p0, int p1)
{
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = p0 + u < p1 ? __ldg(q + 4 * (size_t)(p0 + u)) : 0.0;
    for (int p = p0; p < p1; p += 8) {
        double w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) w[u] = p + 8 + u < p1 ? __ldg(q + 4 * (size_t)(p + 8 + u)) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (p + u < p1) acc = __dadd_rn(acc, v[u]);
            v[u] = w[u];
        }
    }
    return acc;
}

__device__ __forceinline__ void split_df(double v, float &hi, float &lo)
{
    hi = __double2float_rn(v);
    lo = __double2float_rn(__dsub_rn(v, (double)hi));
}

// (cell side)^2 at depth d, box_length / (2 << d), for the group walk's
// opening test.  The divisor is a power of two, so the product with its
// exact reciprocal (built from the exponent bits) equals the quotient.
__device__ __forceinline__ float cell_side2(const double *__restrict__ frame, int depth)
{
    const int e = min(depth, OCT_MAX_LEVEL + 1) + 1;
    const double side = __dmul_rn(frame[4], __longlong_as_double((long long)(1023 - e) << 52));
    return (float)(side * side);
}

// Walk record of a node: centre of mass relative to the frame centre as
// (hi, lo) FP32 pairs, FP32 mass, (cell side)^2.  The same arithmetic for
// every node, whichever kernel computes its multipoles.
__device__ __forceinline__ void write_node_record(int id, double M, double c0, double c1, double c2,
                                                  int depth, const double *__restrict__ frame,
                                                  float4 *na, float4 *nb, float h[3], float l[3])
{
    split_df(__dsub_rn(c0, frame[0]), h[0], l[0]);
    split_df(__dsub_rn(c1, frame[1]), h[1], l[1]);
    split_df(__dsub_rn(c2, frame[2]), h[2], l[2]);
    na[id] = make_float4(h[0], h[1], h[2], (float)M);
    nb[id] = make_float4(l[0], l[1], l[2], cell_side2(frame, depth));
}

// m (3 d d^T - |d|^2 I) added to the packed quadrupole (xx, xy, xz, yy, yz, zz).
__device__ __forceinline__ void add_quad(float Q[6], float mp, float d0, float d1, float d2)
{
    const float r2 = d0 * d0 + d1 * d1 + d2 * d2;
    const float m3 = 3.0f * mp;
    Q[0] += mp * (3.0f * d0 * d0 - r2);
    Q[1] += m3 * d0 * d1;
    Q[2] += m3 * d0 * d2;
    Q[3] += mp * (3.0f * d1 * d1 - r2);
    Q[4] += m3 * d1 * d2;
    Q[5] += mp * (3.0f * d2 * d2 - r2);
}

__device__ __forceinline__ void store_quad(float4 *nq, int id, const float Q[6])
{
    nq[2 * (size_t)id] = make_float4(Q[0], Q[1], Q[2], Q[3]);
    nq[2 * (size_t)id + 1] = make_float4(Q[4], Q[5], 0.0f, 0.0f);
}

// Offset of a (hi, lo) FP32 pair point from a (hi, lo) centre, in FP32:
// the hi parts of points in one cell are close, so their difference is
// exact, and the lo parts carry the rest.
__device__ __forceinline__ float df_offset(float ph, float pl, float ch, float cl)
{
    return (ph - ch) + (pl - cl);
}

struct MultipoleArgs {
    const double *mx;   // sorted (m, m x, m y, m z) records
    const int4 *in_rec; // internal nodes: (first child, children | inner mask << 8, parent, id)
    const int4 *nc;     // nodes: (first child, children, first particle, particles)
    const int *t_depth;
    const double *frame;
    int *in_arrive;
    double *t_sum, *t_mass, *t_com;   // t_sum: (m, m x, m y, m z) of internal nodes by id
    float4 *na, *nb, *nq;   // nq null: no quadrupoles
};

// Multipoles of the internal node of record rec from its children (reference
// :652-735): mass and the mass-weighted coordinate sums in child order, the
// centre of mass by division, its walk record, and, when nq is not null, the
// quadrupole from the children's by the parallel-axis shift
// Q = sum_c [Q_c + M_c (3 s s^T - |s|^2 I)], s = com_c - com, in FP32 from the
// children's walk records (FP64 runs at 1/64 of the FP32 rate here, and the walk
// uses FP32 quadrupoles).  Children's values written by other threads of the
// same launch are read through L2 (__ldcg), after the acquire on the
// arrival counter.
//
// A node is computed by the four lanes of a group: lane j keeps one of the
// four ordered sums (j = 0 the mass, j = 1..3 the sums of m x, m y, m z), so
// a particle costs one FP64 addition for all four sums, and the three quotients
// are one division.  Each sum sees the same operands in the same order as a
// one-thread loop would, so the values are the same bit for bit.
//
// Near the root a single group climbs alone, and what bounds it is the chain of
// dependent loads of each level.  The record and the sums are laid out so that
// a level is one round of loads: the record says which children are internal,
// their sums are indexed by node id, and all of them, the leaf children's
// particle ranges and the children's quadrupoles (two children a lane) are
// issued before the first is used; the caller loads the parent's record
// meanwhile.  With child type, index and sums each behind the other, eight times
// in a row, a level took about 17 us and the kernel 309 us at N = 60,000 and
// 311 us at N = 1,048,576; with the quadrupoles in a round of their own and
// the particles of leaf children four at a time 103 and 157 us; now 55 and 91.
template <bool QUAD>
__device__ __forceinline__ void multipole_node4(const int4 rec, int j, unsigned gmask, const MultipoleArgs &A)
{
    const int fc = rec.x, nch = rec.y & 255, inner = rec.y >> 8, id = rec.w;
    // this lane's sum of every internal child, the particles of every leaf child
    __shared__ double s_sum[8][OT_THREADS];
    __shared__ int2 s_leaf[8][OT_THREADS];
    {
        double v[8];
        int2 leaf[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            v[r] = 0.0;
            leaf[r] = make_int2(0, 0);
            if (r < nch) {
                if ((inner >> r) & 1)
                    v[r] = __ldcg(A.t_sum + 4 * (size_t)(fc + r) + j);
                else
                    leaf[r] = reinterpret_cast<const int2 *>(A.nc + fc + r)[1];
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            s_sum[r][threadIdx.x] = v[r];
            s_leaf[r][threadIdx.x] = leaf[r];
        }
    }
    // quadrupoles of children j and j + 4
    float4 ca[2], cb[2], qa[2], qb[2];
    if (QUAD) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (j + 4 * k < nch) {
                const size_t c = fc + j + 4 * k;
                ca[k] = __ldcg(A.na + c);
                cb[k] = __ldcg(A.nb + c);
                qa[k] = __ldcg(A.nq + 2 * c);
                qb[k] = __ldcg(A.nq + 2 * c + 1);
            }
    }
    // children in order; the particles of consecutive leaf children are one run
    double acc = 0.0;
    for (int r = 0; r < nch;) {
        int p0 = 0, p1 = 0;
        for (; r < nch && !((inner >> r) & 1); ++r) {
            const int2 leaf = s_leaf[r][threadIdx.x];
            if (p1 <= p0) p0 = leaf.x;
            p1 = leaf.x + leaf.y;
        }
        acc = add_run(acc, A.mx + j, p0, p1);
        for (; r < nch && ((inner >> r) & 1); ++r) acc = __dadd_rn(acc, s_sum[r][threadIdx.x]);
    }
    A.t_sum[4 * (size_t)id + j] = acc;
    const double M = __shfl_sync(gmask, acc, 0, 4);
    const double cj = __ddiv_rn(acc, M);   // lanes 1..3: coordinate j - 1 of the centre
    float hj = 0.0f, lj = 0.0f;
    if (j == 0) {
        A.t_mass[id] = M;
    } else {
        A.t_com[3 * (size_t)id + j - 1] = cj;
        split_df(__dsub_rn(cj, A.frame[j - 1]), hj, lj);
    }
    float h[3], l[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        h[k] = __shfl_sync(gmask, hj, k + 1, 4);
        l[k] = __shfl_sync(gmask, lj, k + 1, 4);
    }
    if (j == 0) {
        A.na[id] = make_float4(h[0], h[1], h[2], (float)M);
        A.nb[id] = make_float4(l[0], l[1], l[2], cell_side2(A.frame, A.t_depth[id]));
    }
    if (QUAD) {
        float Q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 2; ++k)
            // a massless child (no centre of mass: 0 / 0) adds nothing
            if (j + 4 * k < nch && !(ca[k].w == 0.0f && isnan(ca[k].x))) {
                add_quad(Q, ca[k].w, df_offset(ca[k].x, cb[k].x, h[0], l[0]),
                         df_offset(ca[k].y, cb[k].y, h[1], l[1]),
                         df_offset(ca[k].z, cb[k].z, h[2], l[2]));
                Q[0] += qa[k].x;
                Q[1] += qa[k].y;
                Q[2] += qa[k].z;
                Q[3] += qa[k].w;
                Q[4] += qb[k].x;
                Q[5] += qb[k].y;
            }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            Q[q] += __shfl_xor_sync(gmask, Q[q], 1, 4);
            Q[q] += __shfl_xor_sync(gmask, Q[q], 2, 4);
        }
        if (j == 0) store_quad(A.nq, id, Q);
    }
}

// All internal nodes in one launch, bottom-up.  A group of four lanes starts
// at each internal node none of whose children is internal, computes it, and
// climbs: it counts itself in the parent's arrival counter, and the group that
// completes the count (the last of the parent's internal children to finish)
// computes the parent.  Nothing waits: a group that is not last stops.  Every
// node is computed once, by the same arithmetic in the same child order as a
// level-by-level pass, so the sums are identical to it.  Every decision below
// is the same for the four lanes of a group (they share the node), so the
// group's shuffles and barriers see all four.  Two CTAs per SM with quadrupoles
// (three or four: the registers of the loads in flight spill, 8 to 17 us longer at
// N = 60,000), four without (95 us at N = 150,000 with one particle per leaf,
// three and six 109).
template <bool QUAD>
__global__ void __launch_bounds__(OT_THREADS, QUAD ? 2 : 4) k_multipole_up(const int *__restrict__ ctr,
                                                             MultipoleArgs A)
{
    const int ni = ctr[CTR_SAFE_INTERNAL];
    const int j = threadIdx.x & 3;
    const unsigned gmask = 0xFu << ((threadIdx.x & 31) & ~3);
    const int groups = (gridDim.x * blockDim.x) >> 2;
    for (int i0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; i0 < ni; i0 += groups) {
        int4 rec = A.in_rec[i0];
        if (rec.y >> 8) continue;   // has internal children
        for (;;) {
            const int p = rec.z;
            const int4 up = p >= 0 ? A.in_rec[p] : make_int4(0, 0, 0, 0);
            multipole_node4<QUAD>(rec, j, gmask, A);
            if (p < 0) break;
            // The lanes' writes happen before the barrier, and lane 0's release
            // makes them visible with its own; its acquire orders the other
            // groups' writes before the reads below.
            __syncwarp(gmask);
            int arrived = 0;
            if (j == 0)
                asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;"
                             : "=r"(arrived)
                             : "l"(A.in_arrive + p)
                             : "memory");
            arrived = __shfl_sync(gmask, arrived, 0, 4);
            if (arrived != __popc(up.y >> 8) - 1) break;
            __syncwarp(gmask);
            rec = up;
        }
    }
}

// Every node: its walk record (first child, children, first particle,
// particles) and the membership key the per-particle walks read.
// Leaves get their own mass and centre of mass (non-compat trees; zero in a
// compat tree), their walk records, and, when nq is not null, their quadrupole
// sum_p m (3 d d^T - |d|^2 I) about the centre of mass, from the particles'
// (hi, lo) FP32 pairs.
__global__ void k_leaf_multipoles(const int *__restrict__ ctr, int compat, MultipoleArgs A,
                                  const float4 *__restrict__ pa, const float4 *__restrict__ pb,
                                  const uint64_t *__restrict__ keys, const int *__restrict__ sidx,
                                  const int *__restrict__ t_np, const int *__restrict__ t_fp,
                                  const int *__restrict__ t_int, int *__restrict__ t_nc,
                                  int *__restrict__ t_fc, int4 *__restrict__ nc,
                                  uint64_t *__restrict__ nkey)
{
    const int nn = tree_nodes(ctr);
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < nn; id += gridDim.x * blockDim.x) {
        const int fp = t_fp[id], np = t_np[id], ii = t_int[id];
        const int2 kids = ii >= 0 ? *reinterpret_cast<const int2 *>(A.in_rec + ii) : make_int2(-1, 0);
        t_fc[id] = kids.x;
        t_nc[id] = kids.y & 255;
        nc[id] = make_int4(kids.x, kids.y & 255, fp, np);
        // the reference's membership test reads keys[sorted_indices[first]]
        // from the sorted key array (src/acceleration_barnes_hut.c:145)
        nkey[id] = compat ? keys[sidx[fp]] : keys[fp];
        if (ii >= 0) continue;
        double M = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0;
        if (!compat) {
            double S0 = 0.0, S1 = 0.0, S2 = 0.0;
            add_particles(A.mx, fp, np, M, S0, S1, S2);
            c0 = __ddiv_rn(S0, M);
            c1 = __ddiv_rn(S1, M);
            c2 = __ddiv_rn(S2, M);
        }
        A.t_mass[id] = M;
        A.t_com[3 * (size_t)id + 0] = c0;
        A.t_com[3 * (size_t)id + 1] = c1;
        A.t_com[3 * (size_t)id + 2] = c2;
        float h[3], l[3];
        write_node_record(id, M, c0, c1, c2, A.t_depth[id], A.frame, A.na, A.nb, h, l);
        if (A.nq) {
            float Q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int p = fp; p < fp + np; ++p) {
                const float4 a = pa[p], b = pb[p];
                add_quad(Q, a.w, df_offset(a.x, b.x, h[0], l[0]), df_offset(a.y, b.y, h[1], l[1]),
                         df_offset(a.z, b.z, h[2], l[2]));
            }
            store_quad(A.nq, id, Q);
        }
    }
}

__global__ void k_walk_particles(int n, const double *__restrict__ frame, const double *__restrict__ x,
                                 const double *__restrict__ m, const int *__restrict__ sidx,
                                 float4 *__restrict__ pa, float4 *__restrict__ pb,
                                 double *__restrict__ mx,
                                 const unsigned char *__restrict__ misplaced,
                                 int *__restrict__ mlist)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int id = sidx[p];
    if (misplaced[id]) {   // rare: the count, and the sorted positions of the first ones
        const int at = atomicAdd(&mlist[0], 1);
        if (at < kMisplacedCap) mlist[1 + at] = p;
    }
    const double mp = m[id];
    double2 *out = reinterpret_cast<double2 *>(mx + 4 * (size_t)p);
    out[0] = make_double2(mp, __dmul_rn(mp, x[3 * id + 0]));
    out[1] = make_double2(__dmul_rn(mp, x[3 * id + 1]), __dmul_rn(mp, x[3 * id + 2]));
    float h0, l0, h1, l1, h2, l2;
    split_df(__dsub_rn(x[3 * id + 0], frame[0]), h0, l0);
    split_df(__dsub_rn(x[3 * id + 1], frame[1]), h1, l1);
    split_df(__dsub_rn(x[3 * id + 2], frame[2]), h2, l2);
    pa[p] = make_float4(h0, h1, h2, (float)mp);
    pb[p] = make_float4(l0, l1, l2, 0.0f);
}

// ------------------------------------------------------------------------
ErrorStatus OctreeDevice::setup(int n_, int leaf_max_, bool compat_, bool quad_)
{
    n = n_;
    leaf_max = leaf_max_;
    compat = compat_;
    quad = quad_ && !compat_;
    int cap = 4 * n + 4096;
    if (cap < n) return GS_RAISE(GRAV_VALUE_ERROR, "too many particles for the octree: %d", n);
    cap_nodes = cap;
    const size_t ci = (size_t)cap * sizeof(int);
    GS_TRY(ctr.reserve(CTR_SIZE * sizeof(int)));
    int c0[CTR_SIZE] = {};   // status word clear, no CTA counted
    c0[CTR_N] = n;
    GS_CUDA(cudaMemcpy(ctr.p, c0, sizeof(c0), cudaMemcpyHostToDevice));
    GS_TRY(frame.reserve(8 * sizeof(double)));
    GS_TRY(bbox_part.reserve((size_t)BBOX_BLOCKS * 6 * sizeof(double)));
    GS_TRY(keys.reserve((size_t)n * sizeof(uint64_t)));
    GS_TRY(sidx.reserve((size_t)n * sizeof(int)));
    DBuf *ints[] = {&in_nch, &in_arrive, &t_np, &t_nc, &t_fp, &t_fc, &t_depth, &t_int};
    for (DBuf *b : ints) GS_TRY(b->reserve(ci));
    GS_TRY(pre_of.reserve((size_t)n * sizeof(int)));
    GS_TRY(in_sd.reserve((size_t)cap * sizeof(int2)));
    GS_TRY(in_end.reserve((size_t)cap * 8 * sizeof(int)));
    GS_TRY(in_rec.reserve((size_t)cap * sizeof(int4)));
    const DeviceInfo *dev = nullptr;
    GS_TRY(device_info(&dev));
    const int small_tiles = TN_MANY * TN_GRID * dev->sm_count + TN_ROUNDS;
    GS_TRY(scan_tiles.reserve(
        (size_t)(std::max(std::max((n + TC_TILE - 1) / TC_TILE, small_tiles),
                          cap / (TN_ROUND * TN_ROUNDS) + 1) +
                 1) *
        sizeof(unsigned)));
    GS_TRY(t_mass.reserve((size_t)cap * sizeof(double)));
    GS_TRY(t_com.reserve((size_t)cap * 3 * sizeof(double)));
    GS_TRY(t_sum.reserve((size_t)cap * 4 * sizeof(double)));
    GS_TRY(w_na.reserve((size_t)cap * sizeof(float4)));
    GS_TRY(w_nb.reserve((size_t)cap * sizeof(float4)));
    GS_TRY(w_nc.reserve((size_t)cap * sizeof(int4)));
    GS_TRY(w_nkey.reserve((size_t)cap * sizeof(uint64_t)));
    GS_TRY(misplaced.reserve((size_t)n));
    GS_TRY(mlist.reserve((size_t)(1 + kMisplacedCap) * sizeof(int)));
    GS_TRY(w_pa.reserve((size_t)n * sizeof(float4)));
    GS_TRY(w_pb.reserve((size_t)n * sizeof(float4)));
    GS_TRY(mx.reserve((size_t)n * 4 * sizeof(double)));
    GS_TRY(g_list.reserve((size_t)n * sizeof(int2)));
    GS_TRY(g_ctr.reserve(4 * sizeof(int)));
    if (quad) GS_TRY(w_nq.reserve((size_t)cap * 2 * sizeof(float4)));
    if (links) {
        GS_TRY(t_parent.reserve((size_t)cap * sizeof(int)));
        GS_TRY(leaf_of.reserve((size_t)n * sizeof(int)));
    }
    GS_TRY(sorter.reserve(n));
    return ok();
}

int OctreeDevice::launches_per_build() const
{
    // bbox 2, morton 1, sort, topology 4, walk particles 1, leaves 1,
    // multipoles 1
    return 2 + 1 + RadixSorter::launches(63) + 4 + 1 + 1 + 1 + (links ? 1 : 0);
}

ErrorStatus OctreeDevice::build(const double *d_x, const double *d_m, cudaStream_t s,
                                const double *box_center, double box_width)
{
    const int nb = std::min(BBOX_BLOCKS, std::max(1, (n + OT_THREADS - 1) / OT_THREADS));
    k_bbox_partial<<<nb, OT_THREADS, 0, s>>>(d_x, n, bbox_part.as<double>());
    const bool own_box = box_center && box_width > 0.0;
    k_bbox_final<<<1, OT_THREADS, 0, s>>>(bbox_part.as<double>(), nb, own_box ? box_center[0] : 0.0,
                                  own_box ? box_center[1] : 0.0, own_box ? box_center[2] : 0.0,
                                  own_box ? box_width : -1.0, frame.as<double>());
    const int pb = (n + OT_THREADS - 1) / OT_THREADS;
    if (tm_morton) GS_TRY(tm_morton->begin(s));
    k_morton<<<pb, OT_THREADS, 0, s>>>(d_x, n, frame.as<double>(), keys.as<uint64_t>(),
                                       sidx.as<int>(), misplaced.as<unsigned char>());
    if (tm_morton) GS_TRY(tm_morton->end(s));
    GS_CUDA(cudaGetLastError());
    if (tm_sort) GS_TRY(tm_sort->begin(s));
    GS_TRY(sorter.sort(keys.as<uint64_t>(), sidx.as<int>(), ctr.as<int>() + CTR_N, n, 63,
                       reinterpret_cast<unsigned *>(ctr.as<int>() + CTR_STATUS), s));
    if (tm_sort) GS_TRY(tm_sort->end(s));

    const DeviceInfo *dev = nullptr;
    GS_TRY(device_info(&dev));
    // Kernels over internal nodes or nodes, whose count only the device knows,
    // stride over them: a grid for the capacity would be mostly empty CTAs.
    const int grid = dev->sm_count * TN_GRID;
    const int ptiles = (n + TC_TILE - 1) / TC_TILE;
    unsigned *tiles = scan_tiles.as<unsigned>();
    k_tree_count<<<ptiles, OT_THREADS, 0, s>>>(keys.as<uint64_t>(), n, leaf_max, cap_nodes, tiles,
                                               ctr.as<int>());
    k_tree_emit<<<ptiles, OT_THREADS, 0, s>>>(keys.as<uint64_t>(), n, leaf_max, tiles,
                                              ctr.as<int>(), pre_of.as<int>(), in_sd.as<int2>());
    k_tree_children<<<grid, OT_THREADS, 0, s>>>(keys.as<uint64_t>(), n, cap_nodes,
                                                in_sd.as<int2>(), in_end.as<int>(),
                                                in_nch.as<int>(), tiles, ctr.as<int>());
    k_tree_nodes<<<grid, OT_THREADS, 0, s>>>(n, leaf_max, tiles, ctr.as<int>(), in_sd.as<int2>(),
                                             in_end.as<int>(), in_nch.as<int>(), pre_of.as<int>(),
                                             in_rec.as<int4>(), in_arrive.as<int>(),
                                             t_np.as<int>(), t_fp.as<int>(), t_depth.as<int>(),
                                             t_int.as<int>());
    GS_CUDA(cudaGetLastError());
    if (links)
        k_tree_links<<<grid, OT_THREADS, 0, s>>>(ctr.as<int>(), in_rec.as<int4>(), t_np.as<int>(),
                                                 t_fp.as<int>(), t_int.as<int>(),
                                                 t_parent.as<int>(), leaf_of.as<int>());
    MultipoleArgs A;
    A.mx = mx.as<double>();
    A.in_rec = in_rec.as<int4>();
    A.nc = w_nc.as<int4>();
    A.t_depth = t_depth.as<int>();
    A.frame = frame.as<double>();
    A.in_arrive = in_arrive.as<int>();
    A.t_sum = t_sum.as<double>();
    A.t_mass = t_mass.as<double>();
    A.t_com = t_com.as<double>();
    A.na = w_na.as<float4>();
    A.nb = w_nb.as<float4>();
    A.nq = quad ? w_nq.as<float4>() : nullptr;
    // particle records first: the leaves' quadrupoles are formed from them
    GS_CUDA(cudaMemsetAsync(mlist.p, 0, sizeof(int), s));
    k_walk_particles<<<pb, OT_THREADS, 0, s>>>(n, frame.as<double>(), d_x, d_m, sidx.as<int>(),
                                               w_pa.as<float4>(), w_pb.as<float4>(),
                                               mx.as<double>(), misplaced.as<unsigned char>(),
                                               mlist.as<int>());
    k_leaf_multipoles<<<grid, OT_THREADS, 0, s>>>(
        ctr.as<int>(), compat ? 1 : 0, A, w_pa.as<float4>(), w_pb.as<float4>(),
        keys.as<uint64_t>(), sidx.as<int>(), t_np.as<int>(), t_fp.as<int>(), t_int.as<int>(),
        t_nc.as<int>(), t_fc.as<int>(), w_nc.as<int4>(), w_nkey.as<uint64_t>());
    // four lanes per internal node: a larger grid, so that every node of a
    // tree of up to about 2^16 internal nodes starts at once
    (A.nq ? k_multipole_up<true> : k_multipole_up<false>)<<<dev->sm_count * 8, OT_THREADS, 0, s>>>(
        ctr.as<int>(), A);
    GS_CUDA(cudaGetLastError());
    return ok();
}

ErrorStatus OctreeDevice::read_counts(cudaStream_t s, int *nodes, unsigned *status)
{
    int h[3];
    GS_CUDA(cudaMemcpyAsync(h, ctr.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    GS_CUDA(cudaStreamSynchronize(s));
    if (nodes) *nodes = h[CTR_NODES];
    if (status) *status = (unsigned)h[CTR_STATUS];
    return ok();
}

ErrorStatus OctreeDevice::clear_status(cudaStream_t s)
{
    GS_CUDA(cudaMemsetAsync(ctr.as<int>() + CTR_STATUS, 0, sizeof(int), s));
    GS_CUDA(cudaStreamSynchronize(s));
    return ok();
}

// Self-check of div_by_width against the division it replaces: per sample,
// a width w (a random significand, every tenth one all ones, an exponent in
// [-100, 100]) and a dividend x (a random 64-bit pattern for even k: every
// class of double; for odd k one whose quotient lies next to a midpoint of
// two doubles), the frame built as k_bbox_final builds it.
__device__ __forceinline__ unsigned long long wmix(unsigned long long z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__global__ void k_width_div_selftest(long long n, unsigned long long seed, unsigned long long *bad)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    unsigned long long local = 0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += stride) {
        const unsigned long long h = wmix(seed ^ wmix((unsigned long long)k));
        unsigned long long sig = wmix(h + 7) >> 12;
        if (h % 10 == 0) sig = (1ull << 52) - 1ull;
        const int ew = (int)(wmix(h + 3) % 201) - 100;
        const double w = scalbn(__longlong_as_double((long long)(0x3ff0000000000000ull | sig)), ew);
        double frame[8];
        frame[3] = w;
        frame[5] = __ddiv_rn(1.0, w);
        frame[6] = __ddiv_rn(__fma_rn(-frame[5], w, 1.0), w);
        frame[7] = 1.0;
        double x;
        if (k & 1) {
            const unsigned long long m = (wmix(h + 11) >> 11) | (1ull << 52);
            const int e = (int)(wmix(h + 13) % 241) - 120;
            const double q0 = scalbn((double)m, e - 52);
            x = __fma_rn(q0, w, __dmul_rn(scalbn(1.0, e - 53), w));
        } else {
            x = __longlong_as_double((long long)wmix(h + 17));
        }
        const double a = div_by_width(x, frame), b = __ddiv_rn(x, w);
        const bool ok = (isnan(a) && isnan(b)) || __double_as_longlong(a) == __double_as_longlong(b);
        local += ok ? 0 : 1;
    }
    if (local) atomicAdd(bad, local);
}

}  // namespace gs

extern "C" int gsgpu_width_division_selftest(long long n, unsigned long long seed,
                                             long long *mismatches)
{
    if (!mismatches || n < 0) return GRAV_POINTER_ERROR;
    gs::DBuf bad;
    ErrorStatus st = bad.reserve(sizeof(unsigned long long));
    if (st.return_code != GRAV_SUCCESS) {
        free_traceback(&st);
        return GRAV_MEMORY_ERROR;
    }
    cudaError_t e = cudaMemset(bad.p, 0, sizeof(unsigned long long));
    if (e == cudaSuccess) {
        gs::k_width_div_selftest<<<1216, 256>>>(n, seed, bad.as<unsigned long long>());
        e = cudaGetLastError();
    }
    unsigned long long h = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&h, bad.p, sizeof(h), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        std::fprintf(stderr, "gsgpu_width_division_selftest: %s\n", cudaGetErrorString(e));
        return GRAV_FAILURE;
    }
    *mismatches = (long long)h;
    return GRAV_SUCCESS;
}
