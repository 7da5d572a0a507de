// k_walk.cu -- Barnes-Hut tree walk and the Barnes-Hut engine.
//
// Replaces helper_compute_acceleration (src/acceleration_barnes_hut.c:78-248)
// and acceleration_barnes_hut (:33-76).
//
// Warp-cooperative walk.  A warp owns 32 consecutive particles in Morton
// order and walks the union of their traversals.  A shared stack holds nodes
// with the mask of the lanes whose walk reaches them; each step pops up to 32
// nodes, every lane loads the records of one into shared memory, and then all
// lanes go through the batch, each making the reference's own decision for its
// particle --
//   cell-membership test (compat: the reference's Morton prefixes with its
//   sorted-keys-by-particle-id read, src/acceleration_barnes_hut.c:120/:145;
//   otherwise the sorted index in the cell's range, which is the same test on the
//   particle's own key), then the opening test
//   (w_level)^2 < theta^2 |R|^2 (:157-162) -> monopole (:164-174),
//   else leaf -> particle terms skipping itself (:181-214), else descend --
// and the nodes that some lanes open push their children with those lanes'
// mask (leaves: their particles are staged and summed the same way).  Each
// particle sees exactly the nodes of the reference's depth-first walk, in
// another order.
//
// What bounds it is instruction issue.  Walking one child at a time (a stack
// of node, next child and mask per depth) cost about 220 instructions and a
// chain of dependent loads per interaction; in a batch the loads of 32 nodes are
// one, and a node costs about 45 instructions.  Walk of the galaxy pair at
// N = 150,000, theta 0.5: 2.79 -> 1.13 ms.
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
constexpr int WK_STACK = 512;    // stack entries per warp
// Entries kept free for a depth-first descent: popping one node and pushing its
// (at most 8) children grows the stack by 7 per level.  Batches shrink so that the
// stack never passes WK_STACK - WK_RESERVE before such a descent starts.
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
    const int *gate;                // when set, the launch runs only if *gate != 0
};

// Kahan-compensated sums of x, y (as a pair, through the paired FP32 operations)
// and z; n* hold the negated compensations.
struct Acc3 {
    float2 s, n;
    float sz, nz;
};

__device__ __forceinline__ void add3(Acc3 &a, float2 pxy, float pz)
{
    const float2 minus = make_float2(-1.0f, -1.0f);
    const float2 y = __fadd2_rn(pxy, a.n);
    const float2 t = __fadd2_rn(a.s, y);
    a.n = __ffma2_rn(__ffma2_rn(a.s, minus, t), minus, y);   // y - (t - s)
    a.s = t;
    const float yz = __fadd_rn(pz, a.nz);
    const float tz = __fadd_rn(a.sz, yz);
    a.nz = __fsub_rn(yz, __fsub_rn(tz, a.sz));
    a.sz = tz;
}

// One batch of nodes or of leaf particles in shared memory.
template <bool QUAD, bool COMPAT>
struct WalkShared {
    int2 stack[WK_STACK];    // (node, lanes that reach it)
    float4 a[32], b[32];     // com or position: (hi, mass), (lo, cell side^2)
    int4 c[32];              // (first child, children, first particle, particles)
    unsigned mask[32];
    float4 q[QUAD ? 64 : 1];
    uint64_t key[COMPAT ? 32 : 1];
    int level[COMPAT ? 32 : 1];
};

template <bool QUAD, bool COMPAT>
__global__ void __launch_bounds__(WK_THREADS)
k_bh_walk(WalkArgs A)
{
    __shared__ WalkShared<QUAD, COMPAT> shared_all[WK_WARPS];

    if (A.gate && *A.gate == 0) return;   // block-uniform
    if (*A.status & ST_TREE_OVERFLOW) return;   // the build overflowed: no tree to walk
    WalkShared<QUAD, COMPAT> &w = shared_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;

    const int s = blockIdx.x * WK_THREADS + threadIdx.x;
    const bool valid = s < A.n;
    const int id = valid ? A.sidx[s] : -1;
    uint64_t key_i = 0;
    // negated particle position
    float2 nxyh = make_float2(0.f, 0.f), nxyl = nxyh;
    float nzh = 0.f, nzl = 0.f;
    if (valid) {
        if (COMPAT) key_i = A.skeys[id];
        const float4 ph = A.pa[s], pl = A.pb[s];
        nxyh = make_float2(-ph.x, -ph.y);
        nxyl = make_float2(-pl.x, -pl.y);
        nzh = -ph.z;
        nzl = -pl.z;
    }
    const float th2f = (float)A.theta2;
    Acc3 acc = {};
    int n_cell = 0, n_pp = 0;

    const unsigned valid_mask = __ballot_sync(0xffffffffu, valid);
    if (valid_mask == 0) return;   // warp-uniform
    // the root is opened by every lane without a test: its children start the walk
    const int4 root = A.nc[0];
    if (lane < root.y) w.stack[lane] = make_int2(root.x + lane, (int)valid_mask);
    int top = root.y;
    __syncwarp();
    while (top > 0) {
        int k = min(32, top);
        const int room = (WK_STACK - WK_RESERVE - top) / 7;
        if (room < k) k = max(1, room);
        // load: one node per lane
        int4 ci = make_int4(0, 0, 0, 0);
        if (lane < k) {
            const int2 e = w.stack[top - k + lane];
            ci = A.nc[e.x];
            w.a[lane] = A.na[e.x];
            w.b[lane] = A.nb[e.x];
            // what the loop needs of the node: (node, -, first particle, particles)
            w.c[lane] = make_int4(e.x, ci.y, ci.z, ci.w);
            w.mask[lane] = (unsigned)e.y;
            if (QUAD) {
                w.q[2 * lane] = A.nq[2 * (size_t)e.x];
                w.q[2 * lane + 1] = A.nq[2 * (size_t)e.x + 1];
            }
            if (COMPAT) {
                w.key[lane] = A.nkey[e.x];
                w.level[lane] = A.depth[e.x];
            }
        }
        top -= k;
        __syncwarp();
        unsigned opened = 0;   // lanes that open this lane's node
#pragma unroll 2
        for (int j = 0; j < k; ++j) {
            const float4 ca = w.a[j], cb = w.b[j];
            const bool act = (w.mask[j] >> lane) & 1u;
            const float2 dxy = __fadd2_rn(__fadd2_rn(make_float2(ca.x, ca.y), nxyh),
                                          __fadd2_rn(make_float2(cb.x, cb.y), nxyl));
            const float dz = (ca.z + nzh) + (cb.z + nzl);
            const float ns = fmaf(dxy.x, dxy.x, fmaf(dxy.y, dxy.y, dz * dz));
            const float t = th2f * ns;
            bool accept = act && cb.w < t;
            bool inside;
            if (COMPAT) {
                const int sh = 3 * (OCT_MAX_LEVEL - w.level[j]);
                inside = (key_i >> sh) == (w.key[j] >> sh);
            } else {
                const int4 cj = w.c[j];
                inside = (unsigned)(s - cj.z) < (unsigned)cj.w;
            }
            if (act && !inside && fabsf(cb.w - t) <= 1e-5f * cb.w) {
                // exact FP64 test, reference operation order
                const int c = w.c[j].x;
                const double r0 = __dsub_rn(A.x[3 * (size_t)id + 0], A.ncom[3 * (size_t)c + 0]);
                const double r1 = __dsub_rn(A.x[3 * (size_t)id + 1], A.ncom[3 * (size_t)c + 1]);
                const double r2 = __dsub_rn(A.x[3 * (size_t)id + 2], A.ncom[3 * (size_t)c + 2]);
                const double nsd = __dadd_rn(__dadd_rn(__dmul_rn(r0, r0), __dmul_rn(r1, r1)),
                                             __dmul_rn(r2, r2));
                // box_length / (2 << level)  (src/acceleration_barnes_hut.c:157)
                const double wd = __ddiv_rn(A.frame[4], (double)(2 << A.depth[c]));
                accept = __dmul_rn(wd, wd) < __dmul_rn(A.theta2, nsd);
            }
            accept = accept && !inside;
            const unsigned om = __ballot_sync(0xffffffffu, act && !accept);
            if (lane == j) opened = om;
            if (!__any_sync(0xffffffffu, accept)) continue;
            // lanes that do not accept add zeros
            const float ri = accept ? rsqrt_approx(ns + A.eps2) : 0.0f;
            const float ri2 = ri * ri;
            const float ri3 = ri2 * ri;
            const float sc = ca.w * ri3;
            float2 pxy = __fmul2_rn(dxy, make_float2(sc, sc));
            float pz = dz * sc;
            if (QUAD) {
                // d = com - x = -R:  G [-Q d / r^5 + 2.5 (d.Q.d) d / r^7]
                const float4 q0 = w.q[2 * j], q1 = w.q[2 * j + 1];
                const float qx = q0.x * dxy.x + q0.y * dxy.y + q0.z * dz;
                const float qy = q0.y * dxy.x + q0.w * dxy.y + q1.x * dz;
                const float qz = q0.z * dxy.x + q1.x * dxy.y + q1.y * dz;
                const float dqd = dxy.x * qx + dxy.y * qy + dz * qz;
                const float ri5 = ri3 * ri2;
                const float f = 2.5f * dqd * ri5 * ri2;
                pxy.x += f * dxy.x - qx * ri5;
                pxy.y += f * dxy.y - qy * ri5;
                pz += f * dz - qz * ri5;
            }
            add3(acc, pxy, pz);
            n_cell += accept ? 1 : 0;
        }
        __syncwarp();   // the batch is read
        // children of opened nodes, with the opening lanes
        const int ch = opened ? ci.y : 0;
        int cin = ch;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, cin, o);
            if (lane >= o) cin += t;
        }
        const int pushes = __shfl_sync(0xffffffffu, cin, 31);
        if (top + pushes > WK_STACK) {
            if (lane == 0) atomicOr(A.status, ST_STACK_OVERFLOW);
            break;
        }
        for (int q = 0; q < ch; ++q) w.stack[top + cin - ch + q] = make_int2(ci.x + q, (int)opened);
        top += pushes;
        // particles of opened leaves, 32 at a time
        const int cnt = (opened && ci.y <= 0) ? ci.w : 0;
        unsigned leaves = __ballot_sync(0xffffffffu, cnt > 0);
        int skip = 0;   // particles of the first remaining leaf already taken
        while (leaves) {
            // lanes take the particles of the remaining leaves in turn
            int have = 0;
            int mine = -1;
            unsigned open_m = 0;
            while (leaves && have < 32) {
                const int src = __ffs(leaves) - 1;
                const int first = __shfl_sync(0xffffffffu, ci.z, src) + skip;
                const int left = __shfl_sync(0xffffffffu, cnt, src) - skip;
                const unsigned om = __shfl_sync(0xffffffffu, opened, src);
                const int take = min(left, 32 - have);
                if (lane >= have && lane < have + take) {
                    mine = first + lane - have;
                    open_m = om;
                }
                have += take;
                skip += take;
                if (take == left) {
                    leaves &= leaves - 1;
                    skip = 0;
                }
            }
            __syncwarp();
            if (mine >= 0) {
                w.a[lane] = A.pa[mine];
                w.b[lane] = A.pb[mine];
                w.mask[lane] = open_m;
                w.c[lane].x = mine;
            }
            __syncwarp();
#pragma unroll 2
            for (int j = 0; j < have; ++j) {
                const float4 qa = w.a[j], qb = w.b[j];
                const bool act = ((w.mask[j] >> lane) & 1u) && w.c[j].x != s;
                const float2 dxy = __fadd2_rn(__fadd2_rn(make_float2(qa.x, qa.y), nxyh),
                                              __fadd2_rn(make_float2(qb.x, qb.y), nxyl));
                const float dz = (qa.z + nzh) + (qb.z + nzl);
                const float r2 = fmaf(dxy.x, dxy.x, fmaf(dxy.y, dxy.y, fmaf(dz, dz, A.eps2)));
                const float ri = rsqrt_approx(r2);
                const float sc = act ? qa.w * ri * ri * ri : 0.0f;
                add3(acc, __fmul2_rn(dxy, make_float2(sc, sc)), dz * sc);
                n_pp += act ? 1 : 0;
            }
            __syncwarp();
        }
        __syncwarp();
    }
    if (valid) {
        A.a[3 * (size_t)id + 0] = A.G * ((double)acc.s.x + (double)acc.n.x);
        A.a[3 * (size_t)id + 1] = A.G * ((double)acc.s.y + (double)acc.n.y);
        A.a[3 * (size_t)id + 2] = A.G * ((double)acc.sz + (double)acc.nz);
    }
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

static void launch_walk_kernel(const WalkArgs &w, bool quad, bool compat, cudaStream_t s)
{
    const int grid = (w.n + WK_THREADS - 1) / WK_THREADS;
    if (compat)
        k_bh_walk<false, true><<<grid, WK_THREADS, 0, s>>>(w);
    else if (quad)
        k_bh_walk<true, false><<<grid, WK_THREADS, 0, s>>>(w);
    else
        k_bh_walk<false, false><<<grid, WK_THREADS, 0, s>>>(w);
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
        w.gate = nullptr;
        GS_CUDA(cudaMemsetAsync(counters_.p, 0, 2 * sizeof(unsigned long long), s));
        if (group_) {
            if (timer) GS_TRY(timer->begin(s));
            GS_TRY(launch_bh_group_walk(tree_, theta_, eps_, G_, d_a, w.counters, s));
            if (timer) GS_TRY(timer->end(s));
            return ok();
        }
        if (timer) GS_TRY(timer->begin(s));
        launch_walk_kernel(w, quad_, compat_, s);
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

// Walk of a built (non-compat) tree, for engines that walk one tree several
// times (the learned method's cheap walk and its gated fallback).
ErrorStatus launch_bh_walk(const OctreeDevice &t, const double *d_x, double theta, double eps,
                           double G, double *d_a, const int *gate,
                           unsigned long long *counters, cudaStream_t s)
{
    WalkArgs w;
    w.na = t.w_na.as<float4>();
    w.nb = t.w_nb.as<float4>();
    w.nq = t.quad ? t.w_nq.as<float4>() : nullptr;
    w.nc = t.w_nc.as<int4>();
    w.nkey = t.w_nkey.as<uint64_t>();
    w.ncom = t.t_com.as<double>();
    w.depth = t.t_depth.as<int>();
    w.pa = t.w_pa.as<float4>();
    w.pb = t.w_pb.as<float4>();
    w.sidx = t.sidx.as<int>();
    w.skeys = t.keys.as<uint64_t>();
    w.x = d_x;
    w.frame = t.frame.as<double>();
    w.n = t.n;
    w.eps2 = (float)(eps * eps);
    w.theta2 = theta * theta;
    w.G = G;
    w.a = d_a;
    w.counters = counters;
    w.status = reinterpret_cast<unsigned *>(t.ctr.as<int>() + CTR_STATUS);
    w.gate = gate;
    launch_walk_kernel(w, t.quad, t.compat, s);
    GS_CUDA(cudaGetLastError());
    return ok();
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
