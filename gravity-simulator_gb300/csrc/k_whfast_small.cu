// k_whfast_small.cu -- WHFast steps of small planetary systems, many per launch.
//
// The step of k_whfast.cu (src/integrator_whfast.c:290-343) takes eight
// launches, and a system of a few bodies leaves each of them waiting on one
// thread's chain of FP64 operations: 119 us a step for the Sun and eight planets.
// On this GPU an FP64 instruction holds its SM sub-partition's pipe for 64 cycles
// whatever its lanes do (measured with 1 to 32 active lanes and 1 to 8 independent
// operations per lane), so for a small system the time is the number of FP64
// warp instructions, not operations.  Here one CTA of four warps, one per
// sub-partition, keeps a system in shared memory for a whole batch of steps and
// spreads every operation that does not depend on another over lanes:
//   * Kepler solve: eight lanes per body.  The twelve quotients of the two Stumpff
//     series are two instructions' worth of lanes, the series' chains run side by
//     side, the six products of the Newton step are one instruction (39 FP64
//     instructions an iteration where one thread took about 110);
//   * Jacobi -> Cartesian: a lane per component; divisions by the eta_i use
//     reciprocals formed when the order of the bodies changes;
//   * interaction: a lane per pair distance, per quotient and per ordered sum.
// Every value is formed by the operations, and every sum in the order, of
// k_whfast.cu, so the results are the same bit for bit.  19 us a step for the Sun
// and eight planets.
#include "gs_fp64.cuh"
#include "gs_internal.h"
#include "gs_whfast.cuh"

namespace gs {

constexpr int WS_THREADS = 128;
constexpr int WS_PAIRS = kSmallMassive * (kSmallMassive - 1) / 2;
constexpr unsigned WS_ALL = 0xffffffffu;

struct SmallSystem {
    double jx[3][kSmallMax], jv[3][kSmallMax], x[3][kSmallMax], v[3][kSmallMax];
    double m[kSmallMax], eta[kSmallMax], zh[kSmallMax], zl[kSmallMax], gm[kSmallMax];
    double chain[kSmallMax][6];               // m j, then the offsets x - j of the chain
    double J[kSmallMax][3], T[kSmallMax][3];  // j / |j|^3, (x - x0) / |x - x0|^3
    double jc[kSmallMax], tc[kSmallMax];
    double pd[WS_PAIRS][4];                   // massive pairs: x_q - x_p, |.|^3
    double S[WS_PAIRS][3];                    // G m_p m_q d / |d|^3
    double Q[2][WS_PAIRS][3];                 // G m_p d / |d|^3 (felt by q), G m_q d / |d|^3 (by p)
    double V[(kSmallMax - 1) * (kSmallMassive - 1)][3];   // massless - massive terms
    double slots[2 * (kSmallMassive + 1)][3];
    unsigned long long key[kSmallMax];
    int ids[kSmallMax], rank[kSmallMax], before[kSmallMax], hv[kSmallMassive + 1], light[kSmallMax];
    int eta_ok[kSmallMax], rm[kSmallMax];
    int n, nh, nl;
};

__device__ __forceinline__ double bcast8(double v, int src)
{
    return __shfl_sync(WS_ALL, v, src, 8);
}

__device__ __forceinline__ double div_eta(const SmallSystem &w, double x, int i)
{
    if (w.eta_ok[i] && is_zero(x)) return x;   // +-0 over a positive divisor
    return div_known(x, w.eta[i], w.zh[i], w.zl[i], w.eta_ok[i] != 0);
}

// What depends on the order and the masses alone: eta and its reciprocals
// (src/integrator_whfast.c:1266-1279), the Kepler solves' G m_0 eta_i / eta_{i-1}
// (also the massive bodies' primary factor), the massive and massless lists.
__device__ void small_order(SmallSystem &w, double G, bool pairwise, bool form_eta)
{
    const int t = threadIdx.x;
    if (t == 0) {
        if (form_eta) {
            double e = w.m[0];
            w.eta[0] = e;
            for (int i = 1; i < w.n; ++i) {
                e = __dadd_rn(e, w.m[i]);
                w.eta[i] = e;
            }
        }
        int nh = 0, nl = 0;
        for (int i = 0; i < w.n; ++i) {
            const bool h = pairwise || !is_zero(w.m[i]);
            w.before[i] = nh;
            w.rank[i] = h ? nh : -1;
            if (h) {
                if (nh < kSmallMassive) w.hv[nh] = i;
                ++nh;
            } else {
                w.light[nl++] = i;
            }
        }
        w.nh = nh;
        w.nl = nl;
    }
    __syncthreads();
    if (t < w.n) {
        const double e = w.eta[t];
        reciprocal2(e, w.zh[t], w.zl[t]);
        w.eta_ok[t] = e > 0.0 && exponent_within(e, 100);
        if (t > 0) w.gm[t] = __ddiv_rn(__dmul_rn(__dmul_rn(G, w.m[0]), e), w.eta[t - 1]);
    }
    __syncthreads();
}

// Order by distance from the primary (k_wh_sort); returns false when no
// particle has id 0.
__device__ bool small_sort(SmallSystem &w, double G, bool pairwise)
{
    const int t = threadIdx.x, n = w.n;
    int prim = -1;
    for (int i = 0; i < n && prim < 0; ++i)
        if (w.ids[i] == 0) prim = i;
    if (prim < 0) return false;
    // squared distances: four lanes per particle, one component each
    for (int e = t; e < ((4 * n + 31) & ~31); e += WS_THREADS) {
        const int i = min(e >> 2, n - 1), c = min(e & 3, 2);
        const double d = __dsub_rn(w.jx[c][i], w.jx[c][prim]);
        const double p = __dmul_rn(d, d);
        double s = __dadd_rn(p, __shfl_down_sync(WS_ALL, p, 1, 4));
        s = __dadd_rn(s, __shfl_down_sync(WS_ALL, p, 2, 4));
        if ((e & 3) == 0 && (e >> 2) < n) w.key[i] = i == prim ? 0ull : dist_key(s);
    }
    __syncthreads();
    if (!__syncthreads_or(t + 1 < n && w.key[t] > w.key[t + 1])) return true;
    // the keys become the distances; rounded square roots can tie
    if (t < n && t != prim)
        w.key[t] = dist_key(__dsqrt_rn(__longlong_as_double((long long)w.key[t])));
    __syncthreads();
    if (!__syncthreads_or(t + 1 < n && w.key[t] > w.key[t + 1])) return true;
    int to = 0, id = 0;
    double mm = 0.0, q[6];
    if (t < n) {
        const unsigned long long k = w.key[t];
        for (int i = 0; i < n; ++i) to += (w.key[i] < k || (w.key[i] == k && i < t)) ? 1 : 0;
        id = w.ids[t];
        mm = w.m[t];
        for (int c = 0; c < 3; ++c) {
            q[c] = w.jx[c][t];
            q[3 + c] = w.jv[c][t];
        }
    }
    __syncthreads();
    if (t < n) {
        w.ids[to] = id;
        w.m[to] = mm;
        for (int c = 0; c < 3; ++c) {
            w.jx[c][to] = q[c];
            w.jv[c][to] = q[3 + c];
        }
    }
    __syncthreads();
    small_order(w, G, pairwise, true);
    return true;
}

// Universal-variable Kepler drift of all bodies but the primary (kepler_drift in
// k_whfast.cu, src/integrator_whfast.c:424-600), eight lanes per body.
__device__ void small_drift(SmallSystem &w, double dt, const StumpffDiv dA, const StumpffDiv dB,
                            const StumpffDiv dC)
{
    const int l = threadIdx.x & 7;
    const int groups = WS_THREADS / 8;
    for (int i0 = 1; i0 < w.n; i0 += groups) {   // CTA-uniform
        const int i = i0 + (int)(threadIdx.x >> 3);
        const bool act = i < w.n;
        if (!__any_sync(WS_ALL, act)) continue;
        // idle groups of a warp compute on ones
        const double gm = act ? w.gm[i] : 1.0;
        const double comp = !act ? 1.0 : l < 3 ? w.jx[l][i] : w.jv[l < 6 ? l - 3 : 0][i];
        // |x|^2 in lane 0, |v|^2 in lane 3, x.v in lane 0
        const double p1 = __dmul_rn(comp, comp);
        const double p2 = __dmul_rn(comp, __shfl_down_sync(WS_ALL, comp, 3, 8));
        double s1 = __dadd_rn(p1, __shfl_down_sync(WS_ALL, p1, 1, 8));
        s1 = __dadd_rn(s1, __shfl_down_sync(WS_ALL, p1, 2, 8));
        double s2 = __dadd_rn(p2, __shfl_down_sync(WS_ALL, p2, 1, 8));
        s2 = __dadd_rn(s2, __shfl_down_sync(WS_ALL, p2, 2, 8));
        const double root = __dsqrt_rn(s1);
        const double xn = bcast8(root, 0), vn = bcast8(root, 3), xv = bcast8(s2, 0);
        const double quo = __ddiv_rn(l == 0 ? xv : l == 1 ? __dmul_rn(2.0, gm) : dt, xn);
        const double rv = bcast8(quo, 0);
        const double alpha = __dsub_rn(bcast8(quo, 1), __dmul_rn(vn, vn));
        double s = bcast8(quo, 2);
        const double xrv = __dmul_rn(xn, rv);
        // lanes 0..2: the terms of F; 3..5: those of dF
        const int part = l < 3 ? l : l < 6 ? l - 3 : 2;
        const double coef = part == 0 ? xn : part == 1 ? xrv : gm;
        const double c_init = act ? 0.0 : 1.0;
        double c0 = c_init, c1 = c_init, c2 = c_init, c3 = c_init, term = 0.0, sum = 0.0;
        bool conv = !act, bad_z = false, done = !act;
        // the terms at s with the c's held, and their sums in lanes 0 and 3
        auto terms = [&](double ss, double sss) {
            const double pw = l == 0 ? s : l == 1 ? ss : l == 2 ? sss : l == 3 ? 1.0 : l == 4 ? s : ss;
            const double cc = l == 0 ? c1 : l == 1 ? c2 : l == 2 ? c3 : l == 3 ? c0 : l == 4 ? c1 : c2;
            term = __dmul_rn(__dmul_rn(coef, pw), cc);
            sum = __dadd_rn(term, __shfl_down_sync(WS_ALL, term, 1, 8));
            sum = __dadd_rn(sum, __shfl_down_sync(WS_ALL, term, 2, 8));
        };
        for (int it = 0; it < 500; ++it) {
            if (__all_sync(WS_ALL, done)) break;
            const double ss = __dmul_rn(s, s);
            double z = __dmul_rn(alpha, ss);
            if (!done && !finite_bits(z)) bad_z = done = true;
            if (done) z = 0.0625;   // any value in the fast range
            // src/integrator_whfast.c:774-815
            int quarter = 0;
            while (abs_bits(z) > __double_as_longlong(0.1)) {   // |z| > 0.1
                z = __dmul_rn(z, 0.25);
                ++quarter;
            }
            const double qa = div_known(z, dA.d, dA.zh, dA.zl, true);
            const double qb = div_known(z, dB.d, dB.zh, dB.zl, true);
            double t = 1.0;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const double a = bcast8(qa, k), b = bcast8(qb, k);
                const double f = l == 1 ? b : a;
                t = __dsub_rn(1.0, k == 0 ? f : __dmul_rn(f, t));
            }
            // lane 0: t / 6, lane 1: t / 2
            const double head = div_known(t, dC.d, dC.zh, dC.zl, true);
            double u3 = bcast8(head, 0), u2 = bcast8(head, 1);
            const double one = __dsub_rn(1.0, __dmul_rn(z, l == 1 ? u2 : u3));
            double u1 = bcast8(one, 0), u0 = bcast8(one, 1);
            for (; quarter > 0; --quarter) {
                u3 = __dmul_rn(__dadd_rn(u2, __dmul_rn(u0, u3)), 0.25);
                u2 = __dmul_rn(__dmul_rn(u1, u1), 0.5);
                u1 = __dmul_rn(u0, u1);
                u0 = __dsub_rn(__dmul_rn(__dmul_rn(2.0, u0), u0), 1.0);
            }
            if (!done) {
                c0 = u0;
                c1 = u1;
                c2 = u2;
                c3 = u3;
            }
            terms(ss, __dmul_rn(ss, s));
            const double F = __dsub_rn(sum, dt);   // lane 0's
            const double ds = __ddiv_rn(-bcast8(F, 0), bcast8(sum, 3));
            const double next = __dadd_rn(s, ds);
            if (!done) {
                s = next;
                if (abs_bits(ds) < __double_as_longlong(1e-12)) conv = done = true;
            }
        }
        const double ss = __dmul_rn(s, s);
        const double sss = __dmul_rn(ss, s);
        terms(ss, sss);
        const double r = bcast8(sum, 3);
        bool remove = false;
        if (__any_sync(WS_ALL, act && !conv)) {
            const double err = __ddiv_rn(__dsub_rn(bcast8(sum, 0), dt), r);
            remove = !conv && ((err > 1e-5) || bad_z);
        }
        const double t2 = bcast8(term, 2), t5 = bcast8(term, 5);
        const double num = __dmul_rn(__dmul_rn(-gm, s), c1);
        const double rx = __dmul_rn(r, xn);
        const double fr = __ddiv_rn(l == 1 ? num : t5, l == 0 ? xn : l == 1 ? rx : r);
        const double om = __dsub_rn(1.0, fr);
        const double f = bcast8(om, 0), df = bcast8(fr, 1), dg = bcast8(om, 2);
        const double g = __dsub_rn(dt, t2);
        const int k = l < 3 ? l : l < 6 ? l - 3 : 0;
        const double xk = bcast8(comp, k), vk = bcast8(comp, 3 + k);
        const double out = __dadd_rn(__dmul_rn(l < 3 ? f : df, xk), __dmul_rn(l < 3 ? g : dg, vk));
        __syncwarp();
        if (act) {
            if (l < 3)
                w.jx[l][i] = out;
            else if (l < 6)
                w.jv[l - 3][i] = out;
            if (l == 0) w.rm[i] = remove ? 1 : 0;
        }
    }
}

// Stable compaction of the bodies not marked (src/system.c:444-528, :530-577).
__device__ void small_remove(SmallSystem &w, double G, bool pairwise)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        int k = 1;
        for (int i = 1; i < w.n; ++i) {
            if (w.rm[i]) continue;
            w.ids[k] = w.ids[i];
            w.m[k] = w.m[i];
            for (int c = 0; c < 3; ++c) {
                w.jx[c][k] = w.jx[c][i];
                w.jv[c][k] = w.jv[c][i];
            }
            ++k;
        }
        w.n = k;
    }
    __syncthreads();
    small_order(w, G, pairwise, true);
}

// Jacobi -> Cartesian (src/integrator_whfast.c:726-772) by warp 0, a lane per
// component, while the other warps form |j|^3 of every body.  A massless body
// leaves the centre at a fixed point after a step or two, from where on the
// bodies of its run share one offset (k_wh_seq_chain).
__device__ void small_cartesian(SmallSystem &w, double e3)
{
    const int t = threadIdx.x, n = w.n;
    if (t < 32) {
        for (int e = t; e < 6 * n; e += 32) {
            const int i = e / 6, c = e % 6;
            w.chain[i][c] = __dmul_rn(w.m[i], c < 3 ? w.jx[c][i] : w.jv[c - 3][i]);
        }
        __syncwarp();
        const bool on = t < 6;
        const int c = on ? t : 0;
        double xc = __dmul_rn(w.eta[n - 1], c < 3 ? w.jx[c][0] : w.jv[c - 3][0]);
        double y = 0.0;
        bool fixed = false;
        for (int i = n - 1; i >= 1; --i) {
            const double mj = w.chain[i][c];
            const bool light = is_zero(w.m[i]) && __all_sync(WS_ALL, is_zero(mj));
            if (!(light && fixed)) {
                const double old = xc;
                y = div_eta(w, __dsub_rn(xc, mj), i);
                xc = __dmul_rn(w.eta[i - 1], y);
                fixed = light && __all_sync(WS_ALL, __double_as_longlong(xc) ==
                                                            __double_as_longlong(old) &&
                                                        finite_bits(xc) && !neg_zero(xc));
            }
            __syncwarp();
            if (on) w.chain[i][c] = y;
        }
        const double x0 = __ddiv_rn(xc, w.m[0]);
        if (on) (c < 3 ? w.x[c] : w.v[c - 3])[0] = x0;
    } else {
        for (int i = 1 + t - 32; i < n; i += WS_THREADS - 32) {
            const double j[3] = {w.jx[0][i], w.jx[1][i], w.jx[2][i]};
            const double jn = norm3d(j);
            w.jc[i] = __dadd_rn(__dmul_rn(__dmul_rn(jn, jn), jn), e3);
        }
    }
    __syncthreads();
    for (int e = t; e < 6 * (n - 1); e += WS_THREADS) {
        const int i = 1 + e / 6, c = e % 6;
        const double j = c < 3 ? w.jx[c][i] : w.jv[c - 3][i];
        (c < 3 ? w.x[c] : w.v[c - 3])[i] = __dadd_rn(j, w.chain[i][c]);
    }
    __syncthreads();
}

// Interaction accelerations and the kick (k_wh_pairs, k_wh_accel, k_wh_kick;
// src/integrator_whfast.c:839-1264); a_out receives the accelerations.
__device__ void small_accel_kick(SmallSystem &w, double G, double e3, double h,
                                 double *__restrict__ a_out)
{
    const int t = threadIdx.x, n = w.n, nh = w.nh, nl = w.nl;
    const int npairs = nh * (nh - 1) / 2;
    // distances: the primary's, then the massive pairs'; pair (p, q), p < q in
    // list order, is at q (q - 1) / 2 + p
    for (int e = t; e < n - 1 + npairs; e += WS_THREADS) {
        int i = 1 + e, j = 0;
        const int pr = e - (n - 1);
        if (pr >= 0) {
            int q = 1;
            while ((q + 1) * q / 2 <= pr) ++q;
            i = w.hv[q];
            j = w.hv[pr - q * (q - 1) / 2];
        }
        const double d[3] = {__dsub_rn(w.x[0][i], w.x[0][j]), __dsub_rn(w.x[1][i], w.x[1][j]),
                             __dsub_rn(w.x[2][i], w.x[2][j])};
        const double dn = norm3d(d);
        const double dc = __dadd_rn(__dmul_rn(__dmul_rn(dn, dn), dn), e3);
        if (pr >= 0) {
            for (int c = 0; c < 3; ++c) w.pd[pr][c] = d[c];
            w.pd[pr][3] = dc;
        } else {
            w.tc[i] = dc;
            for (int c = 0; c < 3; ++c) w.T[i][c] = d[c];
        }
    }
    // massless - massive terms G m_j (x_i - x_j) / |.|^3
    const int nv = nl * (nh > 1 ? nh - 1 : 0);
    for (int e = t; e < nv; e += WS_THREADS) {
        const int i = w.light[e / (nh - 1)], j = w.hv[1 + e % (nh - 1)];
        const double d[3] = {__dsub_rn(w.x[0][i], w.x[0][j]), __dsub_rn(w.x[1][i], w.x[1][j]),
                             __dsub_rn(w.x[2][i], w.x[2][j])};
        const double dn = norm3d(d);
        const double dc = __dadd_rn(__dmul_rn(__dmul_rn(dn, dn), dn), e3);
        const double Gm = __dmul_rn(G, w.m[j]);
        for (int c = 0; c < 3; ++c) w.V[e][c] = __ddiv_rn(__dmul_rn(Gm, d[c]), dc);
    }
    __syncthreads();
    // quotients: 6 per body (j / jc, d / tc), 9 per massive pair
    const int nb = 6 * (n - 1);
    for (int e = t; e < nb + 9 * npairs; e += WS_THREADS) {
        double num, den;
        double *out;
        if (e < nb) {
            const int i = 1 + e / 6, c = e % 6;
            out = c < 3 ? &w.J[i][c] : &w.T[i][c - 3];
            num = c < 3 ? w.jx[c][i] : *out;
            den = c < 3 ? w.jc[i] : w.tc[i];
        } else {
            const int pr = (e - nb) / 9, c = (e - nb) % 9;
            int q = 1;
            while ((q + 1) * q / 2 <= pr) ++q;
            const int j = w.hv[pr - q * (q - 1) / 2], kk = w.hv[q];
            const double Gp = __dmul_rn(G, w.m[c < 6 ? j : kk]);
            const double f = c < 3 ? __dmul_rn(Gp, w.m[kk]) : Gp;
            out = c < 3 ? &w.S[pr][c] : c < 6 ? &w.Q[0][pr][c - 3] : &w.Q[1][pr][c - 6];
            num = __dmul_rn(f, w.pd[pr][c % 3]);
            den = w.pd[pr][3];
        }
        *out = __ddiv_rn(num, den);
    }
    __syncthreads();
    // ordered sums: bodies' interior and exterior terms on warps 0 and 1, the
    // shared pair sums on warps 2 and 3 (slots as in k_wh_pairs)
    const int bodies = 3 * (n - 1);
    constexpr int HALF = WS_THREADS / 2;
    constexpr int PER = (3 * (kSmallMax - 1) + HALF - 1) / HALF;
    double acc[PER], ext[PER];
    if (t < HALF) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = u * HALF + t;
            if (e >= bodies) break;
            const int i = 1 + e / 3, c = e % 3;
            const int r = w.rank[i], g = w.before[i];
            double in = 0.0, ex = 0.0;
            if (r >= 0) {
                for (int p = 1; p < r; ++p) in = __dadd_rn(in, w.Q[0][r * (r - 1) / 2 + p][c]);
                for (int q = max(r + 1, 1); q < nh; ++q)
                    ex = __dadd_rn(ex, w.Q[1][q * (q - 1) / 2 + r][c]);
            } else {
                const double(*V)[3] = w.V + (i - g) * (nh - 1);   // i - g massless bodies before i
                for (int p = 1; p < g; ++p) in = __dadd_rn(in, V[p - 1][c]);
                for (int q = max(g, 1); q < nh; ++q) ex = __dadd_rn(ex, -V[q - 1][c]);
            }
            const double Gm0 = __dmul_rn(G, w.m[0]);
            double a = __dmul_rn(r >= 0 ? w.gm[i] : Gm0, __dsub_rn(w.J[i][c], w.T[i][c]));
            const double scaled = div_eta(w, __dmul_rn(in, w.eta[i]), i - 1);
            a = __dsub_rn(a, r >= 0 ? scaled : in);
            acc[u] = a;
            ext[u] = ex;
        }
    } else {
        for (int e = t - HALF; e < 6 * (nh + 1); e += HALF) {
            const int slot = e / 3, c = e % 3;
            int p_end, q_begin;
            if (slot <= nh) {
                p_end = q_begin = slot;
            } else {
                p_end = slot - (nh + 1);
                q_begin = p_end + 1;
            }
            double aux = 0.0;
            for (int p = 0; p < p_end; ++p)
                for (int q = q_begin; q < nh; ++q) aux = __dadd_rn(aux, w.S[q * (q - 1) / 2 + p][c]);
            w.slots[slot][c] = aux;
        }
    }
    __syncthreads();
    if (t < HALF) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = u * HALF + t;
            if (e >= bodies) break;
            const int i = 1 + e / 3, c = e % 3;
            const int r = w.rank[i];
            const double pr = w.slots[r >= 0 ? nh + 1 + r : w.before[i]][c];
            const double a = __dsub_rn(__dadd_rn(acc[u], ext[u]), div_eta(w, pr, i - 1));
            if (a_out) a_out[3 * i + c] = a;
            w.jv[c][i] = __dadd_rn(w.jv[c][i], __dmul_rn(a, h));
        }
    } else if (t < HALF + 3) {
        // the primary's acceleration is zero; its kick is an add of +0 h
        const int c = t - HALF;
        if (a_out) a_out[c] = 0.0;
        w.jv[c][0] = __dadd_rn(w.jv[c][0], __dmul_rn(0.0, h));
    }
    __syncthreads();
}

__global__ void __launch_bounds__(WS_THREADS) k_wh_small(EnsDev E, int steps, double h)
{
    __shared__ SmallSystem w;
    const int s = blockIdx.x, t = threadIdx.x;
    const int base = E.off[s];
    const int n0 = E.cnt[s];
    if (n0 <= 0) return;
    if (n0 > kSmallMax) {   // the host does not launch such systems
        if (t == 0) atomicOr(E.status, ST_CAPACITY);
        return;
    }
    const bool pairwise = E.variant == WH_PAIRWISE;
    const double e3 = __dmul_rn(__dmul_rn(E.eps, E.eps), E.eps);
    // this lane's divisors: the quotients z / d of the two series, and the
    // series' heads t / 6 and t / 2
    constexpr int kA[6] = {SD210, SD156, SD110, SD72, SD42, SD20};
    constexpr int kB[6] = {SD182, SD132, SD90, SD56, SD30, SD12};
    const int l = t & 7;
    StumpffDiv dA = kStumpffDiv[SD20], dB = kStumpffDiv[SD12], dC = kStumpffDiv[SD6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
        if (l == k) {
            dA = kStumpffDiv[kA[k]];
            dB = kStumpffDiv[kB[k]];
        }
    if (l == 1) dC = StumpffDiv{2.0, 0.5, 0.0};
    for (int i = t; i < n0; i += WS_THREADS) {
        w.ids[i] = E.ids[base + i];
        w.m[i] = E.m[base + i];
        w.eta[i] = E.eta[base + i];
        w.rm[i] = 0;
        for (int c = 0; c < 3; ++c) {
            w.jx[c][i] = E.jx[3 * (size_t)(base + i) + c];
            w.jv[c][i] = E.jv[3 * (size_t)(base + i) + c];
        }
    }
    if (t == 0) w.n = n0;
    __syncthreads();
    small_order(w, E.G, pairwise, false);
    if (w.nh > kSmallMassive) {   // CTA-uniform; the host does not launch such systems
        if (t == 0) atomicOr(E.status, ST_CAPACITY);
        return;
    }
    for (int k = 0; k < steps; ++k) {
        if (!small_sort(w, E.G, pairwise)) {   // CTA-uniform
            if (t == 0) atomicOr(E.status, ST_NO_PRIMARY);
            return;
        }
        small_drift(w, h, dA, dB, dC);
        __syncthreads();
        if (__syncthreads_or(t > 0 && t < w.n && w.rm[t] && E.remove_invalid))
            small_remove(w, E.G, pairwise);
        small_cartesian(w, e3);
        small_accel_kick(w, E.G, e3, h, k == steps - 1 ? E.a + 3 * (size_t)base : nullptr);
    }
    const int n = w.n;
    if (t == 0) E.cnt[s] = n;
    for (int i = t; i < n; i += WS_THREADS) {
        const size_t p = (size_t)base + i;
        E.ids[p] = w.ids[i];
        E.m[p] = w.m[i];
        E.eta[p] = w.eta[i];
        for (int c = 0; c < 3; ++c) {
            E.jx[3 * p + c] = w.jx[c][i];
            E.jv[3 * p + c] = w.jv[c][i];
            E.x[3 * p + c] = w.x[c][i];
            E.v[3 * p + c] = w.v[c][i];
        }
    }
}

void launch_wh_small(const EnsDev &E, int steps, double h, cudaStream_t s)
{
    k_wh_small<<<E.S, WS_THREADS, 0, s>>>(E, steps, h);
}

}  // namespace gs
