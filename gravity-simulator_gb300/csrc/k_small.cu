// k_small.cu -- integrator steps of small systems by one CTA.
//
// A step of a few bodies through the general kernels is a chain of launches (a
// drift, a force, a kick; IAS15: about a hundred) whose threads each run a long
// chain of FP64 instructions, 64 cycles apiece whatever the lanes do.  For systems
// of up to kTinyMax bodies under the FP64 forces (GRAV_GPU_PAIRWISE_FP64,
// GRAV_GPU_MASSLESS) the kernels here keep the state in shared memory and take a
// batch of fixed steps (k_tiny_fixed), a whole embedded Runge-Kutta attempt
// (k_tiny_rk) or a whole IAS15 step with its predictor-corrector iterations
// (k_tiny_ias15) per launch, with one lane per pair, per element and coefficient or
// per ordered sum.  Every value is formed by the operations of the general kernels
// (k_direct.cu, k_massless.cu, k_integrate.cu, k_ias15.cu) in the same order, so the
// results are the same bit for bit.  Step-size control stays on the host.
#include "gs_fp64.cuh"
#include "gs_internal.h"
#include "gs_ptx.cuh"

namespace gs {

constexpr int TY_THREADS = 128;   // a warp per SM sub-partition
constexpr int TY_L = 3 * kTinyMax;
constexpr int TY_PAIRS = kTinyMax * (kTinyMax - 1) / 2;

constexpr int TY_FEW = TY_THREADS / 3;   // pairs with a thread per component

// Force state: t (x_i - x_j) of every interacting pair, or, of at most TY_FEW
// pairs, its products with the masses (of the first body, negated, and of the
// second; of a light body's pair with the heavy one's), and the lists of the
// massless variant.
struct TinyForce {
    union {
        double tr[TY_PAIRS][3];
        struct {
            double pr[2][TY_FEW][3];
            int i[TY_FEW], j[TY_FEW], mi[TY_FEW];   // bodies of a pair, index of its first mass
        } few;
    };
    double m[kTinyMax];
    int heavy[kTinyMax], light[kTinyMax];
    int nh, nl;
    bool is_few;
};

__device__ void tiny_lists(TinyForce &f, const double *__restrict__ m, int n, bool massless)
{
    for (int i = threadIdx.x; i < n; i += TY_THREADS) f.m[i] = m[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        int nh = 0, nl = 0;
        for (int i = 0; i < n; ++i) {
            if (massless && is_zero(f.m[i]))
                f.light[nl++] = i;
            else
                f.heavy[nh++] = i;
        }
        f.nh = nh;
        f.nl = nl;
        f.is_few = nh * (nh - 1) / 2 + nl * nh <= TY_FEW && 3 * n <= TY_THREADS;
    }
    __syncthreads();
    const int nh = f.nh, np = nh * (nh - 1) / 2;
    const int e = threadIdx.x;
    if (f.is_few && e < np + f.nl * nh) {
        if (e < np) {
            int q = 1;
            while ((q + 1) * q / 2 <= e) ++q;
            f.few.i[e] = f.few.mi[e] = f.heavy[e - q * (q - 1) / 2];
            f.few.j[e] = f.heavy[q];
        } else {
            f.few.i[e] = f.heavy[(e - np) % nh];
            f.few.mi[e] = (e - np) % nh;
            f.few.j[e] = f.light[(e - np) / nh];
        }
    }
    __syncthreads();
}

// t (x_i - x_j) of a pair, t = G / (|x_i - x_j|^2 + eps^2)^(3/2).
__device__ __forceinline__ void tiny_pair(const double *x, int i, int j, double G, double eps2, double r[3],
                                          double &t)
{
#pragma unroll
    for (int c = 0; c < 3; ++c) r[c] = __dsub_rn(x[3 * i + c], x[3 * j + c]);
    const double rn = __dsqrt_rn(__dadd_rn(
        __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2])), eps2));
    t = __ddiv_rn(G, __dmul_rn(__dmul_rn(rn, rn), rn));
}

// Accelerations at x (shared, 3 n) into a (shared): src/acceleration.c:177-234,
// and :236-367 when massless bodies are listed apart (weighted by the mass at the
// loop index, as there).  Entered and left in step.
//
// What bounds it is the chain of FP64 operations (65 cycles each).  With at most
// TY_FEW pairs a thread per pair and component forms the component's two products
// with the masses, so that the ordered sums are additions alone (the Sun and eight
// planets, with products formed inside the sums and so: leapfrog step 5.5 and 4.1 us;
// an IAS15 step takes 225).
__device__ void tiny_force(TinyForce &f, const double *x, double *a, double G, double eps2)
{
    const int nh = f.nh, nl = f.nl;
    const int np = nh * (nh - 1) / 2;
    if (f.is_few) {
        const int e = threadIdx.x / 3, c = threadIdx.x % 3;
        if (e < np + nl * nh) {
            double r[3], t;
            tiny_pair(x, f.few.i[e], f.few.j[e], G, eps2, r, t);
            const double tr = __dmul_rn(t, c == 0 ? r[0] : c == 1 ? r[1] : r[2]);
            const double mi = f.m[f.few.mi[e]];
            f.few.pr[0][e][c] = __dmul_rn(e < np ? -tr : tr, mi);
            if (e < np) f.few.pr[1][e][c] = __dmul_rn(tr, f.m[f.few.j[e]]);
        }
        __syncthreads();
        if (threadIdx.x < 3 * (nh + nl)) {
            const int b = e;
            double acc = 0.0;
            if (b < nh) {
                for (int q = 0; q < b; ++q) acc = __dsub_rn(acc, f.few.pr[0][b * (b - 1) / 2 + q][c]);
                for (int q = b + 1; q < nh; ++q) acc = __dsub_rn(acc, f.few.pr[1][q * (q - 1) / 2 + b][c]);
                a[3 * f.heavy[b] + c] = acc;
            } else {
                const int first = np + (b - nh) * nh;
                for (int p = 0; p < nh; ++p) acc = __dadd_rn(acc, f.few.pr[0][first + p][c]);
                a[3 * f.light[b - nh] + c] = acc;
            }
        }
        __syncthreads();
        return;
    }
    // pair (p, q), p < q in list order, at q (q - 1) / 2 + p, then (light l, heavy p)
    for (int e = threadIdx.x; e < np + nl * nh; e += TY_THREADS) {
        int i, j;
        if (e < np) {
            int q = 1;
            while ((q + 1) * q / 2 <= e) ++q;
            i = f.heavy[e - q * (q - 1) / 2];
            j = f.heavy[q];
        } else {
            i = f.heavy[(e - np) % nh];
            j = f.light[(e - np) / nh];
        }
        double r[3], t;
        tiny_pair(x, i, j, G, eps2, r, t);
#pragma unroll
        for (int c = 0; c < 3; ++c) f.tr[e][c] = __dmul_rn(t, r[c]);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * (nh + nl); e += TY_THREADS) {
        const int c = e % 3, b = e / 3;
        double acc = 0.0;
        if (b < nh) {
            // seen from body b, the pair vector of an earlier body is reversed
            for (int q = 0; q < b; ++q)
                acc = __dsub_rn(acc, __dmul_rn(-f.tr[b * (b - 1) / 2 + q][c], f.m[f.heavy[q]]));
            for (int q = b + 1; q < nh; ++q)
                acc = __dsub_rn(acc, __dmul_rn(f.tr[q * (q - 1) / 2 + b][c], f.m[f.heavy[q]]));
            a[3 * f.heavy[b] + c] = acc;
        } else {
            const double(*tr)[3] = f.tr + np + (b - nh) * nh;
            for (int p = 0; p < nh; ++p) acc = __dadd_rn(acc, __dmul_rn(tr[p][c], f.m[p]));
            a[3 * f.light[b - nh] + c] = acc;
        }
    }
    __syncthreads();
}

// ---- fixed steps ------------------------------------------------------------
struct FixedShared {
    TinyForce f;
    double x[TY_L], v[TY_L], xe[TY_L], ve[TY_L], a[TY_L], x0[TY_L], v0[TY_L];
    double xk[4][TY_L], vk[4][TY_L];
};

__device__ __forceinline__ double tiny_rk4_incr(double k1, double k2, double k3, double k4, double dt)
{
    const double s = __dadd_rn(__dadd_rn(__dadd_rn(k1, __dmul_rn(2.0, k2)), __dmul_rn(2.0, k3)), k4);
    return __ddiv_rn(__dmul_rn(s, dt), 6.0);
}

__global__ void __launch_bounds__(TY_THREADS)
k_tiny_fixed(TinySystem S, int integrator, int steps, double h)
{
    extern __shared__ __align__(16) unsigned char ty_smem[];
    FixedShared &w = *reinterpret_cast<FixedShared *>(ty_smem);
    const int L = 3 * S.n, t = threadIdx.x;
    const double eps2 = __dmul_rn(S.eps, S.eps);
    for (int k = t; k < L; k += TY_THREADS) {
        w.x[k] = S.x[k];
        w.v[k] = S.v[k];
        w.xe[k] = S.xe[k];
        w.ve[k] = S.ve[k];
        w.a[k] = S.a[k];
    }
    tiny_lists(w.f, S.m, S.n, S.massless);
    for (int step = 0; step < steps; ++step) {
        if (integrator == INTEGRATOR_LEAPFROG) {
            for (int k = t; k < L; k += TY_THREADS) comp_update(w.x[k], w.xe[k], w.v[k], h);
            __syncthreads();
            tiny_force(w.f, w.x, w.a, S.G, eps2);
            for (int k = t; k < L; k += TY_THREADS) comp_update(w.v[k], w.ve[k], w.a[k], h);
            // the same thread reads v[k] next
        } else if (integrator == INTEGRATOR_RK4) {
            for (int k = t; k < L; k += TY_THREADS) {
                w.x0[k] = w.x[k];
                w.v0[k] = w.v[k];
            }
            __syncthreads();
            for (int s = 0; s < 4; ++s) {
                if (s > 0) {
                    const double coef = s == 3 ? 1.0 : 0.5;
                    for (int k = t; k < L; k += TY_THREADS) {
                        w.x[k] = __dadd_rn(w.x0[k], __dmul_rn(__dmul_rn(coef, w.xk[s - 1][k]), h));
                        w.v[k] = __dadd_rn(w.v0[k], __dmul_rn(__dmul_rn(coef, w.vk[s - 1][k]), h));
                    }
                    __syncthreads();
                }
                tiny_force(w.f, w.x, w.vk[s], S.G, eps2);
                for (int k = t; k < L; k += TY_THREADS) w.xk[s][k] = w.v[k];
            }
            for (int k = t; k < L; k += TY_THREADS) {
                double ev = __dadd_rn(
                    w.ve[k], tiny_rk4_incr(w.vk[0][k], w.vk[1][k], w.vk[2][k], w.vk[3][k], h));
                double ex = __dadd_rn(
                    w.xe[k], tiny_rk4_incr(w.xk[0][k], w.xk[1][k], w.xk[2][k], w.xk[3][k], h));
                const double vn = __dadd_rn(w.v0[k], ev), xn = __dadd_rn(w.x0[k], ex);
                w.ve[k] = __dadd_rn(ev, __dsub_rn(w.v0[k], vn));
                w.xe[k] = __dadd_rn(ex, __dsub_rn(w.x0[k], xn));
                w.v[k] = vn;
                w.x[k] = xn;
                w.a[k] = w.vk[3][k];
            }
            __syncthreads();
        } else {
            tiny_force(w.f, w.x, w.a, S.G, eps2);
            for (int k = t; k < L; k += TY_THREADS) {
                if (integrator == INTEGRATOR_EULER) {
                    const double v0 = w.v[k];
                    comp_update(w.v[k], w.ve[k], w.a[k], h);
                    comp_update(w.x[k], w.xe[k], v0, h);
                } else {   // Euler-Cromer
                    comp_update(w.v[k], w.ve[k], w.a[k], h);
                    comp_update(w.x[k], w.xe[k], w.v[k], h);
                }
            }
            __syncthreads();
        }
    }
    for (int k = t; k < L; k += TY_THREADS) {
        S.x[k] = w.x[k];
        S.v[k] = w.v[k];
        S.xe[k] = w.xe[k];
        S.ve[k] = w.ve[k];
        S.a[k] = w.a[k];
    }
}

// ---- embedded Runge-Kutta -----------------------------------------------------
struct RkShared {
    TinyForce f;
    double x[TY_L], v[TY_L], xe[TY_L], ve[TY_L], xs[TY_L], end[4][TY_L];
    double xk[13][TY_L], vk[13][TY_L];
};

// One attempt of size h (src/integrator_rk_embedded.c:721-856) from the state,
// after the previous attempt's result became the state if it was accepted.  The
// squared error terms go to terms[2 L] in the order in which the host adds them;
// attempt false: only the acceptance.
__global__ void __launch_bounds__(TY_THREADS)
k_tiny_rk(TinySystem S, TinyRk R, bool accept, bool attempt, double h, double tol,
          double *__restrict__ terms)
{
    extern __shared__ __align__(16) unsigned char ty_smem[];
    RkShared &w = *reinterpret_cast<RkShared *>(ty_smem);
    const int L = 3 * S.n, t = threadIdx.x;
    const double eps2 = __dmul_rn(S.eps, S.eps);
    for (int k = t; k < L; k += TY_THREADS) {
        const double *x = accept ? S.x1 : S.x, *v = accept ? S.v1 : S.v;
        const double *xe = accept ? S.txe : S.xe, *ve = accept ? S.tve : S.ve;
        w.x[k] = x[k];
        w.v[k] = v[k];
        w.xe[k] = xe[k];
        w.ve[k] = ve[k];
        if (accept) {
            S.x[k] = w.x[k];
            S.v[k] = w.v[k];
            S.xe[k] = w.xe[k];
            S.ve[k] = w.ve[k];
        }
        w.xk[0][k] = w.v[k];
    }
    if (!attempt) return;
    tiny_lists(w.f, S.m, S.n, S.massless);
    tiny_force(w.f, w.x, w.vk[0], S.G, eps2);
    for (int s = 1; s < R.stages; ++s) {
        for (int e = t; e < 2 * L; e += TY_THREADS) {
            const bool pos = e >= L;
            const int k = pos ? e - L : e;
            double q = 0.0;
            for (int i = 0; i < s; ++i)
                q = __dadd_rn(q, __dmul_rn(R.a[s][i], pos ? w.xk[i][k] : w.vk[i][k]));
            q = __dadd_rn(__dadd_rn(pos ? w.x[k] : w.v[k], __dmul_rn(h, q)), pos ? w.xe[k] : w.ve[k]);
            (pos ? w.xs : w.xk[s])[k] = q;
        }
        __syncthreads();
        tiny_force(w.f, w.xs, w.vk[s], S.G, eps2);
    }
    // the weighted sums of velocity, position and their error terms
    for (int e = t; e < 4 * L; e += TY_THREADS) {
        const int kind = e / L, k = e % L;
        double q = 0.0;
        for (int s = 0; s < R.stages; ++s)
            q = __dadd_rn(q, __dmul_rn(kind < 2 ? R.b[s] : R.dtdw[s], kind & 1 ? w.xk[s][k] : w.vk[s][k]));
        w.end[kind][k] = q;
    }
    __syncthreads();
    for (int e = t; e < 2 * L; e += TY_THREADS) {
        const bool pos = e >= L;
        const int k = pos ? e - L : e;
        const double y0 = pos ? w.x[k] : w.v[k];
        double err = __dadd_rn(pos ? w.xe[k] : w.ve[k], __dmul_rn(h, w.end[pos ? 1 : 0][k]));
        const double yn = __dadd_rn(y0, err);
        err = __dadd_rn(err, __dsub_rn(y0, yn));
        (pos ? S.x1 : S.v1)[k] = yn;
        (pos ? S.txe : S.tve)[k] = err;
        const double scale = __dadd_rn(tol, __dmul_rn(fmax(fabs(y0), fabs(yn)), tol));
        const double q = __ddiv_rn(w.end[pos ? 3 : 2][k], scale);
        terms[2 * k + (pos ? 1 : 0)] = __dmul_rn(q, q);
    }
}

// ---- IAS15 ----------------------------------------------------------------------
struct IasShared {
    TinyForce f;
    double x[TY_L], v[TY_L], a[TY_L], xe[TY_L], ve[TY_L], x1[TY_L], x1_first[TY_L];
    double f0[TY_L], fi[TY_L], b6_old[TY_L];
    double b[7][TY_L], g[7][TY_L], q[14][TY_L];
    double cg[28][TY_L];   // c_jr g_j, j >= r, at j (j + 1) / 2 + r
    unsigned long long top[2];
};

// The divisors of the position and velocity series, with their reciprocals.
struct Known {
    double d, zh, zl;
};

__device__ __forceinline__ double quotient(const Known &k, double x)
{
    return is_zero(x) ? x : div_known(x, k.d, k.zh, k.zl, true);
}

// Largest |u| and |w| over the elements, NaN skipped (launch_ias_absmax2).
__device__ void tiny_absmax(IasShared &w, const double *u, const double *v, int L)
{
    if (threadIdx.x < 2) w.top[threadIdx.x] = 0ull;
    __syncthreads();
    for (int k = threadIdx.x; k < L; k += TY_THREADS) {
        const long long mu = abs_bits(u[k]), mv = abs_bits(v[k]);
        if (mu <= 0x7ff0000000000000ll) atomicMax(&w.top[0], (unsigned long long)mu);
        if (mv <= 0x7ff0000000000000ll) atomicMax(&w.top[1], (unsigned long long)mv);
    }
    __syncthreads();
}

// One IAS15 step of size h (src/integrator_ias15.c:229-616) from the state, after
// the previous step became the state, and its b were carried over, if it was
// accepted.  out[0..1] receive the bits of max |b_6| and max |a(x1)|; step false:
// only the acceptance.
__global__ void __launch_bounds__(TY_THREADS)
k_tiny_ias15(TinySystem S, TinyIas I, bool accept, bool refine, bool step, double h,
             unsigned long long *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char ty_smem[];
    __shared__ Known s_px[7], s_pv[7];
    IasShared &w = *reinterpret_cast<IasShared *>(ty_smem);
    const int L = 3 * S.n, t = threadIdx.x;
    const double eps2 = __dmul_rn(S.eps, S.eps);
    if (t < 14) {
        // x: b_r over (r + 2)(r + 3) / 2; v: b_r over r + 2
        const int r = t % 7;
        Known k;
        k.d = t < 7 ? (double)((r + 2) * (r + 3) / 2) : (double)(r + 2);
        reciprocal2(k.d, k.zh, k.zl);
        (t < 7 ? s_px : s_pv)[r] = k;
    }
    for (int k = t; k < L; k += TY_THREADS) {
        if (accept) {
            S.x[k] = S.x1[k];
            S.v[k] = S.v1[k];
            S.xe[k] = S.txe[k];
            S.ve[k] = S.tve[k];
            S.a[k] = I.a1[k];
        }
        w.x[k] = S.x[k];
        w.v[k] = S.v[k];
        w.xe[k] = S.xe[k];
        w.ve[k] = S.ve[k];
        w.a[k] = S.a[k];
        w.b6_old[k] = I.b6_old[k];
    }
    for (int e = t; e < 7 * L; e += TY_THREADS) {
        const int r = e / L, k = e % L;
        w.g[r][k] = I.g[e];
        w.b[r][k] = I.b[e];
    }
    __syncthreads();
    if (accept) {
        // b of the next step (src/integrator_ias15.c:1276-1382): row r of the
        // binomial triangle, highest b first
        for (int e = t; e < 7 * L; e += TY_THREADS) {
            const int r = e / L, k = e % L;
            int c = 1;
            for (int j = r; j < 6; ++j) c = c * (j + 2) / (j + 1 - r);   // C(7, r + 1)
            double s = 0.0;
            for (int j = 6; j >= r; --j) {
                const double term = j == r ? w.b[j][k] : __dmul_rn(w.b[j][k], (double)c);
                s = j == 6 ? term : __dadd_rn(s, term);
                c = c * (j - r) / (j + 1);   // C(j, r + 1)
            }
            const double en = __dmul_rn(I.q[r], s);
            const double db = refine ? __dsub_rn(w.b[r][k], I.e[e]) : 0.0;
            I.e[e] = en;
            w.q[r][k] = __dadd_rn(en, db);
        }
        __syncthreads();
        for (int e = t; e < 7 * L; e += TY_THREADS) {
            const int r = e / L, k = e % L;
            w.b[r][k] = w.q[r][k];
            if (!step) I.b[e] = w.q[r][k];
        }
        __syncthreads();
    }
    if (!step) return;
    tiny_lists(w.f, S.m, S.n, S.massless);
    // The predictor's quotients, b_r over its divisor (b_6 times the spacing): kept
    // up to date where b or the spacing changes, beside other work, instead of all
    // formed again at every spacing (650 of 6,800 cycles).
    for (int e = t; e < 7 * L; e += TY_THREADS) {
        const int r = e / L, k = e % L;
        w.q[r][k] = quotient(s_px[r], r == 6 ? __dmul_rn(I.spacing[0], w.b[6][k]) : w.b[r][k]);
    }
    // Products of b = sum_j c_jr g_j: at a spacing only g_{i-1} changes, so one of
    // the seven is formed and the chain of b is additions.
    for (int e = t; e < 28 * L; e += TY_THREADS) {
        const int row = e / L, k = e % L;
        int j = 0;
        while ((j + 1) * (j + 2) / 2 <= row) ++j;
        w.cg[row][k] = __dmul_rn(I.c[j][row - j * (j + 1) / 2], w.g[j][k]);
    }
    __syncthreads();
    for (int it = 0; it < 12; ++it) {
        for (int i = 0; i < 8; ++i) {
            // predictor at spacing hi (:808-919); the velocities are not needed,
            // the force depends on positions alone
            const double hi = I.spacing[i], next = I.spacing[(i + 1) & 7];
            const double dth = __dmul_rn(h, hi);
            bool same = it > 0 && i == 0;
            for (int k = t; k < L; k += TY_THREADS) {
                double p = __dadd_rn(w.q[5][k], w.q[6][k]);
                for (int r = 4; r >= 0; --r) p = __dadd_rn(w.q[r][k], __dmul_rn(hi, p));
                const double acc = __dmul_rn(
                    __dmul_rn(dth, __dadd_rn(w.a[k], __dmul_rn(hi, p))), 0.5);
                const double xv = __dadd_rn(
                    w.x[k], __dadd_rn(w.xe[k], __dmul_rn(dth, __dadd_rn(w.v[k], acc))));
                w.x1[k] = xv;
                if (i == 0) {
                    same = same && __double_as_longlong(xv) == __double_as_longlong(w.x1_first[k]);
                    w.x1_first[k] = xv;
                }
            }
            if (i == 0) {
                // spacing 0: the same positions in every iteration
                const bool again = __syncthreads_and(same);
                for (int k = t; k < L; k += TY_THREADS)
                    w.q[6][k] = quotient(s_px[6], __dmul_rn(next, w.b[6][k]));
                if (!again) tiny_force(w.f, w.x1, w.f0, S.G, eps2);
                __syncthreads();
                continue;
            }
            __syncthreads();
            tiny_force(w.f, w.x1, w.fi, S.G, eps2);
            // g_{i-1} (:1117-1274); the lower ones have not changed since they
            // were formed in this iteration
            for (int k = t; k < L; k += TY_THREADS) {
                double q = __dmul_rn(__dsub_rn(w.fi[k], w.f0[k]), I.r[i][0]);
                for (int j = 1; j < i; ++j) q = __dmul_rn(__dsub_rn(q, w.g[j - 1][k]), I.r[i][j]);
                w.g[i - 1][k] = q;
            }
            __syncthreads();
            // b from g (:985-1115), and the quotients at the next spacing
            for (int e = t; e < min(i + 1, 7) * L; e += TY_THREADS) {
                const int r = e < i * L ? e / L : 6, k = e % L;
                double q = w.b[r][k];
                if (e < i * L) {
                    const int j0 = i - 1;   // r <= j0
                    const double fresh = __dmul_rn(I.c[j0][r], w.g[j0][k]);
                    w.cg[j0 * (j0 + 1) / 2 + r][k] = fresh;
                    q = r == j0 ? fresh : w.cg[r * (r + 1) / 2 + r][k];
                    for (int j = r + 1; j < 7; ++j)
                        q = __dadd_rn(q, j == j0 ? fresh : w.cg[j * (j + 1) / 2 + r][k]);
                    w.b[r][k] = q;
                }
                w.q[r][k] = quotient(s_px[r], r == 6 ? __dmul_rn(next, q) : q);
            }
            __syncthreads();
        }
        for (int k = t; k < L; k += TY_THREADS) {
            w.q[13][k] = __dsub_rn(w.b[6][k], w.b6_old[k]);
            w.b6_old[k] = w.b[6][k];
        }
        __syncthreads();
        tiny_absmax(w, w.q[13], w.fi, L);
        const double ratio = __ddiv_rn(__longlong_as_double((long long)w.top[0]),
                                       __longlong_as_double((long long)w.top[1]));
        if (ratio < 1e-16) break;   // CTA-uniform
        __syncthreads();
    }
    // end of the step with compensated sums (:921-983)
    for (int e = t; e < 14 * L; e += TY_THREADS) {
        const int r = e / L, k = e % L;
        w.q[r][k] = r < 7 ? quotient(s_px[r], w.b[r][k]) : quotient(s_pv[r - 7], w.b[r - 7][k]);
    }
    __syncthreads();
    for (int e = t; e < 2 * L; e += TY_THREADS) {
        const bool pos = e < L;
        const int k = pos ? e : e - L;
        double s = w.a[k];
        for (int r = 0; r < 7; ++r) s = __dadd_rn(s, w.q[pos ? r : 7 + r][k]);
        double err, y0;
        if (pos) {
            y0 = w.x[k];
            err = __dadd_rn(w.xe[k], __dmul_rn(h, __dadd_rn(w.v[k], __dmul_rn(__dmul_rn(h, s), 0.5))));
        } else {
            y0 = w.v[k];
            err = __dadd_rn(w.ve[k], __dmul_rn(h, s));
        }
        const double yn = __dadd_rn(y0, err);
        err = __dadd_rn(err, __dsub_rn(y0, yn));
        (pos ? S.x1 : S.v1)[k] = yn;
        (pos ? S.txe : S.tve)[k] = err;
        if (pos) w.x1[k] = yn;
    }
    __syncthreads();
    tiny_force(w.f, w.x1, w.fi, S.G, eps2);
    tiny_absmax(w, w.b[6], w.fi, L);
    for (int k = t; k < L; k += TY_THREADS) {
        I.a1[k] = w.fi[k];
        I.b6_old[k] = w.b6_old[k];
    }
    for (int e = t; e < 7 * L; e += TY_THREADS) {
        I.b[e] = w.b[e / L][e % L];
        I.g[e] = w.g[e / L][e % L];
    }
    if (t < 2) out[t] = w.top[t];
}

ErrorStatus tiny_setup()
{
    GS_CUDA(cudaFuncSetAttribute(k_tiny_fixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(FixedShared)));
    GS_CUDA(cudaFuncSetAttribute(k_tiny_rk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RkShared)));
    GS_CUDA(cudaFuncSetAttribute(k_tiny_ias15, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(IasShared)));
    return ok();
}

void launch_tiny_fixed(const TinySystem &S, int integrator, int steps, double h, cudaStream_t s)
{
    k_tiny_fixed<<<1, TY_THREADS, sizeof(FixedShared), s>>>(S, integrator, steps, h);
}

void launch_tiny_rk(const TinySystem &S, const TinyRk &R, bool accept, bool attempt, double h,
                    double tol, double *terms, cudaStream_t s)
{
    k_tiny_rk<<<1, TY_THREADS, sizeof(RkShared), s>>>(S, R, accept, attempt, h, tol, terms);
}

void launch_tiny_ias15(const TinySystem &S, const TinyIas &I, bool accept, bool refine, bool step,
                       double h, unsigned long long *out, cudaStream_t s)
{
    k_tiny_ias15<<<1, TY_THREADS, sizeof(IasShared), s>>>(S, I, accept, refine, step, h, out);
}

}  // namespace gs
