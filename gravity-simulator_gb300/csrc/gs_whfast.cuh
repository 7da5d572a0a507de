// gs_whfast.cuh -- what the WHFast kernels share (k_whfast.cu: ensembles;
// k_whfast_small.cu: small systems, many steps per launch).
#pragma once

#include "gs_fp64.cuh"
#include "gs_internal.h"

namespace gs {

// Ensemble integrator / acceleration variants.
enum { WH_MASSLESS = 0, WH_PAIRWISE = 1 };

// Largest system of an ensemble: the per-system sort holds 12 bytes per
// slot of the next power of two in shared memory (192 KiB at 16384).
constexpr int kEnsembleMaxSystem = 16384;

// Shared pair sums of the interaction acceleration (k_wh_pairs): used when a
// system has at most kPairMax massive bodies.
constexpr int kPairMax = 32;
constexpr int kPairSlots = kPairMax + 1;

struct EnsDev {
    int S;
    const int *off;      // [S+1]
    int *cnt;            // [S]
    const int *sys_of;   // [P]
    int *ids;
    double *x, *v, *m, *jx, *jv, *a, *eta;
    int *hv;             // massive-body list (indices within the system), per system at off[s]
    int *nh;             // [S]
    int *rm;             // [P] removal marks
    int *nrm;            // [S]
    double *pairs;       // [S][2 * kPairSlots][3] shared pair sums
    // Jacobi -> Cartesian pass (k_wh_seq_scan / _chain / _fill)
    int *seq_nmass;      // [S] massive particles (run path), -1: whole chain, -2: empty
    int *seq_runs;       // [S] massless runs recorded
    int *run_lo, *run_hi;   // [S][kSeqMassMax + 1] first / last slot of a run
    double *run_y;       // [S][kSeqMassMax + 1][6] offsets of a run's x and v
    // scratch for the permutation
    int *t_ids;
    double *t_x, *t_v, *t_m;
    unsigned *status;
    double G, eps;
    int variant;
    int remove_invalid;
};

__device__ __forceinline__ double dot3(const double *a, const double *b)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}

__device__ __forceinline__ double norm3d(const double *a) { return __dsqrt_rn(dot3(a, a)); }

// Sort key of a distance: its bit pattern (distances are >= 0, so the
// patterns order like the values), NaN after +inf, padding after all.
// This keeps the comparison a total order whatever the input, so every
// live slot receives a live index.
__device__ __forceinline__ unsigned long long dist_key(double d)
{
    const unsigned long long k = (unsigned long long)abs_bits(d);
    return k > 0x7ff0000000000000ull ? 0x7ff8000000000000ull : k;
}

__device__ __forceinline__ bool neg_zero(double v)
{
    return __double_as_longlong(v) == (long long)0x8000000000000000ull;
}

// Quotients x / d by the divisors d of the Stumpff series, correctly
// rounded without a division.  zh = RN(1/d) and zl = RN(1/d - zh) (exact
// rationals rounded once); q = RN(x zh + RN(x zl)) is within an ulp of x/d
// (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE
// Trans. Computers 53(8), 2004), and one correction with the exact remainder
// r = x - q d gives RN(q + r zh) = RN(x/d) (Markstein, IBM J. Res. Dev.
// 34(1), 1990: a faithful quotient and a correctly rounded reciprocal).
// Where |zl| <= 2^-54 zh, RN(x zh) is itself within an ulp (x zh is within half
// an ulp of x/d), which saves the product with zl: all divisors but 182 and 210.
// The remainder is exact while its last bit stays above the subnormal
// range, so |x| with an exponent outside [-960, 960) (zeros, subnormals,
// infinities, NaN) takes the division itself.  Checked against __ddiv_rn bit for
// bit by gsgpu_stumpff_division_selftest.
struct StumpffDiv {
    double d, zh, zl;
};
enum { SD6, SD12, SD20, SD30, SD42, SD56, SD72, SD90, SD110, SD132, SD156, SD182, SD210, kStumpffDivs };
static __constant__ StumpffDiv kStumpffDiv[kStumpffDivs] = {
    {6.0, 0x1.5555555555555p-3, 0x1.5555555555555p-57},
    {12.0, 0x1.5555555555555p-4, 0x1.5555555555555p-58},
    {20.0, 0x1.999999999999ap-5, -0x1.999999999999ap-59},
    {30.0, 0x1.1111111111111p-5, 0x1.1111111111111p-61},
    {42.0, 0x1.8618618618618p-6, 0x1.8618618618618p-60},
    {56.0, 0x1.2492492492492p-6, 0x1.2492492492492p-60},
    {72.0, 0x1.c71c71c71c71cp-7, 0x1.c71c71c71c71cp-61},
    {90.0, 0x1.6c16c16c16c17p-7, -0x1.f49f49f49f49fp-62},
    {110.0, 0x1.29e4129e4129ep-7, 0x1.04a7904a7904ap-61},
    {132.0, 0x1.f07c1f07c1f08p-8, -0x1.f07c1f07c1f08p-63},
    {156.0, 0x1.a41a41a41a41ap-8, 0x1.0690690690690p-62},
    {182.0, 0x1.6816816816817p-8, -0x1.fa5fa5fa5fa60p-62},
    {210.0, 0x1.3813813813814p-8, -0x1.fb1fb1fb1fb20p-62},
};

// ---- small systems (k_whfast_small.cu) ------------------------------------------
// Largest system and largest number of massive bodies of the small-system path.
constexpr int kSmallMax = 48;
constexpr int kSmallMassive = 16;
// `steps` steps of h of every system, one CTA each.
void launch_wh_small(const EnsDev &E, int steps, double h, cudaStream_t s);

}  // namespace gs
