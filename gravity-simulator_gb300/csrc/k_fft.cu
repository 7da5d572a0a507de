// k_fft.cu -- FP64 convolution of a real g^3 mesh with a real, even kernel given
// by its transform (the particle-mesh potential), for the 15 sizes g of convolve_for:
// 32, 40, 48, 60, 64, 72, 80, 96, 100, 120, 128, 144, 160, 192 and 256.
//
// The mesh is read as g x g x g/2 complex numbers, two neighbours on the last
// axis in one: C = E + i O with E the even and O the odd planes.  Transforms
// along the first two axes act on both at once; the last axis takes the modes
// (kx, ky) and (-kx, -ky) together, which give
//     E = (C(k) + conj C(-k)) / 2,    O = -i (C(k) - conj C(-k)) / 2,
// transforms E and O (length g/2), joins them to the g modes along kz by one more
// radix-2 step, multiplies by the kernel, and goes back the same way.  Five
// launches in place, every pass over g^3 doubles, and no half spectrum:
//     j forward, i forward, k forward x kernel x k inverse, i inverse, j inverse.
//
// A line of N = R1 R2 points, n = c + R2 r, k = q + R1 s (Cooley and Tukey, 1965):
// R2 threads each transform R1 points over r in registers, multiply by
// exp(-2 pi i c q / N), exchange through shared memory, and transform R2 points
// over c (for R1 > R2 several times, and where R2 does not divide R1 with idle
// threads).  The inverse of the last axis takes the same steps backwards, so its
// input is where the forward transform left it.
//
// Bound: the FP64 pipe (an FP64 warp instruction holds its SM sub-partition for
// 64 cycles): at g = 128, 1.38e8 operations, 221 us.  The library's transforms
// took 490 us there and the multiplication 8; these five launches take 292 (46 for
// each pass of lines, 108 for the pairs).  A step with 24^3 particles, before and
// now: g = 32 104 and 54 us, 48 104 and 70, 60 145 and 84, 96 297 and 174, 160 1311
// and 825, 256 4195 and 2762.  Accelerations differ from an extended
// precision computation by as much with either (1e-14 at g = 32 to 256).
#include "gs_fft.h"

namespace gs {
namespace {

constexpr double kSqrtHalf = 0.70710678118654752440;   // cos(pi / 4)
constexpr double kCos8 = 0.92387953251128675613;       // cos(pi / 8)
constexpr double kSin8 = 0.38268343236508977173;       // sin(pi / 8)
constexpr double kSin3 = 0.86602540378443864676;       // sin(2 pi / 3)
constexpr double kCos5 = 0.30901699437494742410;       // cos(2 pi / 5)
constexpr double kSin5 = 0.95105651629515357212;       // sin(2 pi / 5)
constexpr double kCos25 = -0.80901699437494742410;     // cos(4 pi / 5)
constexpr double kSin25 = 0.58778525229247312917;      // sin(4 pi / 5)

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// a (w.x + i w.y), for the inverse a (w.x - i w.y)
template <bool INV>
__device__ __forceinline__ double2 cmul(double2 a, double2 w)
{
    const double wy = INV ? -w.y : w.y;
    return make_double2(fma(a.x, w.x, -(a.y * wy)), fma(a.x, wy, a.y * w.x));
}

// a exp(-+ i pi / 2)
template <bool INV>
__device__ __forceinline__ double2 quarter(double2 a)
{
    return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// a exp(-+ i pi / 4)
template <bool INV>
__device__ __forceinline__ double2 eighth(double2 a)
{
    return INV ? make_double2(kSqrtHalf * (a.x - a.y), kSqrtHalf * (a.x + a.y))
               : make_double2(kSqrtHalf * (a.x + a.y), kSqrtHalf * (a.y - a.x));
}

// In place, natural order: v[k] <- sum_n v[n] exp(-+ 2 pi i n k / R).
template <int R, bool INV>
struct Dft;

template <bool INV>
struct Dft<2, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    }
};

template <bool INV>
struct Dft<3, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = cadd(v[1], v[2]), d = quarter<INV>(csub(v[1], v[2]));
        const double2 p = make_double2(fma(-0.5, a.x, v[0].x), fma(-0.5, a.y, v[0].y));
        v[0] = cadd(v[0], a);
        v[1] = make_double2(fma(kSin3, d.x, p.x), fma(kSin3, d.y, p.y));
        v[2] = make_double2(fma(-kSin3, d.x, p.x), fma(-kSin3, d.y, p.y));
    }
};

template <bool INV>
struct Dft<5, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = cadd(v[1], v[4]), b = cadd(v[2], v[3]);
        const double2 c = quarter<INV>(csub(v[1], v[4])), d = quarter<INV>(csub(v[2], v[3]));
        const double2 p = make_double2(fma(kCos5, a.x, fma(kCos25, b.x, v[0].x)),
                                       fma(kCos5, a.y, fma(kCos25, b.y, v[0].y)));
        const double2 q = make_double2(fma(kCos25, a.x, fma(kCos5, b.x, v[0].x)),
                                       fma(kCos25, a.y, fma(kCos5, b.y, v[0].y)));
        const double2 r = make_double2(fma(kSin5, c.x, kSin25 * d.x), fma(kSin5, c.y, kSin25 * d.y));
        const double2 t = make_double2(fma(kSin25, c.x, -(kSin5 * d.x)), fma(kSin25, c.y, -(kSin5 * d.y)));
        v[0] = cadd(v[0], cadd(a, b));
        v[1] = cadd(p, r);
        v[4] = csub(p, r);
        v[2] = cadd(q, t);
        v[3] = csub(q, t);
    }
};

// R = A B with A and B coprime, without twiddle factors (Good, 1958): with
// n = B n1 + A n2 mod R and k the number that is k1 mod A and k2 mod B.
template <int A, int B, bool INV>
struct Coprime {
    static constexpr int R = A * B;
    static constexpr int index(int k1, int k2)
    {
        int k = 0;
        while (k % A != k1 || k % B != k2) ++k;
        return k;
    }
    template <int K1, int K2>
    static __device__ __forceinline__ void place(double2 *v, const double2 (&t)[A][B])
    {
        constexpr int k = index(K1, K2);
        v[k] = t[K1][K2];
        if constexpr (K2 + 1 < B)
            place<K1, K2 + 1>(v, t);
        else if constexpr (K1 + 1 < A)
            place<K1 + 1, 0>(v, t);
    }
    static __device__ __forceinline__ void run(double2 *v)
    {
        double2 t[A][B];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
            double2 u[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) u[n1] = v[(B * n1 + A * n2) % R];
            Dft<A, INV>::run(u);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) t[k1][n2] = u[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) Dft<B, INV>::run(t[k1]);
        place<0, 0>(v, t);
    }
};

template <bool INV>
struct Dft<6, INV> : Coprime<2, 3, INV> {};
template <bool INV>
struct Dft<10, INV> : Coprime<2, 5, INV> {};
template <bool INV>
struct Dft<12, INV> : Coprime<4, 3, INV> {};

template <bool INV>
struct Dft<4, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const double2 c = cadd(v[1], v[3]), d = quarter<INV>(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};

template <bool INV>
struct Dft<8, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4, INV>::run(e);
        Dft<4, INV>::run(o);
        o[1] = eighth<INV>(o[1]);
        o[2] = quarter<INV>(o[2]);
        o[3] = quarter<INV>(eighth<INV>(o[3]));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    }
};

template <bool INV>
struct Dft<16, INV> {
    static __device__ __forceinline__ void run(double2 *v)
    {
        double2 e[8], o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            e[k] = v[2 * k];
            o[k] = v[2 * k + 1];
        }
        Dft<8, INV>::run(e);
        Dft<8, INV>::run(o);
        o[1] = cmul<INV>(o[1], make_double2(kCos8, -kSin8));
        o[2] = eighth<INV>(o[2]);
        o[3] = cmul<INV>(o[3], make_double2(kSin8, -kCos8));
        o[4] = quarter<INV>(o[4]);
        o[5] = cmul<INV>(o[5], make_double2(-kSin8, -kCos8));
        o[6] = quarter<INV>(eighth<INV>(o[6]));
        o[7] = cmul<INV>(o[7], make_double2(-kCos8, -kSin8));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            v[k] = cadd(e[k], o[k]);
            v[k + 8] = csub(e[k], o[k]);
        }
    }
};

// N = R1 R2.  Where R2 does not divide R1, threads are idle in the second step;
// the order of the factors is the one with fewer operations in all.
constexpr int first_radix(int n)
{
    switch (n) {
    case 16: return 4;
    case 20: return 5;
    case 24: case 30: case 36: case 48: return 6;
    case 32: case 40: case 64: return 8;
    case 50: case 60: case 80: case 100: return 10;
    case 72: case 96: case 120: case 144: return 12;
    default: return 16;   // 128, 160, 192, 256
    }
}
template <int N>
struct Split {
    static constexpr int R1 = first_radix(N), R2 = N / R1;
    static_assert(R1 * R2 == N, "two radices");
};

// Lines take the smaller radix first: a line is then shared by as many threads as
// the larger one, each with less work, which fills the sub-partitions more evenly (in
// the second step as many are busy as the smaller one; neighbouring blocks take
// different ones).  Unless only the other order fills whole warps: a block is eight
// lines, so its threads are a multiple of 32 where the second radix is one of 4.
// Step with 24^3 particles, the larger radix first and the smaller one: g = 32 61.8
// and 53.6 us, 40 68.1 and 62.2, 60 86.3 and 84.3, 72 115 and 108, 80 (10 x 8) 132
// and 142, 96 173 and 174, 120 382 and 347, 128 371 and 351, 160 877 and 825, 192 both
// 1240.
template <int N>
struct LineSplit {
    static constexpr int A = Split<N>::R1, B = Split<N>::R2;
    static constexpr int SMALL = A < B ? A : B, LARGE = A < B ? B : A;
    static constexpr int R1 = LARGE % 4 != 0 && SMALL % 4 == 0 ? LARGE : SMALL, R2 = N / R1;
};

// Lines along one of the first two axes.  A CTA takes LINES neighbouring lines
// (128-byte rows) of one slab; line l of slab o starts at o outer + l, its points
// are `stride` apart.  tw: exp(-2 pi i k / N).  FIRST: the mesh holds densities,
// read as their contrast.
constexpr int LINES = 8;

template <int N, bool INV, bool FIRST = false>
__global__ void __launch_bounds__(LINES *LineSplit<N>::R2)
k_fft_lines(double2 *__restrict__ data, unsigned lines_per_slab, size_t outer, unsigned stride,
            const double2 *__restrict__ tw, MeshScale scale = {nullptr, 1.0})
{
    constexpr int R1 = LineSplit<N>::R1, R2 = LineSplit<N>::R2, M = (R1 + R2 - 1) / R2;
    __shared__ double2 s[N * LINES];
    const unsigned tiles = (lines_per_slab + LINES - 1) / LINES;
    const unsigned slab = blockIdx.x / tiles, tile = blockIdx.x - slab * tiles;
    const int line = threadIdx.x % LINES, t = threadIdx.x / LINES;
    const bool live = tile * LINES + line < lines_per_slab;
    double2 *base = data + (size_t)slab * outer + tile * LINES + line;
    double2 v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r)
        v[r] = live ? base[(size_t)(t + R2 * r) * stride] : make_double2(0.0, 0.0);
    if (FIRST) {
        const double f = scale.device ? *scale.device : scale.value;
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = make_double2(contrast(v[r].x, f), contrast(v[r].y, f));
    }
    Dft<R1, INV>::run(v);
#pragma unroll
    for (int q = 0; q < R1; ++q) {
        if (q > 0) v[q] = cmul<INV>(v[q], __ldg(tw + t * q));
        s[(t * R1 + q) * LINES + line] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < M; ++u) {
        const int q = (R1 < R2 ? (t + (blockIdx.x & 1) * R1) % R2 : t) + R2 * u;
        if (R1 % R2 != 0 && q >= R1) break;
        double2 w[R2];
#pragma unroll
        for (int c = 0; c < R2; ++c) w[c] = s[(c * R1 + q) * LINES + line];
        Dft<R2, INV>::run(w);
        if (live) {
#pragma unroll
            for (int k = 0; k < R2; ++k) base[(size_t)(q + R1 * k) * stride] = w[k];
        }
    }
}

__device__ __forceinline__ double2 from_partner(double2 a)
{
    return make_double2(__shfl_xor_sync(0xffffffffu, a.x, 1), __shfl_xor_sync(0xffffffffu, a.y, 1));
}

__device__ __forceinline__ double2 swapped(double2 a, bool swap)
{
    return swap ? make_double2(a.y, a.x) : a;
}

// The last axis: lines P = (i, j) and Q = (-i, -j), of H = G / 2 points, whose
// modes are conjugates of each other's.  Neighbouring lanes work on the pair:
// the even lane on P and E, the odd lane on Q and O.
template <int G>
struct PairShape {
    static constexpr int H = G / 2, R1 = Split<H>::R1, R2 = Split<H>::R2;
    static constexpr int M = (R1 + R2 - 1) / R2;
    static constexpr int PER = 2 * R2;              // threads of a pair
    static constexpr int PAIRS = 128 / PER;         // pairs of a CTA
    static constexpr int ROW = R2 + 1;              // padded row of the exchange
    // pairs of the mesh: rows i = 1 .. H - 1 whole, rows 0 and H up to j = H
    static constexpr unsigned COUNT = (unsigned)(H - 1) * G + 2u * (H + 1);
};

template <int G>
__global__ void __launch_bounds__(128)
k_fft_pairs(double2 *__restrict__ data, const double *__restrict__ table,
            const double2 *__restrict__ tw)
{
    using S = PairShape<G>;
    constexpr int H = S::H, R1 = S::R1, R2 = S::R2, M = S::M;
    __shared__ double2 s[S::PAIRS * 2 * R1 * S::ROW];
    const int odd = threadIdx.x & 1, t = (threadIdx.x % S::PER) >> 1, local = threadIdx.x / S::PER;
    const unsigned pair = blockIdx.x * S::PAIRS + local;
    const bool held = local < S::PAIRS;   // the block's last threads may have no pair
    const bool live = held && pair < S::COUNT;
    unsigned i = 0, j = 0;
    if (live) {
        constexpr unsigned kWhole = (unsigned)(H - 1) * G;
        if (pair < kWhole) {
            i = 1 + pair / G;
            j = pair % G;
        } else {
            const unsigned e = pair - kWhole;
            i = e < H + 1 ? 0 : H;
            j = e < H + 1 ? e : e - (H + 1);
        }
    }
    const unsigned ni = (G - i) % G, nj = (G - j) % G;
    const bool self = ni == i && nj == j;
    double2 *line = data + (size_t)(odd ? ni * G + nj : i * G + j) * H;
    double2 *ex = s + (min(local, S::PAIRS - 1) * 2 + odd) * R1 * S::ROW;
    // E and O from the two lines
    double2 v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        const double2 own = live ? line[t + R2 * r] : make_double2(0.0, 0.0);
        const double2 a = swapped(own, odd), b = swapped(from_partner(own), odd);
        v[r] = make_double2(a.x + b.x, a.y - b.y);
    }
    Dft<R1, false>::run(v);
#pragma unroll
    for (int q = 0; q < R1; ++q) {
        if (q > 0) v[q] = cmul<false>(v[q], __ldg(tw + 2 * t * q));
        if (held) ex[q * S::ROW + t] = v[q];
    }
    __syncthreads();
    // modes m (even lane) and m + H (odd lane): F = E + w O, E - w O
    const int kx = i <= (unsigned)H ? (int)i : (int)i - G, ky = j <= (unsigned)H ? (int)j : (int)j - G;
    const int k2 = kx * kx + ky * ky;
    const double sign = odd ? -1.0 : 1.0;
    double2 w[M][R2];
#pragma unroll
    for (int u = 0; u < M; ++u) {
        const int q = min(t + R2 * u, R1 - 1);   // threads without one repeat the last
#pragma unroll
        for (int c = 0; c < R2; ++c) w[u][c] = ex[q * S::ROW + c];
        Dft<R2, false>::run(w[u]);
#pragma unroll
        for (int k = 0; k < R2; ++k) {
            const int m = q + R1 * k;
            double2 f = __ldg(tw + m);
            f = odd ? f : make_double2(1.0, 0.0);
            const double2 own = cmul<false>(w[u][k], f);
            const double2 other = from_partner(own);
            const int kz = odd ? H - m : m;   // |m + H - G| on the odd lane
            const double g = 0.5 * __ldg(table + k2 + kz * kz);
            const double2 F = make_double2(fma(sign, own.x, other.x) * g, fma(sign, own.y, other.y) * g);
            const double2 P = from_partner(F);
            // E' = F(m) + F(m + H), O' = conj(w) (F(m) - F(m + H))
            w[u][k] = cmul<true>(make_double2(fma(sign, F.x, P.x), fma(sign, F.y, P.y)), f);
        }
        Dft<R2, true>::run(w[u]);
    }
    // back: twiddle and exchange, then R1 points over q
    __syncthreads();
#pragma unroll
    for (int u = 0; u < M; ++u) {
        const int q = min(t + R2 * u, R1 - 1);
#pragma unroll
        for (int c = 0; c < R2; ++c) {
            if (c > 0) w[u][c] = cmul<true>(w[u][c], __ldg(tw + 2 * c * q));
            if (held && t + R2 * u < R1) ex[q * S::ROW + c] = w[u][c];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < R1; ++q) v[q] = ex[q * S::ROW + t];
    Dft<R1, true>::run(v);
    // P = E + i O, Q = conj E + i conj O
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        const double2 other = from_partner(v[r]);
        const double2 a = swapped(v[r], odd), b = swapped(other, !odd);
        if (live && !(self && odd))
            line[t + R2 * r] = make_double2(fma(-sign, b.x, a.x), fma(sign, b.y, a.y));
    }
}

__global__ void k_fft_table(int g, double2 *__restrict__ tw)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= g) return;
    double sn, cs;
    sincospi(-2.0 * k / g, &sn, &cs);
    tw[k] = make_double2(cs, sn);
}

template <int G>
void convolve(double2 *data, const MeshScale &scale, const double *table, const double2 *tw,
              cudaStream_t s)
{
    constexpr unsigned H = G / 2;
    constexpr int threads = LINES * LineSplit<G>::R2;
    constexpr unsigned slabs = G * ((H + LINES - 1) / LINES), planes = (G * H + LINES - 1) / LINES;
    using S = PairShape<G>;
    k_fft_lines<G, false, true><<<slabs, threads, 0, s>>>(data, H, (size_t)G * H, H, tw, scale);
    k_fft_lines<G, false><<<planes, threads, 0, s>>>(data, G * H, 0, G * H, tw);
    k_fft_pairs<G><<<(S::COUNT + S::PAIRS - 1) / S::PAIRS, 128, 0, s>>>(data, table, tw);
    k_fft_lines<G, true><<<planes, threads, 0, s>>>(data, G * H, 0, G * H, tw);
    k_fft_lines<G, true><<<slabs, threads, 0, s>>>(data, H, (size_t)G * H, H, tw);
}

}  // namespace

using Convolve = void (*)(double2 *, const MeshScale &, const double *, const double2 *, cudaStream_t);

// The sizes that are built: multiples of four whose lines and half lines are products
// of two of the radices above, each measured faster than the library's transforms.
// Every other size goes to the library, also 36 and 50, whose factors would fit.
static Convolve convolve_for(int g)
{
    switch (g) {
    case 32: return convolve<32>;
    case 40: return convolve<40>;
    case 48: return convolve<48>;
    case 60: return convolve<60>;
    case 64: return convolve<64>;
    case 72: return convolve<72>;
    case 80: return convolve<80>;
    case 96: return convolve<96>;
    case 100: return convolve<100>;
    case 120: return convolve<120>;
    case 128: return convolve<128>;
    case 144: return convolve<144>;
    case 160: return convolve<160>;
    case 192: return convolve<192>;
    case 256: return convolve<256>;
    default: return nullptr;
    }
}

bool convolve_supports(int g) { return convolve_for(g) != nullptr; }

ErrorStatus convolve_table(int g, double2 *tw, cudaStream_t s)
{
    k_fft_table<<<(g + 127) / 128, 128, 0, s>>>(g, tw);
    GS_CUDA(cudaGetLastError());
    return ok();
}

ErrorStatus convolve_mesh(double *mesh, int g, const MeshScale &scale, const double *table,
                          const double2 *tw, cudaStream_t s)
{
    const Convolve run = convolve_for(g);
    if (!run) return GS_RAISE(GRAV_VALUE_ERROR, "no convolution of a mesh of %d cells a side", g);
    run(reinterpret_cast<double2 *>(mesh), scale, table, tw, s);
    GS_CUDA(cudaGetLastError());
    return ok();
}

}  // namespace gs
