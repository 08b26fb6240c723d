// Cell expansions of the planetesimals' pull on the tracers (no counterpart in the
// reference), for the mixed step with many planetesimals.
//
// Every tracer feels every planetesimal, but the far ones vary little over a small region.
// So space is cut into a tree of cubic cells, and per RK4 stage every cell that holds
// tracers gets the harmonic expansion, about its centre, of the potential of the
// planetesimals that are far from it; a tracer evaluates its cell's expansion (about 400
// FP32 operations) and takes one by one only the planetesimals that are not far.  On a
// belt of 4,096 planetesimals that is some 300 pairs a stage instead of 4,096 (with a million
// tracers 2.2 ms a step against 7.9 ms with every pair).
//
// Far: a group of 16 planetesimals (consecutive in Hilbert order) whose box is at least
// kFarEdge cell edges from the cell's centre.  The expansion stops at degree kCellP = 10: a
// source at that distance and a tracer at a corner of the 10 % larger cell that it may use
// lose at most 2.6e-6 of that source's pull, most pairs far less, against the 5.6e-7 that
// rsqrt.approx and FP32 rounding leave in every single pull.  Summed pulls are off by
// 1e-8 to 1e-7 in the median, as with every pair.
//
// The tree: nested grids of power-of-two cell edges about the star (CellGrid).  A cell is
// split while more than CellGrid::leaf groups are not far from it and finer cells exist.
// Splitting depends on the planetesimals alone, and a tracer finds its cell from its own
// state, so a tracer's result does not depend on the other tracers: they only decide which
// cells are built.  A child's expansion is its parent's, translated, plus that of the groups
// that are far from the child and were not far from the parent; it tests only those.
//
// Tracers beyond kDistant times the planetesimals' extent (blown-out grains) need no cell: one
// expansion about the origin serves them.
//
// The stages' planetesimals and tracers differ, so every stage has its own tree; a tracer's
// cells are marked where it is expected to be (cell_predict) at the start, middle and end
// of the step.
//
// Harmonics: with (x + iy)^m times a real polynomial in z and r^2, recursions of three FP32
// operations per (n, m):  Q_m = 1, Q_n = z Q_{n-1} - g r^2 Q_{n-2},
// g = ((n-1)^2 - m^2) / ((2n-1)(2n-3)) for the regular ones, and the same with z/r^2 and
// 1/r^2 for the irregular ones (the solid harmonics of W. Dehnen, Comput. Astrophys. Cosmol.
// 1:1 (2014), divided by their leading factors, which go into the coefficients).
#include <algorithm>
#include <climits>
#include <cmath>
#include <complex>
#include <cstring>
#include <memory>
#include <new>
#include "ddx_launch.cuh"
#include "ddx_cells.cuh"
#include "ddx_shift.cuh"
#include "ddx_pull.cuh"
#include "ddx_scan.cuh"

namespace ddx {

struct CellScratch {
    char* arena = nullptr;
    CellScratch* outgrown = nullptr;
    CellView v{};
    uint32_t *count = nullptr, *start = nullptr, *temp = nullptr;   // the tracers' counting sort
    unsigned long long* sums = nullptr;                             // of cells_setup_kernel
    int cap_src = 0, cap_dust = 0;
};

namespace {

constexpr float kFarEdge = 4.5f;
// A cell is split while more groups than this are near it, and the finest cell edge is about
// this share of the planetesimals' mean distance for 4,096 of them (edge_scale for other
// numbers), for a narrow belt and for a set spread over more than half an octave of distance.
// A spread set's tracers share fewer cells, so a cell has to cost less (us a step, start = all
// planetesimals one by one, 24 and 1/30 / 40 and 1/24 / 64 and 1/20):
//   belt of 4,096 with a million tracers              7930 / 2170 / 2560 / 3220
//   belt and halo of 3,001 with 30,000                 677 /  751 /  638 /  658
//   belt and halo of 9,000 with 30,000                1778 / 2002 / 1805 / 1497
constexpr int kLeafNarrow = 24, kLeafSpread = 40, kLeafSpreadMany = 64;      // Many: from 8,192 planetesimals
constexpr float kEdgeNarrow = 1.f / 30.f, kEdgeSpread = 1.f / 24.f;
constexpr float kSpreadOctaves = 0.35f;                   // standard deviation of log2 of the distance

// Cells are for flat sets (disks at any tilt) spread over a few octaves of distance.  Tracers lie where the
// planetesimals do, more or less, and in a set that fills much space few share a cell, whose expansion costs as much as
// some thousand pulls: every planetesimal one by one is then faster below several 100,000 tracers.  The
// choice is the planetesimals' alone, as a tracer's result is not to hang on how many others there are.
// Two limits: kFlat* on the smallest eigenvalue of the mean of r r^T over the planetesimals' directions r from
// the star (4.6e-4 for inclinations up to 3 degrees, 5.1e-3 up to 10, 1/3 for a ball), and kRoom* on its root times the
// standard deviation of log2 |r|, the set's room.  us a step with every pair / with cells, 16,000 - 33,000 - 500,000
// tracers spread like 4,093 planetesimals (a shell: 2,000 - 30,000 - 500,000):
//   narrow: ring of 120 to 140 AU, up to 3 degrees (room 0.0014)   721 / 520     756 / 571     3977 / 1185
//           the same, up to 15 (0.0068)                            829 / 779     885 / 937     4005 / 1751
//           the same, up to 20 (0.0092, over the limit)            716 / 791     740 / 947     4007 / 1733
//           ring of 100 to 160 AU, up to 5 (0.0069)                803 / 705     839 / 836     4031 / 1612
//   spread: disk of 20 to 200 AU, up to 6 (0.036)                  716 / 624     746 / 711     3941 / 1651
//           the same, up to 10 (0.060)                             751 / 714     778 / 814     3967 / 1811
//           the same, up to 15 (0.089, over)                       730 / 844     786 / 969     3999 / 2044
//           disk over two decades, up to 3 (1.9 octaves, over)     845 / 997     891 / 1109    4547 / 2651
//   shell (over)                                                   549 / 627     778 / 2123    4000 / 4984
// Without cells the kernels that build them leave at once: 0.93 to 1.1 times the speed of a step that never had them.
constexpr float kFlatNarrow = 1.25e-2f, kFlatSpread = 6e-3f, kRoomNarrow = 7e-3f, kRoomSpread = 6.2e-2f;
constexpr double kMostOctaves = 1.25;                     // as kSpreadOctaves: 0.96 for one decade, 1.92 for two

__host__ __device__ constexpr int coef_at(int n, int m) { return n * (n + 1) / 2 - 1 + m; }
// A lane's sums of the irregular harmonics, in f2: order 0 in pairs of degrees (2, 3), (4, 5), ..;
// the other orders in columns of two, m = 2 p + 1 and m + 1, entry j holding (m + j, m) and
// (m + 1 + j, m + 1), first the real parts, then the imaginary ones.  The recursion over j then
// runs on both orders in one f32x2 operation (a belt of 4,096 with a million tracers: 188 us for
// cells_far_kernel, 203 us with scalar recursions).  Degree 1 has Kahan sums apart.
static_assert(kCellP % 2 == 0, "the orders 1..kCellP go in pairs");
constexpr int kZonal = kCellP / 2;                                                    // f2 of order 0
__host__ __device__ constexpr int column_len(int p) { return kCellP - 2 * p; }        // degrees of orders 2p + 1, 2p + 2
__host__ __device__ constexpr int column_first(int p) { return kZonal + 2 * p * (kCellP + 1 - p); }
constexpr int kAcc = column_first(kCellP / 2);
__host__ __device__ constexpr float harm_g(int n, int m) {
    return (float)((double)((n - 1) * (n - 1) - m * m) / (double)((2 * n - 1) * (2 * n - 3)));
}

// harm_g of a column's two orders: entry j of column p is for (2p + 1 + j, 2p + 1) and (2p + 2 + j, 2p + 2).
struct ColumnG {
    float2 g[kCellP / 2][kCellP];
    constexpr ColumnG() : g{} {
        for (int p = 0; p < kCellP / 2; ++p)
            for (int j = 2; j < column_len(p); ++j)
                g[p][j] = float2{-harm_g(2 * p + 1 + j, 2 * p + 1), -harm_g(2 * p + 2 + j, 2 * p + 2)};
    }
};
__constant__ ColumnG kColumnG{};

// Cells per axis for n_src planetesimals: the finest level has to reach past them.
int grid_dim(int n_src) { return n_src <= 8192 ? 128 : 256; }
int grid_levels(int G) { return G == 128 ? 6 : 7; }     // down to kCellTop cells per axis at the top

// ---- host tables -------------------------------------------------------------------------

typedef std::complex<double> cd;

double regular_k(int n, int m) {      // leading factor of the regular harmonic (n, m)
    double f = 1.0;
    for (int j = 1; j <= m; ++j) f /= 2.0 * j;
    for (int j = m + 1; j <= n; ++j) f *= (2.0 * j - 1.0) / ((double)j * j - (double)m * m);
    return f;
}

// The regular harmonic (n, m), |m| <= n, at (x, y, z).
cd regular(int n, int m, double x, double y, double z) {
    const int a = m < 0 ? -m : m;
    if (n < 0 || a > n) return 0.0;
    const double r2 = x * x + y * y + z * z;
    double q2 = 0.0, q1 = 1.0;
    for (int j = a + 1; j <= n; ++j) {
        const double g = ((j - 1.0) * (j - 1.0) - (double)a * a) / ((2.0 * j - 1.0) * (2.0 * j - 3.0));
        const double q = z * q1 - (j > a + 1 ? g * r2 * q2 : 0.0);
        q2 = q1;
        q1 = q;
    }
    const cd v = std::pow(cd(x, y), a) * q1 * regular_k(n, a);
    return m < 0 ? (a % 2 ? -std::conj(v) : std::conj(v)) : v;
}

bool make_tables(CellTables& t) {
    std::memset(&t, 0, sizeof(t));
    constexpr int N = 2 * kCellCoef;
    const std::unique_ptr<double[]> M(new (std::nothrow) double[(size_t)N * N]());   // [i][j]: parent coefficient i into child coefficient j
    if (!M) return false;
    for (int n = 1; n <= kCellP; ++n)
        for (int m = 0; m <= n; ++m) {
            double df = 1.0;
            for (int j = 1; j < 2 * n; j += 2) df *= j;
            const int i = 2 * coef_at(n, m);
            t.w[i] = t.w[i + 1] = (float)((m == 0 ? 1.0 : 2.0) * df * regular_k(n, m));
            t.neg[i] = (unsigned char)((m % 2 ? 1 : 0) | ((n + m) % 2 ? 4 : 0));
            t.neg[i + 1] = (unsigned char)((m % 2 ? 0 : 1) | 2 | ((n + m) % 2 ? 4 : 0));
            for (int k = 1; k <= n; ++k)
                for (int l = 0; l <= k; ++l) {
                    const cd c1 = regular(n - k, m - l, 0.25, 0.25, 0.25);
                    const cd c2 = l > 0 ? (l % 2 ? -1.0 : 1.0) * regular(n - k, m + l, 0.25, 0.25, 0.25) : 0.0;
                    // the potential in units of the cell's edge halves with the edge
                    const double f = 0.5 * std::pow(0.5, k) * regular_k(k, l) / regular_k(n, m);
                    const int j = 2 * coef_at(k, l);
                    M[(size_t)i * N + j] += f * (c1.real() + c2.real());
                    if (l > 0) M[(size_t)i * N + j + 1] += f * (-c1.imag() + c2.imag());
                    if (m > 0) {
                        M[(size_t)(i + 1) * N + j] += f * (c1.imag() + c2.imag());
                        if (l > 0) M[(size_t)(i + 1) * N + j + 1] += f * (c1.real() - c2.real());
                    }
                }
        }
    int e = 0;
    for (int j = 0; j < N; ++j) {
        t.sh_first[j] = (unsigned short)e;
        for (int i = 0; i < N; ++i) {
            const double v = M[(size_t)i * N + j];
            if (std::fabs(v) < 1e-14) continue;      // zero by symmetry
            if (i == j && low_of(i) >= 0) continue;  // degree 1 itself (1/4): cells_shift_kernel, in two floats
            if (e == kCellShift) return false;
            t.sh_val[e] = (float)v;
            t.sh_idx[e] = (unsigned char)i;
            ++e;
        }
    }
    t.sh_first[N] = (unsigned short)e;
    int k4 = 0;
    for (int mu = 0; mu < kCellP; ++mu)
        for (int k = mu; k < kCellP; ++k, ++k4) {
            const double kk = regular_k(k, mu);
            t.ap[k4] = mu + 1 <= k + 1 ? (float)(kk / (2.0 * regular_k(k + 1, mu + 1))) : 0.f;
            t.am[k4] = mu >= 1 ? (float)(kk / ((mu == 1 ? 1.0 : 2.0) * regular_k(k + 1, mu - 1))) : 0.f;
            t.az[k4] = (float)(kk / regular_k(k + 1, mu));
        }
    k4 = 0;
    for (int mu = 0; mu <= kCellP + 1; ++mu)
        for (int k = mu > 0 ? mu : 1; k <= kCellP + 1; ++k, ++k4) {
            double df = 1.0;
            for (int j = 1; j < 2 * k; j += 2) df *= j;
            t.fp[k4] = mu + 1 <= k - 1 ? (float)(df * regular_k(k - 1, mu + 1)) : 0.f;
            t.fm[k4] = mu >= 1 && mu - 1 <= k - 1 ? (float)(df * regular_k(k - 1, mu - 1)) : 0.f;
            t.fz[k4] = mu <= k - 1 ? (float)(-(mu == 0 ? 1.0 : 2.0) * df * regular_k(k - 1, mu)) : 0.f;
        }
    return true;
}

// ---- grid and tracers --------------------------------------------------------------------

constexpr int kSetupThreads = 256;

// The finest edge's share of the mean distance over that for 4,096 planetesimals: it goes as n^(-1/4),
// but as n^(-1/8) from 4,096 to 32,768 (us a step with -1/4 / -1/8: belts of 9,000 with 300,000 tracers 2166 /
// 1869, 30,000 with 20,000 5084 / 4564, halos of 20,000 with 30,000 and 500,000 3871 / 3517 and 8624 / 8130; beyond,
// a halo of 40,000 with 300,000 16182 / 17004, a belt of 65,536 with two million 48100 / 73000).
__device__ __forceinline__ float edge_scale(float n) {
    const float q = sqrtf(rsqrtf(fmaxf(n, 1.f) / 4096.f));
    return n > 4096.f && n <= 32768.f ? sqrtf(q) : q;
}

// The grids of this step from the geometric mean distance of the planetesimals to the star
// (largest coordinate difference) and its spread, without the few beyond the last octave of their order.
// Integer sums: the same on every run.  sums: [0] sum of the logarithms, [1] their number, [2] blocks
// done, [3] sum of the logarithms of |z|, [4] of the logarithms' squares, [5..9] of 2^20 times xx, xy, xz, yy, yz of
// the directions, [10] and [11] as [0] and [4] of the distances themselves (all zero before); the last block to
// finish writes the grid.
constexpr int kSetupSums = 12;
__global__ void __launch_bounds__(kSetupThreads)
cells_setup_kernel(const Body* __restrict__ P, int n_exact, int n_src, int G, const int* __restrict__ last_octave,
                   unsigned long long* __restrict__ sums, CellGrid* __restrict__ grid) {
    after_previous();
    __shared__ bool last;
    const Body s = P[0];
    const int k = blockIdx.x * kSetupThreads + threadIdx.x;
    long long sum = 0, sumz = 0, sum2 = 0, sumr = 0, sumr2 = 0;
    int n = 0, dir[5] = {0, 0, 0, 0, 0};
    if (k < n_src) {
        const Body b = P[n_exact + k];
        const float x = (float)(b.x - s.x), y = (float)(b.y - s.y), z = (float)(b.z - s.z);
        const float m = fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z)));
        if (m > 1e-30f && m < 1e30f && (int)(__float_as_uint(m) >> 23) <= *last_octave) {
            const float l = log2f(m);
            sum = (long long)(l * 65536.f);
            sum2 = (long long)(l * l * 65536.f);
            sumz = (long long)(log2f(fmaxf(fabsf(z), 1e-30f)) * 65536.f);
            n = 1;
            const float i = 1.f / m, ux = x * i, uy = y * i, uz = z * i;
            const float u2 = ux * ux + uy * uy + uz * uz, f = 1048576.f / u2, lr = l + 0.5f * log2f(u2);
            sumr = (long long)(lr * 65536.f);
            sumr2 = (long long)(lr * lr * 65536.f);
            dir[0] = __float2int_rn(f * ux * ux); dir[1] = __float2int_rn(f * ux * uy); dir[2] = __float2int_rn(f * ux * uz);
            dir[3] = __float2int_rn(f * uy * uy); dir[4] = __float2int_rn(f * uy * uz);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        sumz += __shfl_xor_sync(0xffffffffu, sumz, o);
        sum2 += __shfl_xor_sync(0xffffffffu, sum2, o);
        sumr += __shfl_xor_sync(0xffffffffu, sumr, o);
        sumr2 += __shfl_xor_sync(0xffffffffu, sumr2, o);
        n += __shfl_xor_sync(0xffffffffu, n, o);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) dir[q] = __reduce_add_sync(0xffffffffu, dir[q]);
    // a block's sums, then one atomic each
    __shared__ long long part[kSetupThreads / 32][kSetupSums];
    if ((threadIdx.x & 31) == 0) {
        long long* const p = part[threadIdx.x >> 5];
        p[0] = sum; p[1] = n; p[2] = 0; p[3] = sumz; p[4] = sum2;
#pragma unroll
        for (int q = 0; q < 5; ++q) p[5 + q] = dir[q];
        p[10] = sumr; p[11] = sumr2;
    }
    __syncthreads();
    if (threadIdx.x < kSetupSums && threadIdx.x != 2) {
        long long t = 0;
        for (int w = 0; w < kSetupThreads / 32; ++w) t += part[w][threadIdx.x];
        atomicAdd(&sums[threadIdx.x], (unsigned long long)t);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&sums[2], 1ull) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    sum = (long long)*(volatile unsigned long long*)&sums[0];
    const long long num = (long long)*(volatile unsigned long long*)&sums[1];
    sumz = (long long)*(volatile unsigned long long*)&sums[3];
    sum2 = (long long)*(volatile unsigned long long*)&sums[4];
    CellGrid g{};
    const float mean = num > 0 ? exp2f((float)(sum / num) * (1.f / 65536.f)) : 1.f;
    const double lm = num > 0 ? (double)sum / (double)num / 65536.0 : 0.0;
    const double var = num > 0 ? (double)sum2 / (double)num / 65536.0 - lm * lm : 0.0;
    const bool spread = var > (double)kSpreadOctaves * kSpreadOctaves;
    g.leaf = spread ? (num < 8192 ? kLeafSpread : kLeafSpreadMany) : kLeafNarrow;
    const float want = mean * (spread ? kEdgeSpread : kEdgeNarrow) * edge_scale((float)num);
    // the nearest of 2^e and 3 2^(e-1): a centre, an odd multiple of half an edge, is exact
    const float l = log2f(want);
    int e = (int)floorf(l);
    e = e < -60 ? -60 : (e > 60 ? 60 : e);
    const float f = l - (float)e;
    const float lead = f < 0.2925f ? 1.f : (f < 0.7925f ? 1.5f : 2.f);
    g.s0 = ldexpf(lead, e);
    g.inv_s0 = 1.f / g.s0;
    g.sx = (float)s.x; g.sy = (float)s.y; g.sz = (float)s.z; g.m0 = (float)s.m;
    const float qx = rintf(g.sx / g.s0), qy = rintf(g.sy / g.s0), qz = rintf(g.sz / g.s0);
    g.ox = qx * g.s0; g.oy = qy * g.s0; g.oz = qz * g.s0;
    // flat: the mean of r r^T less the limit times the identity is not positive definite (Sylvester's minors)
    float d[5];
    const float per = 1.f / (1048576.f * (float)num);
    for (int q = 0; q < 5; ++q) d[q] = (float)(long long)*(volatile unsigned long long*)&sums[5 + q] * per;
    const double lr = num > 0 ? (double)(long long)*(volatile unsigned long long*)&sums[10] / (double)num / 65536.0 : 0.0;
    const double varr = num > 0 ? (double)(long long)*(volatile unsigned long long*)&sums[11] / (double)num / 65536.0 - lr * lr : 0.0;
    const float room = spread ? kRoomSpread : kRoomNarrow;
    const float most = fminf(spread ? kFlatSpread : kFlatNarrow, room * room / fmaxf((float)varr, 1e-12f));
    const float axx = d[0] - most, ayy = d[3] - most, azz = 1.f - d[0] - d[3] - most, m2 = axx * ayy - d[1] * d[1];
    const float m3 = azz * m2 - axx * d[4] * d[4] - ayy * d[2] * d[2] + 2.f * d[1] * d[2] * d[4];
    const bool flat = !(axx > 0.f && m2 > 0.f && m3 > 0.f);
    // centres are exact while the origin is at most 2^20 cells away
    g.ok = num > 0 && flat && var <= kMostOctaves * kMostOctaves && fabsf(qx) < 1048576.f && fabsf(qy) < 1048576.f && fabsf(qz) < 1048576.f;
    g.thin = g.ok && exp2f((float)(sumz / num) * (1.f / 65536.f)) < 0.07f * mean;
    *grid = g;
}

// Hilbert index of a cell of a D-dimensional grid with B bits per axis (Skilling's
// transform, AIP Conf. Proc. 707, 2004).
template <int D, int B>
__device__ __forceinline__ uint32_t hilbert(uint32_t (&X)[D]) {
    constexpr uint32_t M = 1u << (B - 1);
#pragma unroll
    for (uint32_t Q = M; Q > 1; Q >>= 1) {
        const uint32_t P = Q - 1;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            if (X[i] & Q) {
                X[0] ^= P;
            } else {
                const uint32_t t = (X[0] ^ X[i]) & P;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
#pragma unroll
    for (int i = 1; i < D; ++i) X[i] ^= X[i - 1];
    uint32_t t = 0;
#pragma unroll
    for (uint32_t Q = M; Q > 1; Q >>= 1)
        if (X[D - 1] & Q) t ^= Q - 1;
#pragma unroll
    for (int i = 0; i < D; ++i) X[i] ^= t;
    uint32_t key = 0;
#pragma unroll
    for (int b = B - 1; b >= 0; --b)
#pragma unroll
        for (int i = 0; i < D; ++i) key = key << 1 | ((X[i] >> b) & 1u);
    return key;
}

// Place of a position (relative to the origin) in the tracers' visiting order, 21 bits: the
// Hilbert order of 128^3 cells of edge s0 (G = 128; 2 s0 at 256), or, in a thin disk, of
// 256 x 256 x 32 cells of half that edge (32^3 blocks in Hilbert order, the 8 x 8 cells of a
// block in the plane's), clamped at their border.  inside: its cell is not at the border, so it
// holds no clamped position.
__device__ __forceinline__ uint32_t order_code(const CellGrid& g, int G, const CellPos& p, bool& inside) {
    const float sc = g.inv_s0 * (128.f / (float)G);
    if (g.thin) {
        const float ux = floorf(p.x * sc * 2.f) + 128.f, uy = floorf(p.y * sc * 2.f) + 128.f;
        const float uz = floorf(p.z * sc * 2.f) + 16.f;
        inside = ux >= 1.f && ux < 255.f && uy >= 1.f && uy < 255.f && uz >= 1.f && uz < 31.f;
        const uint32_t x = (uint32_t)(int)fminf(fmaxf(ux, 0.f), 255.f);   // NaN gives 0
        const uint32_t y = (uint32_t)(int)fminf(fmaxf(uy, 0.f), 255.f);
        const uint32_t z = (uint32_t)(int)fminf(fmaxf(uz, 0.f), 31.f);
        uint32_t hi[3] = {x >> 3, y >> 3, z}, lo[2] = {x & 7u, y & 7u};
        return hilbert<3, 5>(hi) << 6 | hilbert<2, 3>(lo);
    }
    const float ux = floorf(p.x * sc) + 64.f, uy = floorf(p.y * sc) + 64.f, uz = floorf(p.z * sc) + 64.f;
    inside = ux >= 1.f && ux < 127.f && uy >= 1.f && uy < 127.f && uz >= 1.f && uz < 127.f;
    uint32_t c[3] = {(uint32_t)(int)fminf(fmaxf(ux, 0.f), 127.f), (uint32_t)(int)fminf(fmaxf(uy, 0.f), 127.f),
                     (uint32_t)(int)fminf(fmaxf(uz, 0.f), 127.f)};
    return hilbert<3, 7>(c);
}

__device__ __forceinline__ void mark_cell(const CellView& v, int set, const CellAt& at) {
    const int d = cell_dim(v.G, at.level);
    uint32_t* w = v.own + (size_t)set * v.mark_words + cell_word0(v.G, at.level) + (at.iz * d + at.iy) * (d / 32) + (at.ix >> 5);
    const uint32_t bit = 1u << (at.ix & 31);
    if (!(*(volatile uint32_t*)w & bit)) atomicOr(w, bit);
}

// No position in p's finest cell is distant (a hundredth of slack for the roundings).
__device__ __forceinline__ bool cell_within_distant(const CellGrid& g, const CellPos& p) {
    const float ax = fabsf(p.x) + g.s0, ay = fabsf(p.y) + g.s0, az = fabsf(p.z) + g.s0;
    return ax * ax + ay * ay + az * az < 0.99f * kDistant * kDistant * __uint_as_float(g.b2);
}

// Per tracer: its place in the visiting order (by its expected position in the middle of the
// step; removed tracers last) with an atomic rank in it, and the marks of the cells where
// it is expected to be during the step.  The marks are what this kernel waits for
// (scattered words that every SM reads), so the middle's cell is marked by the first of its
// tracers alone where all tracers of a cell of the order would mark the same one: the order's cells
// are no larger than the tree's finest, the cell holds no clamped position and no distant one.
__global__ void cells_keys_kernel(ddx_state s, StepArgs a, const SizeBin* __restrict__ bins, CellView v,
                                  uint32_t* __restrict__ key, uint32_t* __restrict__ rank,
                                  uint32_t* __restrict__ count) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_dust) return;
    const int t = a.n_grav + i;
    const CellGrid g = *v.grid;
    uint32_t bin = kCellBins, first = 0;
    if (s.N[t] != 0.0) {
        const double x = s.x[t], y = s.y[t], z = s.z[t];
        const double vx = s.vx[t], vy = s.vy[t], vz = s.vz[t];
        const int id = s.id[t];
        const float red = star_reduction(bins, id, a.n_grid);
        const CellPos p1 = cell_predict(g, x, y, z, vx, vy, vz, red, (float)a.dt, 1);
        bool inside;
        bin = order_code(g, v.G, p1, inside);
        first = atomicAdd(&count[bin], 1u);
        if (g.ok) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k == 2) continue;            // the middle stages share their marks
                const CellPos p = k == 1 ? p1 : cell_predict(g, x, y, z, vx, vy, vz, red, (float)a.dt, k);
                if (cell_distant(g, p.x, p.y, p.z)) continue;
                const CellAt at = cell_at(g, v.G, v.levels, p);
                if (at.level < 0) continue;
                if (k == 1 && first != 0 && inside && (v.G == 128 || g.thin) && cell_within_distant(g, p)) continue;
                mark_cell(v, mark_set(k), at);
            }
        }
    } else {
        first = atomicAdd(&count[bin], 1u);
    }
    key[i] = bin;
    rank[i] = first;
}

__global__ void cells_scatter_kernel(int n, const uint32_t* __restrict__ key, const uint32_t* __restrict__ rank,
                                     const uint32_t* __restrict__ start, int* __restrict__ perm) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) perm[start[key[k]] + rank[k]] = k;
}

// Marks every marked cell and its ancestors: a block takes 32^3 cells of one level (of set
// blockIdx.y), halves
// them level by level in shared memory, and follows the last cell up to the top.
__global__ void __launch_bounds__(1024)
cells_ancestors_kernel(CellView v) {
    after_previous();
    __shared__ uint32_t row[2][1024];
    // which level and which chunk of it
    int b = blockIdx.x, level = 0;
    for (;; ++level) {
        const int c = cell_dim(v.G, level) / 32;
        if (b < c * c * c) break;
        b -= c * c * c;
    }
    const int d = cell_dim(v.G, level), nc = d / 32;
    const int bx = b % nc, by = b / nc % nc, bz = b / nc / nc;
    const int t = threadIdx.x;
    int y = t & 31, z = t >> 5;
    const size_t at = cell_word0(v.G, level) + (size_t)((bz * 32 + z) * d + by * 32 + y) * nc + bx;
    uint32_t* const mark = v.mark + (size_t)blockIdx.y * v.mark_words;
    uint32_t w = v.own[(size_t)blockIdx.y * v.mark_words + at];
    if (!__syncthreads_or(w != 0u)) return;
    if (w) atomicOr(mark + at, w);
    row[0][t] = w;
    __syncthreads();
    // origin of the chunk relative to the centre, halved with every level
    int ox = bx * 32 - d / 2, oy = by * 32 - d / 2, oz = bz * 32 - d / 2;
    int n = 32, cur = 0;
    for (int l = level + 1; l < v.levels; ++l) {
        ox >>= 1; oy >>= 1; oz >>= 1;
        const int h = n > 1 ? n / 2 : 1;
        const int dl = cell_dim(v.G, l);
        uint32_t up = 0;
        if (t < h * h) {
            y = t % h; z = t / h;
            if (n > 1) {
                const uint32_t* r = row[cur];
                uint32_t o = r[2 * z * n + 2 * y] | r[2 * z * n + 2 * y + 1] | r[(2 * z + 1) * n + 2 * y] |
                             r[(2 * z + 1) * n + 2 * y + 1];
                o |= o >> 1;                          // pairs of cells along x: their bits at 0, 2, 4, ...
                for (int k = 0; k < h; ++k) up |= ((o >> (2 * k)) & 1u) << k;
            } else {
                up = row[cur][0];
            }
            if (up) {
                const int x0 = ox + dl / 2;           // h cells from x0, which is a multiple of h
                atomicOr(mark + cell_word0(v.G, l) + ((oz + dl / 2 + z) * dl + oy + dl / 2 + y) * (dl / 32) + (x0 >> 5),
                         up << (x0 & 31));
            }
            row[cur ^ 1][z * h + y] = up;
        }
        __syncthreads();
        cur ^= 1;
        n = h;
    }
}

// Per stage: the sources in slot order as (high parts, mass) and (low parts), and the boxes of
// the source groups (a lane per source, high parts) and of the spans, two groups each, for the span
// kernel (store_span_box).  A warp takes a span.
static_assert(2 * kGroupSrc == 2 * kPairSpan && 2 * kGroupSrc == 32, "a span is two groups and a warp");
__global__ void cells_boxes_kernel(BodyPair* __restrict__ PP, int pcap, CellView v) {
    after_previous();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, spans = (v.n_groups + 1) / 2;   // stage * spans + span
    const int u = threadIdx.x % kGroupSrc;
    const unsigned part = ((1u << kGroupSrc) - 1u) << (threadIdx.x & 31 & ~(kGroupSrc - 1));
    if (w >= 4 * spans) return;                                             // a span's lanes leave together
    const int stage = w / spans, span = w - stage * spans, grp = 2 * span + ((threadIdx.x & 31) >= kGroupSrc);
    const bool real = grp < v.n_groups;
    const int k = stage * v.n_groups + grp;
    const int q = grp * kGroupSrc + u;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool bad = false, nan = false;
    if (q < v.n_src) {
        const BodyPair& r = PP[(size_t)stage * pcap + (q >> 1)];
        const float p[3] = {r.hx[q & 1], r.hy[q & 1], r.hz[q & 1]};
        float4* const S = v.src + 2 * ((size_t)stage * v.n_groups * kGroupSrc + q);
        S[0] = make_float4(p[0], p[1], p[2], r.m[q & 1]);
        S[1] = make_float4(r.lx[q & 1], r.ly[q & 1], r.lz[q & 1], 0.f);
        for (int a = 0; a < 3; ++a) {
            bad = bad || !(fabsf(p[a]) < 1e18f);
            nan = nan || !(p[a] == p[a]);
            lo[a] = hi[a] = p[a];
        }
        bad = bad || !(fabsf(r.m[q & 1]) < 1e30f);
        if ((u & 1) == 0) {
            ulonglong2* const N = v.near_rec + (size_t)k * 4 * kGroupPairs + (u >> 1);
            N[0] = *reinterpret_cast<const ulonglong2*>(r.hx);
            N[kGroupPairs] = *reinterpret_cast<const ulonglong2*>(r.hz);
            N[2 * kGroupPairs] = *reinterpret_cast<const ulonglong2*>(r.lx);
            N[3 * kGroupPairs].x = *reinterpret_cast<const unsigned long long*>(r.lz);
        }
    } else if (real && (u & 1) == 0) {            // an empty record: no mass, far from every tracer
        const f2 away = f2_dup(kFarAway);
        ulonglong2* const N = v.near_rec + (size_t)k * 4 * kGroupPairs + (u >> 1);
        N[0] = make_ulonglong2(away, away);
        N[kGroupPairs] = make_ulonglong2(away, 0);
        N[2 * kGroupPairs] = make_ulonglong2(0, 0);
        N[3 * kGroupPairs].x = 0;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int o = kGroupSrc / 2; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(part, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(part, hi[a], o));
        }
    bad = (__ballot_sync(part, bad) & part) != 0u;
    nan = __any_sync(0xffffffffu, nan);
    float slo[3], shi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        slo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], kGroupSrc));
        shi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], kGroupSrc));
    }
    store_span_box(PP + (size_t)stage * pcap + (size_t)span * kPairSpan, slo, shi, nan);
    if (real && u == 0) {   // the box's farthest corner bounds its sources' distances
        const CellGrid& g = *v.grid;
        const float dx = fmaxf(hi[0] - g.ox, g.ox - lo[0]), dy = fmaxf(hi[1] - g.oy, g.oy - lo[1]);
        const float dz = fmaxf(hi[2] - g.oz, g.oz - lo[2]);
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), core = core_edges(v.G) * g.s0;
        if (!bad && r2 <= core * core) {
            atomicMax(&v.grid->b2, __float_as_uint(r2));
        } else {
            atomicOr(&v.outlier[stage * v.words + (grp >> 5)], 1u << (grp & 31));
            atomicAdd(&v.grid->outliers, 1u);
        }
        v.gbox[2 * (size_t)k] = make_float4(lo[0], lo[1], lo[2], bad ? 1.f : 0.f);
        v.gbox[2 * (size_t)k + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
}

// ---- nodes -------------------------------------------------------------------------------

__device__ __forceinline__ void set_node(const CellView& v, const CellGrid& g, int k, int level, int ix, int iy, int iz,
                                         int parent, int stage) {
    const int d = cell_dim(v.G, level);
    const float s = g.s0 * (float)(1 << level);
    CellNode& n = v.node[k];
    n.cx = g.ox + ((float)(ix - d / 2) + 0.5f) * s;
    n.cy = g.oy + ((float)(iy - d / 2) + 0.5f) * s;
    n.cz = g.oz + ((float)(iz - d / 2) + 0.5f) * s;
    n.inv_s = g.inv_s0 / (float)(1 << level);
    n.parent = parent;
    n.stage = stage;
    n.cell = ix | iy << 10 | iz << 20;
}

// The roots: four nodes (one per stage) for every marked cell of the top level, a thread per
// cell.
constexpr int kRootThreads = 256;
__global__ void __launch_bounds__(kRootThreads)
cells_roots_kernel(CellView v) {
    after_previous();
    const int top = v.levels - 1, c = blockIdx.x * kRootThreads + threadIdx.x;   // cell of the top grid
    const CellGrid& g = *v.grid;
    if (!g.ok) return;
    int first = -1;
    const uint32_t* const w = v.mark + cell_word0(v.G, top) + (c >> 5);
    if (((w[0] | w[v.mark_words] | w[2 * v.mark_words]) >> (c & 31) & 1u)) {
        first = (int)atomicAdd(&v.grid->cnt[top], 4u);
        if (first + 4 > v.cap) first = -1;
        else
            for (int st = 0; st < 4; ++st) set_node(v, g, first + st, top, c & 31, c >> 5 & 31, c >> 10, -1, st);
    }
    v.root[c] = first;
}

// f(Index<B>) .. f(Index<E - 1>): loops whose indices have to be constants, so that the
// accumulators stay in registers.
template <int V> struct Index { static constexpr int v = V; };
template <int B, int E, class F>
__device__ __forceinline__ void each(F&& f) {
    if constexpr (B < E) {
        f(Index<B>{});
        each<B + 1, E>(f);
    }
}

__device__ __forceinline__ void kahan_sum(float& S, float& C, float v) {
    const float y = __fsub_rn(v, C), t = __fadd_rn(S, y);
    C = __fsub_rn(__fsub_rn(t, S), y);
    S = t;
}

// acc += one source's irregular harmonics of degree 2 and more, (S, C) += those of degree 1: (dx, dy, dz) from the
// centre in units of the cell's edge.
__device__ __forceinline__ void p2l(float dx, float dy, float dz, float mass, f2 (&acc)[kAcc], float (&S)[3],
                                    float (&C)[3]) {
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float ri = rsqrt_newton(r2);
    const float v = ri * ri, zv = dz * v, ux = dx * v, uy = dy * v, t0 = mass * ri;
    kahan_sum(S[0], C[0], t0 * zv);
    kahan_sum(S[1], C[1], t0 * ux);
    kahan_sum(S[2], C[2], t0 * uy);
    // order 0, pairs of degrees
    float t2 = t0, t1 = zv * t0;
    each<0, kZonal>([&](auto kc) {
        constexpr int k = decltype(kc)::v, n = 2 + 2 * k;
        const float e = fmaf(v * t2, -harm_g(n, 0), zv * t1);
        float o = 0.f;
        if constexpr (n < kCellP) o = fmaf(v * t1, -harm_g(n + 1, 0), zv * e);
        acc[k] = add2(acc[k], f2_join(e, o));
        t2 = e;
        t1 = o;
    });
    // columns of two orders: entry j is degree m + j of order m times (EX, EY)
    const f2 V = f2_dup(v), ZV = f2_dup(zv), ZZ = mul2(ZV, ZV), VZ = mul2(V, ZV);
    const float e1x = t0 * ux, e1y = t0 * uy, wx = ux * ux - uy * uy, wy = 2.f * ux * uy;
    f2 EX = f2_join(e1x, e1x * ux - e1y * uy), EY = f2_join(e1y, e1x * uy + e1y * ux);
    const f2 WX = f2_dup(wx), WY = f2_dup(wy), NWY = f2_dup(-wy);
    each<0, kCellP / 2>([&](auto pc) {
        constexpr int p = decltype(pc)::v, k = column_first(p), len = column_len(p);
        if constexpr (p > 0) {
            const f2 F = fma2(EY, NWY, mul2(EX, WX));
            EY = fma2(EX, WY, mul2(EY, WX));
            EX = F;
        }
        acc[k] = add2(acc[k], EX);
        acc[k + len] = add2(acc[k + len], EY);
        f2 T2 = 0, T1 = ZV;
        each<1, len>([&](auto jc) {
            constexpr int j = decltype(jc)::v;
            f2 T = ZV;
            if constexpr (j > 1) {
                const f2 G = *reinterpret_cast<const f2*>(&kColumnG.g[p][j]);
                if constexpr (j == 2) T = fma2(V, G, ZZ);
                else if constexpr (j == 3) T = fma2(VZ, G, mul2(ZV, T1));
                else T = fma2(mul2(V, T2), G, mul2(ZV, T1));
            }
            acc[k + j] = fma2(T, EX, acc[k + j]);
            acc[k + len + j] = fma2(T, EY, acc[k + len + j]);
            T2 = T1;
            T1 = T;
        });
    });
}

constexpr int kNodeThreads = 128;
constexpr int kNodeWarps = kNodeThreads / 32;
constexpr int kReal = 2 * kCellCoef;             // real coefficients of a node

// First node of a level and their number; 0 nodes for a level that was dropped or that lies
// below one.
__device__ __forceinline__ int level_nodes(const CellView& v, int level, int& first) {
    const CellGrid& g = *v.grid;
    first = (int)g.first[level];
    const int count = (int)g.cnt[level];
    return level >= g.min_level ? count : 0;
}

// One level, a warp per node: which of the groups near the parent are near the node, whether
// it is split, and its children.
__global__ void __launch_bounds__(kNodeThreads)
cells_split_kernel(CellView v, int level, float near_eta) {
    after_previous();
    CellGrid& g = *v.grid;
    const int lane = threadIdx.x & 31;
    const bool top = level == v.levels - 1;       // the levels' nodes lie one after the other
    const int before = top ? 0 : (int)g.first[level + 1], above = top ? 0 : (int)g.cnt[level + 1];
    const int first = before + above, count = level >= g.min_level ? (int)g.cnt[level] : 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) g.first[level] = (uint32_t)first;
    if (count == 0) return;
    if (first + count > v.cap) {                  // no room for this level: its parents are the leaves
        if (blockIdx.x == 0 && threadIdx.x == 0) g.min_level = level + 1;
        return;
    }
    const int leaf = g.leaf;
    for (int b = blockIdx.x * kNodeWarps + (threadIdx.x >> 5); b < count; b += gridDim.x * kNodeWarps) {
        const int k = first + b;
        const CellNode nd = v.node[k];
        const float cx = nd.cx, cy = nd.cy, cz = nd.cz, edge = 1.f / nd.inv_s;
        // far also means beyond the near radius of every tracer that may use the cell
        const float own = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + edge;
        const float far = fmaxf(kFarEdge * edge, fmaf(near_eta, own, edge));
        const float far2 = far * far;
        const float4* const box = v.gbox + 2 * (size_t)(nd.stage & 3) * v.n_groups;
        const uint32_t* const up = nd.parent < 0 ? nullptr : v.near + (size_t)nd.parent * v.words;
        int n_near = 0;
        for (int w0 = 0; w0 < v.words; w0 += 32) {
            const int nw = min(32, v.words - w0);
            uint32_t cand = 0;                    // lane w: the parent's word w0 + w
            if (lane < nw) {
                const int left = v.n_groups - (w0 + lane) * 32;
                cand = up ? up[w0 + lane] : (left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u);
            }
            uint32_t mine = 0;
            for (uint32_t todo = __ballot_sync(0xffffffffu, cand != 0u); todo; todo &= todo - 1) {
                const int w = __ffs(todo) - 1;
                const uint32_t c = __shfl_sync(0xffffffffu, cand, w);
                bool is_near = false;
                if (c >> lane & 1u) {
                    const int gi = (w0 + w) * 32 + lane;
                    const float4 lo = box[2 * gi], hi = box[2 * gi + 1];
                    const float gx = fmaxf(0.f, fmaxf(lo.x - cx, cx - hi.x));
                    const float gy = fmaxf(0.f, fmaxf(lo.y - cy, cy - hi.y));
                    const float gz = fmaxf(0.f, fmaxf(lo.z - cz, cz - hi.z));
                    is_near = lo.w != 0.f || !(gx * gx + gy * gy + gz * gz >= far2);
                }
                const uint32_t nb = __ballot_sync(0xffffffffu, is_near);
                if (lane == w) mine = nb;
                const int at = n_near + __popc(nb & ((1u << lane) - 1u));
                if (is_near && at < kNearList && v.n_groups <= 65536) v.list[(size_t)k * kNearList + at] = (uint16_t)((w0 + w) * 32 + lane);
                n_near += __popc(nb);
            }
            if (lane < nw) v.near[(size_t)k * v.words + w0 + lane] = mine;
        }
        // children: the marked cells of the next finer grid, where it reaches
        int ch = -1;
        if (n_near > leaf && level > 0 && lane < 8) {
            const int d = cell_dim(v.G, level), dc = cell_dim(v.G, level - 1);
            const int ix = 2 * ((nd.cell & 1023) - d / 2) + (lane & 1) + dc / 2;
            const int iy = 2 * ((nd.cell >> 10 & 1023) - d / 2) + (lane >> 1 & 1) + dc / 2;
            const int iz = 2 * ((nd.cell >> 20 & 1023) - d / 2) + (lane >> 2) + dc / 2;
            const uint32_t* const mark = v.mark + (size_t)mark_set(nd.stage & 3) * v.mark_words;
            if (ix >= 0 && iy >= 0 && iz >= 0 && ix < dc && iy < dc && iz < dc &&
                (mark[cell_word0(v.G, level - 1) + (iz * dc + iy) * (dc / 32) + (ix >> 5)] >> (ix & 31) & 1u)) {
                ch = first + count + (int)atomicAdd(&g.cnt[level - 1], 1u);
                if (ch < v.cap) set_node(v, g, ch, level - 1, ix, iy, iz, k, (nd.stage & 3) | (lane ^ 7) << 2);
            }
        }
        if (lane < 8) v.node[k].child[lane] = ch;
        if (lane == 0) v.node[k].n_near = v.n_groups <= 65536 ? n_near : kNearList + 1;   // no list: the mask
    }
}

// The expansions of every node's newly far groups (near the parent, not near the node), all levels at
// once: a warp per node, handed out from the top level down as warps become free (with a block of four
// warps for every node above the finest two levels 4,096 planetesimals with 16,384 tracers took 657 us a
// step, 608 so, 3,001 with a halo and 500,003 1862 and 1769).  What bounds it
// is the FP32 pipe, about 60 % busy: about 200 instructions a source, most of them f32x2, and
// 900 per node (belt of 4,096 with a million tracers: 32,000 nodes, 12 million sources, 190 us).
constexpr int kFarList = 256;                    // far groups listed at once per node
constexpr int kRedParts = (kReal + 31) / 32, kRedRows = (kReal + kRedParts - 1) / kRedParts, kRedStride = 36;
struct FarShared {
    unsigned char list[kNodeWarps][kFarList];
    float red[kNodeWarps][kRedRows][kRedStride];
    float sum[kNodeWarps][kReal];
};

__device__ __forceinline__ void far_sums(const CellView& v, int k, FarShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto& list = sh.list[warp];
    auto& red = sh.red;
    auto& sum = sh.sum;
    const CellNode nd = v.node[k];
    const float cx = nd.cx, cy = nd.cy, cz = nd.cz, inv_s = nd.inv_s;
    const float4* const src = v.src + 2 * (size_t)(nd.stage & 3) * v.n_groups * kGroupSrc;
    const uint32_t* const up = nd.parent < 0 ? nullptr : v.near + (size_t)nd.parent * v.words;
    const uint32_t* const own = v.near + (size_t)k * v.words;
    f2 acc[kAcc];
#pragma unroll
    for (int q = 0; q < kAcc; ++q) acc[q] = 0;
    float S[3] = {0.f, 0.f, 0.f}, C[3] = {0.f, 0.f, 0.f};
    // the node's far groups are listed, 8 words of groups at a time
    for (int w = 0; w < v.words; w += kFarList / 32) {
        uint32_t far = 0;
        if (lane < kFarList / 32 && w + lane < v.words) {
            const int left = v.n_groups - (w + lane) * 32;
            far = (up ? up[w + lane] : (left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u)) & ~own[w + lane];
        }
        int n = 0;
        for (uint32_t todo = __ballot_sync(0xffffffffu, far != 0u); todo; todo &= todo - 1) {
            const int j = __ffs(todo) - 1;
            const uint32_t f = __shfl_sync(0xffffffffu, far, j);
            if (f >> lane & 1u) list[n + __popc(f & ((1u << lane) - 1u))] = (unsigned char)(j * 32 + lane);
            n += __popc(f);
        }
        __syncwarp();
        // 32 sources at a time, one per lane; the next ones are loaded ahead
        constexpr int kPerIt = 32 / kGroupSrc;    // groups
        int e = lane / kGroupSrc;
        const int u = lane & (kGroupSrc - 1);
        float4 h, l;
        int q = -1;
        auto fetch = [&]() {
            q = e < n ? (w * 32 + (int)list[e]) * kGroupSrc + u : v.n_src;
            if (q < v.n_src) {
                h = src[2 * q];
                l = src[2 * q + 1];
            }
            e += kPerIt;
        };
        fetch();
        for (int b = 0; b < n; b += kPerIt) {
            const bool use = q < v.n_src;
            const float dx = ((h.x - cx) + l.x) * inv_s, dy = ((h.y - cy) + l.y) * inv_s;
            const float dz = ((h.z - cz) + l.z) * inv_s, m = h.w;
            fetch();
            if (use) p2l(dx, dy, dz, m, acc, S, C);
        }
        __syncwarp();
    }
    // sums over the lanes through shared memory, a part of the coefficients at a time
    each<0, kRedParts>([&](auto pc) {
        constexpr int part = decltype(pc)::v;
        each<0, kCellP + 1>([&](auto mc) {
            constexpr int m = decltype(mc)::v;
            each<(m > 2 ? m : 2), kCellP + 1>([&](auto nc) {
                constexpr int n = decltype(nc)::v, i = 2 * coef_at(n, m);
                if constexpr (i / kRedRows == part || (i + 1) / kRedRows == part) {
                    constexpr int p = (m - 1) / 2, k = m == 0 ? (n - 2) / 2 : column_first(p) + n - m;
                    constexpr int odd = m == 0 ? n % 2 : (m - 1) % 2;
                    float re0, re1, im0 = 0.f, im1 = 0.f;
                    f2_split(acc[k], re0, re1);
                    if constexpr (m > 0) f2_split(acc[k + column_len(p)], im0, im1);
                    if constexpr (i / kRedRows == part) red[warp][i - part * kRedRows][lane] = odd ? re1 : re0;
                    if constexpr ((i + 1) / kRedRows == part) red[warp][i + 1 - part * kRedRows][lane] = odd ? im1 : im0;
                }
            });
        });
        if constexpr (part == 0) {                // degree 1 and, in the rows of its low parts, its corrections
            red[warp][0][lane] = S[0];
            red[warp][2][lane] = S[1];
            red[warp][3][lane] = S[2];
            red[warp][low_of(0)][lane] = C[0];
            red[warp][low_of(2)][lane] = C[1];
            red[warp][low_of(3)][lane] = C[2];
        }
        __syncwarp();
        float t = 0.f, c = 0.f;
        if (lane < kRedRows) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 f = *reinterpret_cast<const float4*>(&red[warp][lane][4 * j]);
                if constexpr (part == 0) {
                    kahan_sum(t, c, f.x); kahan_sum(t, c, f.y); kahan_sum(t, c, f.z); kahan_sum(t, c, f.w);
                } else {
                    t += (f.x + f.y) + (f.z + f.w);
                }
            }
        }
        if constexpr (part == 0) {                // low part of degree 1: less both corrections
            const float c0 = __shfl_sync(0xffffffffu, c, 0), c2 = __shfl_sync(0xffffffffu, c, 2);
            const float c3 = __shfl_sync(0xffffffffu, c, 3);
            if (is_low(lane)) t = -t - (lane == low_of(0) ? c0 : lane == low_of(2) ? c2 : c3);
        }
        if (lane < kRedRows && part * kRedRows + lane < kReal) sum[warp][part * kRedRows + lane] = t;
        __syncwarp();
    });
    for (int i = lane; i < kReal; i += 32) {
        const float t = sum[warp][i];
        v.lam[(size_t)k * kReal + i] = is_low(i) || low_of(i) >= 0 ? t : t * v.tab->w[i];   // degree 1: w = 1
    }
    __syncwarp();
}

// The expansion of all planetesimals about the origin, per stage, for distant
// tracers: their mass at their centre of mass in FP64, and what that leaves of their field from
// degree 2 on in FP32.  The blocks of a stage write partial sums; the last one adds them in
// block order and forms the force terms: with C the coefficients, X(k, u) = C(k-1, u+1) - C(k-1, u-1),
// Y = -i (C(k-1, u+1) + C(k-1, u-1)), Z = -(2 if u > 0) C(k-1, u) on the irregular harmonics.
__host__ __device__ constexpr int multi_at(int n, int m) { return n * (n + 1) / 2 + m; }

struct DistantShared {
    double mom[kNodeWarps][4], total[4];
    float red[kNodeWarps][2 * kMultiCoef], C[2 * kMultiCoef];
    bool last;
};
__device__ __forceinline__ void distant_sums(const CellView& v, int stage, int block, int blocks, DistantShared& sh) {
    auto& red = sh.red;
    auto& C = sh.C;
    auto& mom = sh.mom;
    auto& total = sh.total;
    auto& last = sh.last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const CellGrid& g = *v.grid;
    const float unit = g.inv_s0 * (1.f / kFarUnit);
    const float4* const src = v.src + 2 * (size_t)stage * v.n_groups * kGroupSrc;
    double M[4] = {0.0, 0.0, 0.0, 0.0};
    float re[kMultiCoef], im[kMultiCoef];
    each<0, kMultiCoef>([&](auto kc) { re[decltype(kc)::v] = im[decltype(kc)::v] = 0.f; });
    for (int q = block * kNodeThreads + threadIdx.x; q < v.n_src; q += blocks * kNodeThreads) {
        const int grp = q / kGroupSrc;
        if (v.outlier[stage * v.words + (grp >> 5)] >> (grp & 31) & 1u) continue;
        const float4 h = src[2 * q], l = src[2 * q + 1];
        const float x = ((h.x - g.ox) + l.x) * unit, y = ((h.y - g.oy) + l.y) * unit, z = ((h.z - g.oz) + l.z) * unit;
        const float r2 = fmaf(x, x, fmaf(y, y, z * z));
        const double m64 = h.w;
        M[0] += m64;
        M[1] = fma(m64, ((double)h.x - g.ox) + l.x, M[1]);
        M[2] = fma(m64, ((double)h.y - g.oy) + l.y, M[2]);
        M[3] = fma(m64, ((double)h.z - g.oz) + l.z, M[3]);
        float ex = h.w, ey = 0.f;                 // mass (x + iy)^m
        each<0, kCellP + 1>([&](auto mc) {
            constexpr int m = decltype(mc)::v;
            if constexpr (m > 0) {
                const float fx = ex * x - ey * y, fy = ex * y + ey * x;
                ex = fx;
                ey = fy;
            }
            float q2 = 0.f, q1 = 1.f;
            each<m, kCellP + 1>([&](auto nc) {
                constexpr int n = decltype(nc)::v;
                const float t = n == m ? 1.f : (n == m + 1 ? z : fmaf(r2 * q2, -harm_g(n, m), z * q1));
                re[multi_at(n, m)] = fmaf(t, ex, re[multi_at(n, m)]);
                if constexpr (m > 0) im[multi_at(n, m)] = fmaf(t, ey, im[multi_at(n, m)]);
                q2 = q1;
                q1 = t;
            });
        });
    }
    each<0, kMultiCoef>([&](auto kc) {
        constexpr int k = decltype(kc)::v;
        float a = re[k], b = im[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) { red[warp][2 * k] = a; red[warp][2 * k + 1] = b; }
    });
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M[k] += __shfl_xor_sync(0xffffffffu, M[k], o);
        if (lane == 0) mom[warp][k] = M[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0.0;
        for (int w = 0; w < kNodeWarps; ++w) t += mom[w][threadIdx.x];
        v.moments[((size_t)stage * kMultiBlocks + block) * 4 + threadIdx.x] = t;
        __threadfence();
    }
    float* const part = v.multi + ((size_t)stage * kMultiBlocks + block) * 2 * kMultiCoef;
    for (int k = threadIdx.x; k < 2 * kMultiCoef; k += kNodeThreads) {
        float t = 0.f;
        for (int w = 0; w < kNodeWarps; ++w) t += red[w][k];
        part[k] = t;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&v.done[stage], 1u) + 1u == (uint32_t)blocks;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = threadIdx.x; k < 2 * kMultiCoef; k += kNodeThreads) {
        float t = 0.f;
        for (int b = 0; b < blocks; ++b)
            t += *(volatile float*)(v.multi + ((size_t)stage * kMultiBlocks + b) * 2 * kMultiCoef + k);
        C[k] = t;
    }
    if (threadIdx.x < 4) {
        double t = 0.0;
        for (int b = 0; b < blocks; ++b)
            t += *(volatile double*)(v.moments + ((size_t)stage * kMultiBlocks + b) * 4 + threadIdx.x);
        total[threadIdx.x] = t;
    }
    __syncthreads();
    // the centre of mass carries the monopole and the dipole in FP64 (Body point); the
    // expansion keeps what its own multipoles about the origin leave of degree 2 and more
    const double inv_m = total[0] != 0.0 ? 1.0 / total[0] : 0.0;
    const double R[3] = {total[1] * inv_m, total[2] * inv_m, total[3] * inv_m};
    if (threadIdx.x == 0) v.point[stage] = make_body(g.ox + R[0], g.oy + R[1], g.oz + R[2], total[0]);
    if (threadIdx.x < kMultiCoef) {
        int n = 0, m = threadIdx.x;
        while (m > n) { m -= n + 1; ++n; }
        const double x = R[0] * unit, y = R[1] * unit, z = R[2] * unit, r2 = x * x + y * y + z * z;
        double ex = 1.0, ey = 0.0, q2 = 0.0, q1 = 1.0;
        for (int j = 0; j < m; ++j) {
            const double fx = ex * x - ey * y;
            ey = ex * y + ey * x;
            ex = fx;
        }
        for (int j = m + 1; j <= n; ++j) {
            const double gj = (double)((j - 1) * (j - 1) - m * m) / (double)((2 * j - 1) * (2 * j - 3));
            const double q = z * q1 - (j > m + 1 ? gj * r2 * q2 : 0.0);
            q2 = q1;
            q1 = q;
        }
        C[2 * threadIdx.x] = n < 2 ? 0.f : (float)((double)C[2 * threadIdx.x] - total[0] * q1 * ex);
        C[2 * threadIdx.x + 1] = n < 2 ? 0.f : (float)((double)C[2 * threadIdx.x + 1] - total[0] * q1 * ey);
    }
    __syncthreads();
    if (threadIdx.x >= kFarTerms) return;
    int mu = 0, rem = threadIdx.x;
    while (rem >= kCellP + 2 - (mu > 0 ? mu : 1)) { rem -= kCellP + 2 - (mu > 0 ? mu : 1); ++mu; }
    const int k = (mu > 0 ? mu : 1) + rem, n = k - 1;
    const float u2 = unit * unit, fp = v.tab->fp[threadIdx.x] * u2, fm = v.tab->fm[threadIdx.x] * u2;
    const float fz = v.tab->fz[threadIdx.x] * u2;
    const float2* L = reinterpret_cast<const float2*>(C);
    const float2 zero = make_float2(0.f, 0.f);
    const float2 lp = mu + 1 <= n ? L[multi_at(n, mu + 1)] : zero, lz = mu <= n ? L[multi_at(n, mu)] : zero;
    float4* const F = v.distant + (size_t)stage * kFarForce4;
    if (mu == 0) {
        F[k - 1] = make_float4(fp * lp.x, fp * lp.y, fz * lz.x, 0.f);
    } else {
        const float2 lm = mu - 1 <= n ? L[multi_at(n, mu - 1)] : zero;
        const float px = fp * lp.x, py = fp * lp.y, mx = fm * lm.x, my = fm * lm.y;
        const int o = kCellP + 1 + 2 * (threadIdx.x - kCellP - 1);
        F[o] = make_float4(px - mx, py - my, py + my, -(px + mx));
        F[o + 1] = make_float4(fz * lz.x, fz * lz.y, 0.f, 0.f);
    }
}

__global__ void __launch_bounds__(kNodeThreads, 3)
cells_far_kernel(CellView v, int distant_blocks) {
    after_previous();
    if (!v.grid->ok) return;
    union Shared {
        FarShared far;
        DistantShared distant;
    };
    __shared__ __align__(16) unsigned char raw[sizeof(Shared)];
    Shared& sh = *reinterpret_cast<Shared*>(raw);
    if ((int)blockIdx.x < 4 * distant_blocks) {
        distant_sums(v, blockIdx.x / distant_blocks, blockIdx.x % distant_blocks, distant_blocks, sh.distant);
        __syncthreads();
    }
    // the levels from the top down are one range of nodes
    int total = 0;
    for (int l = v.levels - 1; l >= 0; --l) {
        int first;
        total += level_nodes(v, l, first);
    }
    for (;;) {
        int k = 0;
        if ((threadIdx.x & 31) == 0) k = (int)atomicAdd(&v.grid->taken, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= total) break;
        far_sums(v, k, sh.far);
    }
}

// a + b; returns the rounding error of the sum that replaces a.
__device__ __forceinline__ float add_exact(float& a, float b) {
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
    a = s;
    return e;
}

// One level: the parents' expansions, translated, added to the nodes', and the terms of the
// force components.  A block takes kShiftNodes nodes, a thread per coefficient.
constexpr int kShiftNodes = 4;
constexpr int kShiftThreads = (kReal + 31) / 32 * 32;
constexpr int kForceSplit = kShiftThreads / kCellForce;     // nodes whose force terms are formed at once

__global__ void __launch_bounds__(kShiftThreads)
cells_shift_kernel(CellView v, int level) {
    after_previous();
    __shared__ __align__(16) float par[kReal][kShiftNodes];    // parents' coefficients, reflected to (+, +, +)
    __shared__ __align__(8) float lam[kShiftNodes][kReal];
    __shared__ int neg[kShiftNodes], parent[kShiftNodes];
    __shared__ float inv_edge[kShiftNodes];
    __shared__ __align__(16) float sh_val[kCellShift];
    __shared__ __align__(16) unsigned char sh_idx[kCellShift];
    int first;
    const int count = level_nodes(v, level, first);
    const int t = threadIdx.x;
    if (blockIdx.x * kShiftNodes >= count) return;
    // this thread's force term (k, mu) = (fk, fmu) and its factors
    const int f = t % kCellForce;
    int fmu = 0, fk = f;
    while (fk >= kCellP - fmu) { fk -= kCellP - fmu; ++fmu; }
    fk += fmu;
    const float ap = v.tab->ap[f], am = v.tab->am[f], az = v.tab->az[f];
    int e0 = 0, e1 = 0;
    if (level < v.levels - 1) {                   // the translation's entries, loaded once per block
        constexpr int kW = (kCellShift / 4 + kShiftThreads - 1) / kShiftThreads, kX = (kCellShift / 16 + kShiftThreads - 1) / kShiftThreads;
        const int nv = (v.tab->sh_first[kReal] + 3) / 4, nx = (v.tab->sh_first[kReal] + 15) / 16;
        uint4 w[kW], x[kX];                       // in flight together
#pragma unroll
        for (int q = 0; q < kW; ++q)
            if (t + q * kShiftThreads < nv) w[q] = __ldg(reinterpret_cast<const uint4*>(v.tab->sh_val) + t + q * kShiftThreads);
#pragma unroll
        for (int q = 0; q < kX; ++q)
            if (t + q * kShiftThreads < nx) x[q] = __ldg(reinterpret_cast<const uint4*>(v.tab->sh_idx) + t + q * kShiftThreads);
#pragma unroll
        for (int q = 0; q < kW; ++q)
            if (t + q * kShiftThreads < nv) reinterpret_cast<uint4*>(sh_val)[t + q * kShiftThreads] = w[q];
#pragma unroll
        for (int q = 0; q < kX; ++q)
            if (t + q * kShiftThreads < nx) reinterpret_cast<uint4*>(sh_idx)[t + q * kShiftThreads] = x[q];
        if (t < kReal) { e0 = v.tab->sh_first[t]; e1 = v.tab->sh_first[t + 1]; }
    }
    for (int b = blockIdx.x * kShiftNodes; b < count; b += gridDim.x * kShiftNodes) {
        const int n = min(kShiftNodes, count - b);
        const bool root = level == v.levels - 1;
        if (t < kShiftNodes && !root) {
            const CellNode& nd = v.node[first + b + min(t, n - 1)];
            parent[t] = nd.parent;
            neg[t] = nd.stage >> 2;
        }
        if (t < kShiftNodes) inv_edge[t] = v.node[first + b + min(t, n - 1)].inv_s;
        const int i = t;
        float val[kShiftNodes];                   // all loads of a thread in flight together
        const int li = low_of(i);                 // degree 1: also its low part
        float low[kShiftNodes];
        if (i < kReal)
#pragma unroll
            for (int j = 0; j < kShiftNodes; ++j) {
                val[j] = v.lam[(size_t)(first + b + min(j, n - 1)) * kReal + i];
                low[j] = li >= 0 ? v.lam[(size_t)(first + b + min(j, n - 1)) * kReal + li] : 0.f;
            }
        __syncthreads();
        if (!root) {
            const unsigned flip = i < kReal ? v.tab->neg[i] : 0;
            if (i < kReal) {
                float p[kShiftNodes], pl[kShiftNodes];
#pragma unroll
                for (int j = 0; j < kShiftNodes; ++j) {
                    p[j] = v.lam[(size_t)parent[j] * kReal + i];
                    pl[j] = li >= 0 ? v.lam[(size_t)parent[j] * kReal + li] : 0.f;
                }
#pragma unroll
                for (int j = 0; j < kShiftNodes; ++j) {
                    par[i][j] = __popc(flip & neg[j]) & 1 ? -p[j] : p[j];
                    if (li >= 0) low[j] += add_exact(val[j], 0.25f * p[j]) + 0.25f * pl[j];
                }
            }
            __syncthreads();
            if (i < kReal) {
                float acc[kShiftNodes] = {};
                shift_sums(par, sh_val, sh_idx, e0, e1, acc);
#pragma unroll
                for (int j = 0; j < kShiftNodes; ++j) {
                    const float rest = __popc(flip & neg[j]) & 1 ? -acc[j] : acc[j];
                    if (li >= 0) {
                        low[j] += add_exact(val[j], rest);
                        if (j < n) v.lam[(size_t)(first + b + j) * kReal + li] = low[j];
                    } else {
                        val[j] += rest;
                    }
                    if (j < n && !is_low(i)) v.lam[(size_t)(first + b + j) * kReal + i] = val[j];
                }
            }
        }
        if (i < kReal)
#pragma unroll
            for (int j = 0; j < kShiftNodes; ++j) {
                if (!is_low(i)) lam[j][i] = val[j];
                if (li >= 0) lam[j][li] = low[j];
            }
        __syncthreads();
        // force terms: with potential coefficients L(n, m), the force components' are
        // X(k, u) = L(k+1, u+1) - L(k+1, u-1), Y = -i (L(k+1, u+1) + L(k+1, u-1)), Z = L(k+1, u)
        if (t < kForceSplit * kCellForce)
            for (int j = t / kCellForce; j < n; j += kForceSplit) {
                const float inv_s = inv_edge[j], is2 = inv_s * inv_s;
                const float2* L = reinterpret_cast<const float2*>(lam[j]);
                const float2 lp = L[coef_at(fk + 1, fmu + 1)], lz = L[coef_at(fk + 1, fmu)];
                float4* F = v.force + (size_t)(first + b + j) * kCellForce4;
                if (fmu == 0) {
                    // fk = 0, the uniform pull (ap = az = 1): high parts here, low parts in the next terms' w
                    const float il = fmaf(inv_s, inv_s, -is2);
                    const int part = fk == 0 ? 2 : fk == 1 ? 3 : 0;
                    const float hi = lam[j][part], ph = hi * is2;
                    const float pl = fmaf(hi, is2, -ph) + fmaf(hi, il, lam[j][low_of(part)] * is2);
                    F[fk] = make_float4(ap * is2 * lp.x, ap * is2 * lp.y, az * is2 * lz.x, fk < 3 ? pl : 0.f);
                } else {
                    const float2 lm = L[coef_at(fk + 1, fmu - 1)];
                    const float px = ap * is2 * lp.x, py = ap * is2 * lp.y, mx = am * is2 * lm.x;
                    const float my = fmu == 1 ? 0.f : am * is2 * lm.y;
                    F[kCellP + 2 * (f - kCellP)] = make_float4(px - mx, py - my, py + my, -(px + mx));
                    F[kCellP + 2 * (f - kCellP) + 1] = make_float4(az * is2 * lz.x, az * is2 * lz.y, 0.f, 0.f);
                }
            }
        __syncthreads();
    }
}

// Sum of the nodes' numbers of near groups (diagnostics).
__global__ void cells_near_kernel(const CellNode* __restrict__ node, int n, unsigned long long* __restrict__ sum) {
    unsigned long long t = 0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) t += (unsigned)node[k].n_near;
    if (t) atomicAdd(sum, t);
}

size_t round256(size_t n) { return (n + 255) / 256 * 256; }

}  // namespace

void cells_free(CellScratch*& c) {
    while (c) {
        CellScratch* const next = c->outgrown;
        cudaFree(c->arena);
        delete c;
        c = next;
    }
}

constexpr long long kCellBytes = 32ll << 30;    // of nodes, at most (reached at 147,000 planetesimals)

bool cells_hold(const CellScratch* c, int n_src, int n_dust) { return c && c->cap_src >= n_src && c->cap_dust >= n_dust; }

cudaError_t cells_count(const CellScratch* c, long long* nodes, long long* room, int* dropped, double* near,
                        cudaStream_t st) {
    CellGrid g;
    cudaError_t e = cudaMemcpyAsync(&g, c->v.grid, sizeof(g), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    *nodes = 0;
    for (int l = g.min_level; l < kCellMaxLevels; ++l) *nodes += g.cnt[l];
    *room = c->v.cap;
    *dropped = g.min_level;
    unsigned long long sum = 0;               // in the setup's sums, which the next step clears
    e = cudaMemsetAsync(c->sums, 0, sizeof(sum), st);
    if (e == cudaSuccess) {
        launch_first(cells_near_kernel, 152, 256, 0, st, c->v.node, (int)*nodes, c->sums);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&sum, c->sums, sizeof(sum), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    *near = *nodes ? (double)sum / (double)*nodes : 0.0;
    return e;
}

cudaError_t cells_ensure(CellScratch*& c, int n_src, int n_dust, int most) {
    if (cells_hold(c, n_src, n_dust)) return cudaSuccess;
    int cap_dust = INT_MAX;
    if (!c && n_dust <= 1 << 29)
        for (cap_dust = 4096; cap_dust < n_dust;) cap_dust *= 2;
    const int want = c && most > n_src ? most : n_src, cap_src = (want + 1023) / 1024 * 1024;
    static CellTables tab;
    static const bool tab_ok = make_tables(tab);
    if (!tab_ok) return cudaErrorInvalidValue;
    // Nodes: a level that does not fit is left out (its parents stay leaves), and then the
    // tracers together decide how far cells are split, so there is room for planetesimals whose surroundings
    // are full of tracers out to the distant expansion.  Measured with six million tracers, the edge just
    // above its rounding's thresholds (the finest it gets), rings and disks up to the limits of the sets that take
    // cells, tilted ones and clumps: at most 112, 103, 90, 91, 86, 64, 58, 50 and 36 nodes per planetesimal at 2,048,
    // 3,069, 4,093, 6,141, 8,189, 16,381, 40,000, 65,536 and 131,072; there is room for 120 (180 at 2,048) and 58.  A belt of 4,096
    // with a million tracers in it takes 32,000, one with a wide halo 120,000.  A tracer needs one cell a level and
    // stage at most, which is less for few tracers (16,384 with 4,096 planetesimals: 1.0 GB instead of 1.5).
    const int groups = cap_src / kGroupSrc, words = (groups + 31) / 32;
    const long long bytes = sizeof(CellNode) + 4 * kReal + 16 * kCellForce4 + 4ll * words + 2 * kNearList;
    const long long want_nodes = 58ll * cap_src + 62ll * (cap_src < 16384 ? cap_src : 16384);
    const long long most_nodes = kCellBytes / bytes > 2097152 ? kCellBytes / bytes : 2097152;
    const int G = grid_dim(cap_src);
    const size_t cap = (size_t)std::min({want_nodes, most_nodes, 4ll * grid_levels(G) * cap_dust});
    const size_t marks = 3 * 4 * (size_t)cell_word0(G, grid_levels(G));
    const size_t sizes[] = {sizeof(CellGrid), sizeof(CellNode) * cap, 4ull * kReal * cap, 16ull * kCellForce4 * cap,
                            4ull * words * cap, 2ull * kNearList * cap, 4ull * kCellTop * kCellTop * kCellTop, 2 * marks,
                            32ull * 4 * groups, 32ull * 4 * (cap_src + 16), 4ull * 64 * kGroupPairs * (groups + 1), kSetupSums * sizeof(unsigned long long) + 4 * (1 + words) * sizeof(uint32_t),
                            4ull * 4 * kMultiBlocks * 2 * kMultiCoef, 8ull * 4 * kMultiBlocks * 4,
                            16ull * 4 * kFarForce4, 4 * sizeof(Body), sizeof(CellTables), 4ull * (kCellBins + 1),
                            4ull * (kCellBins + 1), 4ull * scan_temp_words(kCellBins + 1)};
    size_t total = 0;
    for (const size_t b : sizes) total += round256(b);
    char* arena = nullptr;
    cudaError_t e = cudaMalloc((void**)&arena, total);
    if (e != cudaSuccess) return e;
    CellScratch* n = new (std::nothrow) CellScratch();
    if (!n) {
        cudaFree(arena);
        return cudaErrorMemoryAllocation;
    }
    n->arena = arena;
    n->cap_src = cap_src;
    n->cap_dust = cap_dust;
    char* p = arena;
    int k = 0;
    auto take = [&]() { char* r = p; p += round256(sizes[k++]); return r; };
    CellView& v = n->v;
    v.grid = (CellGrid*)take();
    v.node = (CellNode*)take();
    v.lam = (float*)take();
    v.force = (float4*)take();
    v.near = (uint32_t*)take();
    v.list = (uint16_t*)take();
    v.root = (int*)take();
    v.own = (uint32_t*)take();
    v.gbox = (float4*)take();
    v.src = (float4*)take();
    v.near_rec = (ulonglong2*)take();
    n->sums = (unsigned long long*)take();
    v.done = (uint32_t*)(n->sums + kSetupSums);
    v.outlier = v.done + 4;
    v.multi = (float*)take();
    v.moments = (double*)take();
    v.distant = (float4*)take();
    v.point = (Body*)take();
    v.tab = (const CellTables*)take();
    n->count = (uint32_t*)take();
    n->start = (uint32_t*)take();
    n->temp = (uint32_t*)take();
    v.cap = (int)cap;
    e = cudaMemcpy((void*)v.tab, &tab, sizeof(tab), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cells_free(n);
        return e;
    }
    n->outgrown = c;
    c = n;
    return cudaSuccess;
}

cudaError_t cells_build(CellScratch* c, const ddx_state& s, const StepArgs& a, const MassiveScratch& ms,
                        const SizeBin* bins, CellView& v, cudaStream_t st) {
    if (!cells_hold(c, a.n_grav - a.n_exact, a.n_dust)) return cudaErrorInvalidValue;
    v = c->v;
    v.n_src = a.n_grav - a.n_exact;
    v.n_groups = (v.n_src + kGroupSrc - 1) / kGroupSrc;
    v.words = (v.n_groups + 31) / 32;
    v.G = grid_dim(v.n_src);
    v.levels = grid_levels(v.G);
    v.mark_words = cell_word0(v.G, v.levels);
    const size_t marks = 3 * 4 * (size_t)v.mark_words;
    v.mark = v.own + marks / 4;
    const OrderScratch& o = ms.dust_order;
    cudaError_t e = cudaMemsetAsync(v.own, 0, 2 * marks, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->count, 0, 4 * ((size_t)kCellBins + 1), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->sums, 0, kSetupSums * sizeof(unsigned long long) + 4 * (1 + (size_t)v.words) * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    launch_first(cells_setup_kernel, (v.n_src + kSetupThreads - 1) / kSetupThreads, kSetupThreads, 0, st, ms.P,
                 a.n_exact, v.n_src, v.G, last_octave_of(ms.src_order), c->sums, v.grid);
    launch_after(cells_boxes_kernel, (4 * ((v.n_groups + 1) / 2) * 32 + 127) / 128, 128, 0, st, ms.PP, ms.pcap, v);
    const int blk = (a.n_dust + 255) / 256;
    launch_after(cells_keys_kernel, blk, 256, 0, st, s, a, bins, v, o.key, o.rank, c->count);
    e = exclusive_scan(c->count, c->start, (int)kCellBins + 1, c->temp, nullptr, st);
    if (e != cudaSuccess) return e;
    launch_after(cells_scatter_kernel, blk, 256, 0, st, a.n_dust, o.key, o.rank, c->start, o.perm);
    int chunks = 0;
    for (int l = 0; l < v.levels; ++l) {
        const int n = cell_dim(v.G, l) / 32;
        chunks += n * n * n;
    }
    launch_after(cells_ancestors_kernel, dim3(chunks, 3), 1024, 0, st, v);
    launch_after(cells_roots_kernel, kCellTop * kCellTop * kCellTop / kRootThreads, kRootThreads, 0, st, v);
    // blocks per SM: as many splits and translations as fit, for their latency (a warp or a block per node); the far
    // sums' three by launch bounds
    const int sms = sm_count();
    for (int l = v.levels - 1; l >= 0; --l)
        launch_after(cells_split_kernel, 8 * sms, kNodeThreads, 0, st, v, l, a.near_eta);
    const int db = (v.n_src + 4 * kNodeThreads - 1) / (4 * kNodeThreads);
    launch_after(cells_far_kernel, 3 * sms, kNodeThreads, 0, st, v, db < kMultiBlocks ? db : kMultiBlocks);
    for (int l = v.levels - 1; l >= 0; --l) launch_after(cells_shift_kernel, 10 * sms, kShiftThreads, 0, st, v, l);
    return cudaGetLastError();
}

}  // namespace ddx
