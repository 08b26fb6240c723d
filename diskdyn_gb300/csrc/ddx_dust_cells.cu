// Mixed-precision RK4 of the dust tracers with cell expansions (ddx_cells.cu), for
// kCellMinSources planetesimals or more in a flat set (CellGrid::ok; else it leaves at once and
// ddx_dust_mixed.cu's kernel takes the step).  The physics and the precisions are those of
// ddx_dust_mixed.cu: FP64 state, star term, planets and RK4 combination; FP32 hi/lo
// separations, sums over 16 planetesimals with one FP32 Kahan sum per axis across them, and
// FP64 pulls within the near radius.  The difference is which planetesimals are taken one by
// one: those of the groups that are not far from the tracer's cell; the others act through
// the cell's expansion.
//
// The tracers go in cell order, so the lanes of a warp mostly share one cell and read its
// group list, records and expansion terms by broadcast from L1.  Reading records bounds the
// kernel (18 to 24 cycles of L1 a record against 9 of FP32), so a group's eight pair records lie
// part by part, 16 bytes a record, and a tracer starts at the record given by the group's
// number: lanes with different groups then read different banks (a belt of 4,096 with
// a million tracers 1575 -> 1515 us, 3,001 planetesimals with 30,000 tracers 234 -> 171 us).
// A tracer outside every grid, with a non-finite position, further from its cell's centre
// than kReach edges (it moved more in the step than expected), or expected to be distant but out
// of the distant expansion's reach takes every planetesimal.
#include "ddx_launch.cuh"
#include "ddx_cells.cuh"
#include "ddx_pull.cuh"

namespace ddx {
namespace {

constexpr int kThreads = 128;
constexpr float kReach = 0.55f;
constexpr int kDistantNode = -2;        // the tracer takes the distant expansion
// Few tracers leave most of the GPU idle, so 8 or 4 lanes share one below these numbers (us a
// step with 8 / 4 lanes at 7,000 tracers: 452 / 479 for 2,100 planetesimals, 1131 / 1192 for 9,000;
// at 9,000: 498 / 490 for 3,001; with 4 / 1 at 32,000: 582 / 617 and 1425 / 1539, a narrow belt of 4,096 635 /
// 634; at 40,000, more than one wave of 4 lanes: 664 / 638, 1572 / 1577, 695 / 653).
constexpr int kLanes8 = 8000, kLanes4 = 34000;

__host__ __device__ constexpr float harm_g(int n, int m) {
    return (float)((double)((n - 1) * (n - 1) - m * m) / (double)((2 * n - 1) * (2 * n - 3)));
}

// The cell expansion's acceleration at (x, y, z), in cell edges from the centre: its uniform
// part's high parts in u, the rest in (ax, ay, az).
__device__ __forceinline__ void l2p(const float4* __restrict__ F, float x, float y, float z, float (&u)[3], float& ax,
                                    float& ay, float& az) {
    const float r2 = fmaf(x, x, fmaf(y, y, z * z));
    const float4 c0 = __ldg(F), c1 = __ldg(F + 1), c2 = __ldg(F + 2);
    u[0] = c0.x; u[1] = c0.y; u[2] = c0.z;
    float sx = c0.w, sy = c1.w, sz = c2.w;
    {
        float q2 = 1.f, q1 = 1.f;
#pragma unroll
        for (int n = 1; n < kCellP; ++n) {
            const float q = n == 1 ? z : fmaf(r2 * q2, -harm_g(n, 0), z * q1);
            const float4 c = n == 1 ? c1 : n == 2 ? c2 : __ldg(F + n);
            sx = fmaf(c.x, q, sx); sy = fmaf(c.y, q, sy); sz = fmaf(c.z, q, sz);
            q2 = q1;
            q1 = q;
        }
    }
    f2 SX = f2_join(sx, 0.f), SY = f2_join(sy, 0.f), SZ = f2_join(sz, 0.f);
    float ex = 1.f, ey = 0.f;
    int k = kCellP;
#pragma unroll
    for (int m = 1; m < kCellP; ++m) {
        const float fx = fmaf(ex, x, -(ey * y)), fy = fmaf(ex, y, ey * x);
        ex = fx;
        ey = fy;
        const f2 E = f2_join(ex, ey);
        float q2 = 0.f, q1 = 1.f;
        f2 px = 0, py = 0, pz = 0;
#pragma unroll
        for (int n = m; n < kCellP; ++n, k += 2) {
            const float q = n == m ? 1.f : (n == m + 1 ? z : fmaf(r2 * q2, -harm_g(n, m), z * q1));
            const ulonglong2 c = __ldg(reinterpret_cast<const ulonglong2*>(F + k));
            const f2 cz = __ldg(reinterpret_cast<const unsigned long long*>(F + k + 1));
            const f2 Q = f2_dup(q);
            px = fma2(c.x, Q, px); py = fma2(c.y, Q, py); pz = fma2(cz, Q, pz);
            q2 = q1;
            q1 = q;
        }
        SX = fma2(px, E, SX); SY = fma2(py, E, SY); SZ = fma2(pz, E, SZ);
    }
    float s, t;
    f2_split(SX, s, t); ax = s + t;
    f2_split(SY, s, t); ay = s + t;
    f2_split(SZ, s, t); az = s + t;
}

// Whether a tracer that is expected to be distant may take the distant expansion at (x, y, z) from the
// origin: still kDistantReach times the core's largest distance away (the series is then as good
// as a cell's, 1 / 5.5 against 0.21), and with no planetesimal of the core within its near radius, near_eta times
// its largest |coordinate| own (each is at least 1 - 1 / 5.5 of its distance away).
constexpr float kDistantReach = 5.5f;
__device__ __forceinline__ bool distant_reach(const CellGrid& g, float x, float y, float z, float near_eta, float own) {
    const float r2 = fmaf(x, x, fmaf(y, y, z * z)), near = 1.25f * near_eta * own;
    return r2 >= kDistantReach * kDistantReach * __uint_as_float(g.b2) && r2 >= near * near;
}

// The acceleration of the distant expansion at (x, y, z) from the origin, in its unit.
__device__ __forceinline__ void m2p(const float4* __restrict__ F, float x, float y, float z, float& ax, float& ay,
                                    float& az) {
    const float r2 = fmaf(x, x, fmaf(y, y, z * z));
    const float ri = rsqrt_newton(r2);
    const float v = ri * ri, zv = z * v, ux = x * v, uy = y * v;
    f2 SX = 0, SY = 0, SZ = 0;
    float ex = 1.f, ey = 0.f;
    int k = 0;
#pragma unroll
    for (int m = 0; m <= kCellP + 1; ++m) {
        float t2 = 0.f, t1 = ri;                          // T(m) = 1/r; degrees n - 2 and n - 1 of the recursion
        f2 px = 0, py = 0, pz = 0;
#pragma unroll
        for (int n = m; n <= kCellP + 1; ++n) {
            if (n > m) {
                const float t = n == m + 1 ? zv * t1 : fmaf(v * t2, -harm_g(n, m), zv * t1);
                t2 = t1;
                t1 = t;
            }
            if (n == 0) continue;
            const f2 T = f2_dup(t1);
            if (m == 0) {
                const float4 c = __ldg(F + k);
                px = fma2(f2_join(c.x, 0.f), T, px); py = fma2(f2_join(c.y, 0.f), T, py);
                pz = fma2(f2_join(c.z, 0.f), T, pz);
                ++k;
            } else {
                const ulonglong2 c = __ldg(reinterpret_cast<const ulonglong2*>(F + k));
                const f2 cz = __ldg(reinterpret_cast<const unsigned long long*>(F + k + 1));
                px = fma2(c.x, T, px); py = fma2(c.y, T, py); pz = fma2(cz, T, pz);
                k += 2;
            }
        }
        const f2 E = f2_join(ex, ey);
        SX = fma2(px, E, SX); SY = fma2(py, E, SY); SZ = fma2(pz, E, SZ);
        const float fx = fmaf(ex, ux, -(ey * uy)), fy = fmaf(ex, uy, ey * ux);
        ex = fx;
        ey = fy;
    }
    float u, w;
    f2_split(SX, u, w); ax = u + w;
    f2_split(SY, u, w); ay = u + w;
    f2_split(SZ, u, w); az = u + w;
}

// The FP64 values of a tracer wait in shared memory, one column per thread, while its FP32
// pulls are summed, so that those have the registers: the state at the start of the step,
// the stages' accelerations k_s and the factors of the star term.
enum { qX, qY, qZ, qVx, qVy, qVz, qK1, qK2 = qK1 + 3, qK3 = qK2 + 3, qK4 = qK3 + 3, qG = qK4 + 3, qC, qL, qKept };
struct Column {
    uint32_t at;
    __device__ __forceinline__ double get(int k) const {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + k * kThreads * 8));
        return v;
    }
    __device__ __forceinline__ void put(int k, double v) const {
        asm volatile("st.shared.f64 [%0], %1;" :: "r"(at + k * kThreads * 8), "d"(v));
    }
};

// Position of stage st (0..3) from the column: x + r_{st-1} c, r_s = v + k_{s-1} c.
__device__ __forceinline__ double stage_pos(const Column& col, int axis, int st, const StepArgs& a) {
    const double x = col.get(qX + axis);
    if (st == 0) return x;
    double r = col.get(qVx + axis);
    if (st >= 2) r = fma(col.get(qK1 + 3 * (st - 2) + axis), a.dt2, r);
    return fma(r, st == 3 ? a.dt : a.dt2, x);
}

// The RK4 combination (src/gpu_functions.cu:903-943) with r_s = v + k_{s-1} c_s put in:
// x += dt/6 (v + 2 r_2 + 2 r_3 + r_4), v += dt/6 (k_1 + 2 k_2 + 2 k_3 + k_4).
__device__ __forceinline__ void finish_tracer(const Column& col, const StepArgs& a, const ddx_state& s, int t) {
    double* const X[3] = {s.x, s.y, s.z};
    double* const V[3] = {s.vx, s.vy, s.vz};
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const double v = col.get(qVx + k), k1 = col.get(qK1 + k), k2 = col.get(qK2 + k), k3 = col.get(qK3 + k);
        const double r2 = fma(k1, a.dt2, v), r3 = fma(k2, a.dt2, v), r4 = fma(k3, a.dt, v);
        X[k][t] = fma(a.dt6, fma(2.0, r2 + r3, v) + r4, col.get(qX + k));
        V[k][t] = fma(a.dt6, fma(2.0, k2 + k3, k1) + col.get(qK4 + k), v);
    }
}

// The FP64 pull of one body added to the column's acceleration of stage st.
__device__ __noinline__ void add_point(const Body p, const Column col, int st, const StepArgs& a) {
    const double ex = p.x - stage_pos(col, 0, st, a), ey = p.y - stage_pos(col, 1, st, a), ez = p.z - stage_pos(col, 2, st, a);
    const double f = pull64(p.m, fma(ez, ez, fma(ey, ey, ex * ex)));
    const int kc = qK1 + 3 * st;
    col.put(kc, fma(f, ex, col.get(kc)));
    col.put(kc + 1, fma(f, ey, col.get(kc + 1)));
    col.put(kc + 2, fma(f, ez, col.get(kc + 2)));
}

// The node of a tracer at stage st: the deepest on the way down to the cell where it is
// expected; -1 when it has none or lies outside its reach.  (dx, dy, dz): its place in the cell.
__device__ __forceinline__ int find_node(const CellView& v, const CellAt& at, int st, float xh, float xl, float yh,
                                         float yl, float zh, float zl, float& dx, float& dy, float& dz) {
    const CellGrid& g = *v.grid;
    const int top = v.levels - 1, min_level = g.min_level;
    if (!g.ok || at.level < 0 || min_level > top) return -1;
    const int h = cell_dim(v.G, at.level) / 2;
    const int ix = at.ix - h, iy = at.iy - h, iz = at.iz - h;
    const int up = top - at.level;
    int node = v.root[((((iz >> up) + kCellTop / 2) * kCellTop) + (iy >> up) + kCellTop / 2) * kCellTop + (ix >> up) +
                      kCellTop / 2];
    if (node < 0) return -1;
    node += st;
    for (int l = top - 1; l >= at.level && l >= min_level; --l) {
        const int dn = l - at.level;
        const int c = v.node[node].child[(ix >> dn & 1) | (iy >> dn & 1) << 1 | (iz >> dn & 1) << 2];
        if (c < 0) break;
        node = c;
    }
    const float4 c = *reinterpret_cast<const float4*>(&v.node[node].cx);
    dx = ((xh - c.x) + xl) * c.w; dy = ((yh - c.y) + yl) * c.w; dz = ((zh - c.z) + zl) * c.w;
    return fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz))) <= kReach ? node : -1;
}

// What the FP32 sum over a tracer's groups needs and gives.
struct Pull {
    f2 XH, XL, YH, YL, ZH, ZL;
    float inv_near;
    SpanAcc<false> ax, ay, az;
    __device__ __forceinline__ void start(const float (&X)[6], float near_eta) {
        XH = f2_dup(X[0]); XL = f2_dup(X[1]); YH = f2_dup(X[2]); YL = f2_dup(X[3]); ZH = f2_dup(X[4]); ZL = f2_dup(X[5]);
        inv_near = near_inv(near_eta, fmaxf(fabsf(X[0]), fmaxf(fabsf(X[2]), fabsf(X[4]))));
    }
};
// A stage's sources.
struct Sources {
    const ulonglong2* rec;     // groups of pair records, part by part
    const BodyPair* pair;      // pair records
    const Body*     body;      // FP64 records
    const int*      src;       // source of each slot
};

// One pair record's pulls on a tracer added to (px, py, pz); mx: the largest reciprocal
// distance so far.
__device__ __forceinline__ void pull_record(const ulonglong2 q0, const ulonglong2 q1, const ulonglong2 q2, const f2 lz,
                                            const Pull& p, f2& px, f2& py, f2& pz, float& mx) {
    const f2 dX = add2(sub2(q0.x, p.XH), sub2(q2.x, p.XL));
    const f2 dY = add2(sub2(q0.y, p.YH), sub2(q2.y, p.YL));
    const f2 dZ = add2(sub2(q1.x, p.ZH), sub2(lz, p.ZL));
    const f2 RR = fma2(dX, dX, fma2(dY, dY, mul2(dZ, dZ)));
    float r0, r1;
    f2_split(RR, r0, r1);
    const float i0 = rsqrt_approx(r0), i1 = rsqrt_approx(r1);
    mx = fmax3(mx, i0, i1);
    const f2 ri = f2_join(i0, i1);
    const f2 f = mul2(mul2(q1.y, ri), mul2(ri, ri));
    px = fma2(f, dX, px); py = fma2(f, dY, py); pz = fma2(f, dZ, pz);
}

// The e-th group of a node's list (or of all groups), -1 when the node's mask leaves it out.
__device__ __forceinline__ int group_at(const uint16_t* list, const uint32_t* mask, int e) {
    if (list) return (int)__ldg(list + e);
    return !mask || (__ldg(mask + (e >> 5)) >> (e & 31) & 1u) ? e : -1;
}

// The groups of a tracer's node (n < 0: every group) added to p, one after the other with a
// Kahan sum across them.  A group's records are summed as four chains of two, added in pairs:
// with T > 1 four lanes take a chain each and add them by butterfly, which gives the same
// bits; with T = 8 the next four lanes take the next group.
template <int T>
__device__ __forceinline__ void pull_groups(const CellView& v, int n, bool on, const Sources& S, Pull& p,
                                            const Column col, int st, const StepArgs& a) {
    int cnt = on ? v.n_groups : 0;
    const uint16_t* list = nullptr;
    const uint32_t* mask = nullptr;
    if (n == kDistantNode) {
        mask = v.outlier + (size_t)st * v.words;
        if (v.grid->outliers == 0u) cnt = 0;
    } else if (on && n >= 0) {
        const int nn = v.node[n].n_near;
        if (nn <= kNearList) {
            cnt = nn;
            list = v.list + (size_t)n * kNearList;
        } else {
            mask = v.near + (size_t)n * v.words;
        }
    }
    constexpr int kTeams = T > 4 ? T / 4 : 1;
    const int team = T > 4 ? (threadIdx.x & (T - 1)) / 4 : 0;
    const int end = T > 1 ? (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt) : cnt;   // T > 1: the warp stays together
    for (int e0 = 0; e0 < end; e0 += kTeams) {
        const int e = e0 + team;
        f2 px = 0, py = 0, pz = 0;
        float mx = 0.f;                           // largest reciprocal distance of the group
        const int g = e < cnt ? group_at(list, mask, e) : -1;
        if (g >= 0) {
            const ulonglong2* const R = S.rec + (size_t)g * (4 * kGroupPairs);
            auto record = [&](int slot, f2& x, f2& y, f2& z) {
                pull_record(__ldg(R + slot), __ldg(R + kGroupPairs + slot), __ldg(R + 2 * kGroupPairs + slot),
                            __ldg(reinterpret_cast<const unsigned long long*>(R + 3 * kGroupPairs + slot)), p, x, y, z, mx);
            };
            if (T > 1) {
                const int slot = (g + threadIdx.x) & 3 ^ (g & 4);
                record(slot, px, py, pz);
                record(slot ^ 4, px, py, pz);
            } else {
                f2 hx = 0, hy = 0, hz = 0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    f2 qx = 0, qy = 0, qz = 0;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int slot = (g + 2 * h + k) & 3 ^ (g & 4);
                        f2 x = 0, y = 0, z = 0;
                        record(slot, x, y, z);
                        record(slot ^ 4, x, y, z);
                        if (k == 0) { qx = x; qy = y; qz = z; }
                        else { qx = add2(qx, x); qy = add2(qy, y); qz = add2(qz, z); }
                    }
                    if (h == 0) { hx = qx; hy = qy; hz = qz; }
                    else { px = add2(hx, qx); py = add2(hy, qy); pz = add2(hz, qz); }
                }
            }
        }
        if (T > 1) {
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                px = add2(px, __shfl_xor_sync(0xffffffffu, px, o));
                py = add2(py, __shfl_xor_sync(0xffffffffu, py, o));
                pz = add2(pz, __shfl_xor_sync(0xffffffffu, pz, o));
            }
        }
        const bool near = mx > p.inv_near;        // rare: a source within the near radius
        const unsigned nears = T > 1 ? __ballot_sync(0xffffffffu, near) : 0u;
#pragma unroll
        for (int j = 0; j < kTeams; ++j) {
            f2 sx = px, sy = py, sz = pz;
            int gj = g;
            const int from = (threadIdx.x & 31 & ~(T - 1)) + 4 * j;
            if (kTeams > 1) {
                sx = __shfl_sync(0xffffffffu, px, from);
                sy = __shfl_sync(0xffffffffu, py, from);
                sz = __shfl_sync(0xffffffffu, pz, from);
                gj = __shfl_sync(0xffffffffu, g, from);
            }
            if (gj < 0) continue;
            if (T > 1 ? (nears >> from & 15u) != 0u : near) {   // its pulls again, the near ones in FP64
                const int kc = qK1 + 3 * st;
                double kx = col.get(kc), ky = col.get(kc + 1), kz = col.get(kc + 2);
                sx = sy = sz = 0;
                near_span<kGroupPairs>(S.pair + (size_t)gj * kGroupPairs, gj * kGroupSrc, p.XH, p.XL, p.YH, p.YL, p.ZH,
                                       p.ZL, stage_pos(col, 0, st, a), stage_pos(col, 1, st, a), stage_pos(col, 2, st, a),
                                       p.inv_near, S.body, S.src, sx, sy, sz, kx, ky, kz);
                col.put(kc, kx); col.put(kc + 1, ky); col.put(kc + 2, kz);
            }
            p.ax.add(sx); p.ay.add(sy); p.az.add(sz);
        }
    }
}

// Six blocks an SM (80 registers): us a step with 6 / 7 / 8 for one lane per tracer, 4,096 planetesimals with a
// million tracers 2075 / 2065 / 2147, with 60,000 684 / 700 / 734, 3,001 with a halo and 500,003 1645 / 1639 / 1736, 9,000
// with a halo and 300,003 2743 / 2841 / 2952.  Seven with four and eight lanes (4,096 with 28,000: 618 / 623 /
// 634, but 30,000 tracers no longer fit into one wave of six: 3,001 with a halo 617 / 594 / 600).
template <int T>
__global__ void __launch_bounds__(kThreads, T > 1 ? 7 : 6)
dust_cells_kernel(ddx_state s, StepArgs a, MassiveScratch ms, const SizeBin* __restrict__ bins,
                  const int* __restrict__ perm, CellView v, const int* __restrict__ src) {
    after_previous();
    if (!v.grid->ok) return;
    __shared__ double held[qKept][kThreads];
    const Column col{(uint32_t)__cvta_generic_to_shared(&held[0][threadIdx.x])};
    const int slot = (blockIdx.x * blockDim.x + threadIdx.x) / T;
    const int i = slot < a.n_dust ? perm[slot] : a.n_dust;
    const int t = a.n_grav + i;
    bool alive = false;
    float red = 1.f;
    if (i < a.n_dust && s.N[t] != 0.0) {
        alive = true;
        col.put(qX, s.x[t]); col.put(qY, s.y[t]); col.put(qZ, s.z[t]);
        col.put(qVx, s.vx[t]); col.put(qVy, s.vy[t]); col.put(qVz, s.vz[t]);
        const int id = s.id[t];
        red = star_reduction(bins, id, a.n_grid);
        SizeBin b{0.f, 0.f, 0.f, 0.f};
        if (id >= 0 && id < a.n_grid) b = bins[id];
        const StarCoef k = star_coef(ms.P[0].m, b.beta, b.betasw, b.q, s.m[t], a);
        col.put(qG, k.g); col.put(qC, k.c); col.put(qL, k.l);
    }
    const float dtf = (float)a.dt;
    int removed = 0;                              // 1: sublimated, 2: coincidence, 3: sublimated at stage 4

#pragma unroll 1
    for (int st = 0; st < 4; ++st) {
        // stage s evaluates k_s at x_s = x + r_{s-1} c_s and r_s = v + k_{s-1} c_s
        // (src/gpu_functions.cu:627-943)
        const double c = st == 3 ? a.dt : a.dt2;
        float X[6] = {}, fx = 0.f, fy = 0.f, fz = 0.f;   // hi and lo parts of the position; the expansion's pull
        float uni[3] = {0.f, 0.f, 0.f};                  // its uniform part
        int node = -1;
        if (alive) {
            const double xt = stage_pos(col, 0, st, a), yt = stage_pos(col, 1, st, a), zt = stage_pos(col, 2, st, a);
            double rx = col.get(qVx), ry = col.get(qVy), rz = col.get(qVz);
            if (st > 0) {
                const int kp = qK1 + 3 * (st - 1);
                rx = fma(col.get(kp), c, rx); ry = fma(col.get(kp + 1), c, ry); rz = fma(col.get(kp + 2), c, rz);
            }
            double kx = 0, ky = 0, kz = 0;
            const Body ps = ms.P[st * ms.cap + 0];
            const StarCoef sc{col.get(qG), col.get(qC), col.get(qL)};
            if (!star_term(xt - ps.x, yt - ps.y, zt - ps.z, rx, ry, rz, sc, a, kx, ky, kz)) {
                alive = false;
                removed = st == 3 ? 3 : 1;
            }
            // the planets, in FP64
            for (int j = 1; alive && j < a.n_exact; ++j) {
                const Body p = ms.P[st * ms.cap + j];
                const double ex = p.x - xt, ey = p.y - yt, ez = p.z - zt;
                const double RR = fma(ez, ez, fma(ey, ey, ex * ex));
                if ((__double_as_longlong(RR) << 1) == 0) {
                    alive = false;
                    removed = 2;
                    break;
                }
                const double f = pull64(p.m, RR);
                kx = fma(f, ex, kx); ky = fma(f, ey, ky); kz = fma(f, ez, kz);
            }
            const int kc = qK1 + 3 * st;
            col.put(kc, kx); col.put(kc + 1, ky); col.put(kc + 2, kz);
            split2(xt, X[0], X[1]);
            split2(yt, X[2], X[3]);
            split2(zt, X[4], X[5]);
        }
        if (alive) {
            const CellGrid& g = *v.grid;
            float dx = (X[0] - g.ox) + X[1], dy = (X[2] - g.oy) + X[3], dz = (X[4] - g.oz) + X[5];
            // the expected place decides, as it did when the cells were marked: another place could
            // send the tracer to a cell that only others' marks have built
            const CellPos at = cell_predict(g, col.get(qX), col.get(qY), col.get(qZ), col.get(qVx), col.get(qVy),
                                            col.get(qVz), red, dtf, st);
            if (cell_distant(g, at.x, at.y, at.z)) {
                if (distant_reach(g, dx, dy, dz, a.near_eta, fmaxf(fabsf(X[0]), fmaxf(fabsf(X[2]), fabsf(X[4]))))) {
                    node = kDistantNode;
                    const float u = g.inv_s0 * (1.f / kFarUnit);
                    m2p(v.distant + (size_t)st * kFarForce4, dx * u, dy * u, dz * u, fx, fy, fz);
                    add_point(v.point[st], col, st, a);
                }
            } else {
                node = find_node(v, cell_at(g, v.G, v.levels, at), st, X[0], X[1], X[2], X[3], X[4], X[5], dx, dy, dz);
                if (node >= 0) l2p(v.force + (size_t)node * kCellForce4, dx, dy, dz, uni, fx, fy, fz);
            }
        }
        Pull p;
        p.start(X, a.near_eta);
        p.ax.add(f2_join(uni[0], 0.f)); p.ay.add(f2_join(uni[1], 0.f)); p.az.add(f2_join(uni[2], 0.f));
        const Sources S{v.near_rec + (size_t)st * v.n_groups * (4 * kGroupPairs), ms.PP + (size_t)st * ms.pcap,
                        ms.P + (size_t)st * ms.cap + a.n_exact, src};
        pull_groups<T>(v, node, alive, S, p, col, st, a);
        if (alive) {
            const int kc = qK1 + 3 * st;
            const double kx = col.get(kc), ky = col.get(kc + 1), kz = col.get(kc + 2);
            // An exact coincidence makes RR = 0, the rsqrt infinite and the sum NaN.
            if (!(isfinite(p.ax.S + fx) && isfinite(p.ay.S + fy) && isfinite(p.az.S + fz) && finite64(kx) &&
                  finite64(ky) && finite64(kz))) {
                alive = false;
                removed = 2;
            }
            col.put(kc, (kx + f2d_bits(p.ax.S)) + f2d_bits(fx - p.ax.C));
            col.put(kc + 1, (ky + f2d_bits(p.ay.S)) + f2d_bits(fy - p.ay.C));
            col.put(kc + 2, (kz + f2d_bits(p.az.S)) + f2d_bits(fz - p.az.C));
        }
    }
    if (i >= a.n_dust || (T > 1 && (threadIdx.x & (T - 1)))) return;
    if (removed) {
        if (removed == 3 && a.mode == DDX_MODE_REFERENCE) s.N[i] = 0;
        else s.N[t] = 0;
    } else if (alive) {
        finish_tracer(col, a, s, t);
    }
}

}  // namespace

cudaError_t launch_dust_cells(const ddx_state& s, const StepArgs& a, const MassiveScratch& ms, const SizeBin* bins,
                              const int*& done, cudaStream_t st) {
    CellView v;
    const cudaError_t e = cells_build(ms.cells, s, a, ms, bins, v, st);
    if (e != cudaSuccess) return e;
    done = &v.grid->ok;
    const int* const perm = ms.dust_order.perm;
    const int* const src = ms.slot ? ms.src : nullptr;
    const int lanes = a.n_dust < kLanes8 ? 8 : a.n_dust < kLanes4 ? 4 : 1;
    const int blocks = (int)(((long long)a.n_dust * lanes + kThreads - 1) / kThreads);
    if (lanes == 8) launch_first(dust_cells_kernel<8>, blocks, kThreads, 0, st, s, a, ms, bins, perm, v, src);
    else if (lanes == 4) launch_first(dust_cells_kernel<4>, blocks, kThreads, 0, st, s, a, ms, bins, perm, v, src);
    else launch_first(dust_cells_kernel<1>, blocks, kThreads, 0, st, s, a, ms, bins, perm, v, src);
    return cudaGetLastError();
}

}  // namespace ddx
