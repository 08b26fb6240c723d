// Cell expansions of the planetesimals' pull (ddx_cells.cu): declarations shared by the
// kernels that build them and the dust kernel that evaluates them.
#pragma once
#include "ddx_internal.cuh"
#include "ddx_f32x2.cuh"

namespace ddx {

constexpr int kCellP = 10;                                 // degree of the potential expansions
constexpr int kCellCoef = kCellP * (kCellP + 3) / 2;       // complex coefficients, degrees 1..kCellP
constexpr int kCellForce = kCellP * (kCellP + 1) / 2;      // terms of each force component, degrees 0..kCellP-1
constexpr int kFarTerms = (kCellP + 1) * (kCellP + 4) / 2;    // terms of the distant expansion's force, degrees 1..kCellP+1
constexpr int kFarForce4 = kCellP + 1 + 2 * (kFarTerms - kCellP - 1);
constexpr int kCellForce4 = kCellP + 2 * (kCellForce - kCellP);   // float4 per node: m = 0, then two per m > 0 term
constexpr int kGroupPairs = 8;                             // pair records per source group (16 sources)
constexpr int kGroupSrc = 2 * kGroupPairs;
constexpr int kCellMaxLevels = 8;
constexpr int kCellTop = 32;                               // cells per axis of the coarsest level
constexpr uint32_t kCellBins = 1u << 21;                   // cells of the tracer order, one more for removed tracers

// The nested grids of one step: level l has cubic cells of edge s0 2^l (s0: a power of two, or
// three times one), concentric with the origin (the star's position rounded to a multiple of
// s0, so every cell centre and every step between centres is exact in FP32).  Levels 0 to 3 have G cells per axis, the levels
// above cover the same region as level 3 with half as many per level, down to kCellTop.
struct CellGrid {
    float ox, oy, oz;          // origin
    float s0, inv_s0;
    float sx, sy, sz, m0;      // star at the start of the step (predicted stage positions)
    uint32_t b2;               // bits of the core's largest squared distance to the origin (all stages)
    uint32_t outliers;         // groups outside the core (all stages)
    int   ok;                  // 0: no cells this step (the span kernel takes every source)
    int   thin;                // a disk: the tracer order cuts it finer in its plane
    int   leaf;                // most groups near a cell that is not split
    int   min_level;           // levels below it were dropped (out of nodes)
    uint32_t cnt[kCellMaxLevels];     // nodes per level
    uint32_t taken;                   // nodes taken by cells_far_kernel
    uint32_t first[kCellMaxLevels];   // first node of each level (the top's is 0)
};

// One node: a cell of one RK4 stage's tree.
constexpr int kNearList = 128;                             // (of up to 65,536 groups)
struct __align__(16) CellNode {
    float cx, cy, cz, inv_s;   // centre, 1 / edge
    int   child[8];            // node of each octant (bit 0: +x, 1: +y, 2: +z), -1: none
    int   parent;              // -1: a root
    int   stage;               // RK4 stage | octant of the parent << 2 (bit set: the lower half of an axis)
    int   cell;                // ix | iy << 10 | iz << 20 on its level's grid
    int   n_near;              // groups near it (listed in CellView::list up to kNearList of them)
};

// Constants of the translation and of the force terms, formed on the host in FP64.
constexpr int kCellShift = 5120;                           // room for the translation's non-zero entries
struct CellTables {
    float w[2 * kCellCoef];                                // weight of each real coefficient after P2L
    float ap[kCellForce], am[kCellForce], az[kCellForce];  // force terms (k, mu) from the potential's
    float fp[kFarTerms], fm[kFarTerms], fz[kFarTerms];     // the same of the distant expansion
    // translation by (+1/4, +1/4, +1/4) of the parent's edge: column j (child coefficient) has
    // entries sh_first[j] .. sh_first[j + 1] - 1, parent coefficient and factor
    alignas(16) float sh_val[kCellShift];
    alignas(16) unsigned char sh_idx[kCellShift];
    unsigned short sh_first[2 * kCellCoef + 2];
    unsigned char neg[2 * kCellCoef];                      // bit a: the coefficient changes sign under axis a's reflection
};

constexpr int kMultiCoef = (kCellP + 1) * (kCellP + 2) / 2;  // complex coefficients, degrees 0..kCellP
constexpr int kMultiBlocks = 16;

// Degree 1 (the uniform pull, most of it) is carried in two floats.  The low parts of the
// real coefficients 0, 2 and 3 (degree 1) sit in imaginary parts of order 0, which are zero.
__host__ __device__ constexpr int low_of(int i) { return i == 0 ? 1 : i == 2 ? 5 : i == 3 ? 11 : -1; }
__host__ __device__ constexpr bool is_low(int i) { return i == 1 || i == 5 || i == 11; }

struct CellView {
    CellGrid*   grid;
    CellNode*   node;          // [cap]
    float*      lam;           // [cap][2 kCellCoef] potential coefficients (re, im); low parts of degree 1 at low_of
    float4*     force;         // [cap][kCellForce4]
    uint32_t*   near;          // [cap][words] source groups taken one by one
    uint16_t*   list;          // [cap][kNearList] the same as a list
    int*        root;          // [kCellTop^3] first of a root's four nodes (one per stage), -1: none
    uint32_t*   own;           // [3] marked cells per level, the levels one after the other: where tracers
                               // are expected at stage 0, at stages 1 and 2, at stage 3
    uint32_t*   mark;          // [3] the same with every marked cell's ancestors marked too
    int         mark_words;    // of one of the three
    float4*     gbox;          // [4][n_groups][2] source group boxes: min (w: 1 when a coordinate is not finite), max
    float*      multi;         // [4][kMultiBlocks][2 kMultiCoef] partial sums of the distant expansion
    double*     moments;       // [4][kMultiBlocks][4] partial sums of m, m x, m y, m z
    float4*     distant;       // [4][kFarForce4] its force terms
    Body*       point;         // [4] the planetesimals' mass at their centre of mass
    uint32_t*   outlier;       // [4][words] groups outside the core
    uint32_t*   done;          // [4] blocks of a stage that have written theirs
    float4*     src;           // [4][n_groups * 16][2] sources by slot: high parts and mass, low parts
    ulonglong2* near_rec;      // [4][n_groups][4][8] pair records of a group, part by part (cells_boxes_kernel)
    const CellTables* tab;
    int cap, words, n_groups, n_src;
    int G, levels;
};

// Cells per axis of level l, and the first word of its marks.
__host__ __device__ inline int cell_dim(int G, int l) { return l <= 3 ? G : G >> (l - 3); }
__host__ __device__ inline int cell_level_words(int G, int l) {
    const int d = cell_dim(G, l);
    return d * d * (d / 32);
}
__host__ __device__ inline int cell_word0(int G, int l) {
    int w = 0;
    for (int k = 0; k < l; ++k) w += cell_level_words(G, k);
    return w;
}

// Builds the trees of one step for the tracers of s from the massive set's stage records (ms:
// P, PP and the tracer order's buffers), unless the planetesimals are none for cells (CellGrid::ok),
// orders the tracers into ms.dust_order.perm and fills v for the dust kernel.  Stream-ordered.
cudaError_t cells_build(CellScratch* c, const ddx_state& s, const StepArgs& a, const MassiveScratch& ms,
                        const SizeBin* bins, CellView& v, cudaStream_t st);
// The tracers' step with cells.  done: on the device, 0 when the planetesimals were none for cells and
// the tracers are as they were.
cudaError_t launch_dust_cells(const ddx_state& s, const StepArgs& a, const MassiveScratch& ms, const SizeBin* bins,
                              const int*& done, cudaStream_t st);

// x^(-1/2) within an FP32 rounding: rsqrt.approx and one Newton step whose residual 1 - x y^2 is
// formed with the square's rounding error.  (With a factor near one instead, y (1.5 - x y^2 / 2),
// the unequal spacing of FP32 on both sides of one made the far pulls of a belt weaker by 3e-9 in
// the mean, the same for every tracer.)
__device__ __forceinline__ float rsqrt_newton(float x) {
    const float y = rsqrt_approx(x), u = y * y;
    const float e = fmaf(-x, fmaf(y, y, -u), fmaf(-x, u, 1.f));
    return fmaf(0.5f * y, e, y);
}

// 1 - beta - beta_sw of a tracer's bin (1 without one), as cell_predict takes it.
__device__ __forceinline__ float star_reduction(const SizeBin* __restrict__ bins, int id, int n_grid) {
    if (id < 0 || id >= n_grid) return 1.f;
    const SizeBin b = bins[id];
    return __fsub_rn(__fsub_rn(1.f, b.beta), b.betasw);
}

// Tracers at kDistant times the core's largest distance or more from the origin take it
// through one expansion about the origin (the error bound is that of a cell's).  The core:
// the groups within core_edges finest cell edges of the origin (the grids reach kDistant times
// as far: 512 edges with 128 cells per axis, 1,024 with 256); they take the others, planetesimals
// scattered outwards, one by one.
constexpr float kDistant = 6.f;
__host__ __device__ constexpr float core_edges(int G) { return G == 128 ? 80.f : 160.f; }
__device__ __forceinline__ bool cell_distant(const CellGrid& g, float rx, float ry, float rz) {
    const float r2 = __fmaf_rn(rx, rx, __fmaf_rn(ry, ry, __fmul_rn(rz, rz)));
    return g.ok && r2 >= __fmul_rn(kDistant * kDistant, __uint_as_float(g.b2)) && r2 < 1e30f;
}

// Which marks a stage has.
__host__ __device__ constexpr int mark_set(int stage) { return (stage + 1) / 2; }

struct CellPos { float x, y, z; };
struct CellAt { int level, ix, iy, iz; };   // level < 0: outside every grid

// Where a tracer is expected at stage k (0: the start, 1 and 2: the middle, 3: the end of the
// step), relative to the origin: its start state advanced under the star's reduced gravity.
// The keys kernel (which marks cells) and the dust kernel (which looks them up) have to
// agree to the bit, so every operation is rounded on its own.
__device__ __forceinline__ CellPos cell_predict(const CellGrid& g, const double x, const double y, const double z,
                                                const double vx, const double vy, const double vz, float red,
                                                float dt, int k) {
    const float px = d2f_toward0(x), py = d2f_toward0(y), pz = d2f_toward0(z);
    CellPos p{__fsub_rn(px, g.ox), __fsub_rn(py, g.oy), __fsub_rn(pz, g.oz)};
    if (k == 0) return p;
    const float rx = __fsub_rn(px, g.sx), ry = __fsub_rn(py, g.sy), rz = __fsub_rn(pz, g.sz);
    const float rr = __fmaf_rn(rx, rx, __fmaf_rn(ry, ry, __fmul_rn(rz, rz)));
    const float ri = rsqrt_approx(rr);
    const float f = __fmul_rn(__fmul_rn(g.m0, red), __fmul_rn(ri, __fmul_rn(ri, ri)));
    const float t = k == 3 ? dt : __fmul_rn(0.5f, dt);
    const float h = __fmul_rn(__fmul_rn(-0.5f, f), __fmul_rn(t, t));
    p.x = __fmaf_rn(h, rx, __fmaf_rn(d2f_toward0(vx), t, p.x));
    p.y = __fmaf_rn(h, ry, __fmaf_rn(d2f_toward0(vy), t, p.y));
    p.z = __fmaf_rn(h, rz, __fmaf_rn(d2f_toward0(vz), t, p.z));
    return p;
}

// The unit of length of the distant expansion, in finest cell edges.
constexpr float kFarUnit = 32.f;

// The finest cell that holds p.
__device__ __forceinline__ CellAt cell_at(const CellGrid& g, int G, int levels, const CellPos& p) {
    CellAt c{-1, 0, 0, 0};
    const float ux = __fmul_rn(p.x, g.inv_s0), uy = __fmul_rn(p.y, g.inv_s0), uz = __fmul_rn(p.z, g.inv_s0);
    const float m = fmaxf(fabsf(ux), fmaxf(fabsf(uy), fabsf(uz)));
    const float half = 0.5f * (float)G * 0.999f;
    if (!(m < half * 8.f) || !(ux == ux) || !(uy == uy) || !(uz == uz)) return c;
    int l = 0;
    float sc = 1.f;
    while (m >= half / sc) { ++l; sc *= 0.5f; }            // l <= 3
    c.level = l;
    c.ix = (int)floorf(ux * sc) + G / 2;
    c.iy = (int)floorf(uy * sc) + G / 2;
    c.iz = (int)floorf(uz * sc) + G / 2;
    return c;
}

}  // namespace ddx
