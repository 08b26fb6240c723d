// Pieces of the planetesimals' FP32 pull shared by the mixed dust kernels: the FP64 pull of
// near sources and the sums across spans of pair records.
#pragma once
#include "ddx_internal.cuh"
#include "ddx_f32x2.cuh"

namespace ddx {
namespace {

// Box of a span's sources (high parts, padding slots left out) at one stage, written
// into the pad slots of the span's first four pair records R, so it reaches shared memory with
// the tile: record 0 {min x, max x}, record 1 {min y, max y}, record 2 {min z, max z},
// record 3 {max |coordinate|, 0}; the maximum is NaN when a coordinate is NaN (such a span
// never counts as far).  Every lane of the span's warp has the whole box and calls it.
__device__ __forceinline__ void store_span_box(BodyPair* R, const float (&lo)[3], const float (&hi)[3], bool nan) {
    const int u = threadIdx.x & 31;
    if (u < 3) {
        R[u].pad[0] = u == 0 ? lo[0] : u == 1 ? lo[1] : lo[2];
        R[u].pad[1] = u == 0 ? hi[0] : u == 1 ? hi[1] : hi[2];
    } else if (u == 3) {
        float xm = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) xm = fmaxf(xm, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
        R[3].pad[0] = nan ? __int_as_float(0x7FC00000) : xm;
        R[3].pad[1] = 0.f;
    }
}

// N pair records (slots q0 .. q0 + 2 N - 1) summed again for a tracer with a near source
// among them: the FP32 partial sum, added to (px, py, pz), of the sources at or beyond the
// near radius (the same operations as the main loop, so each of their pulls is the same), and
// the FP64 pull of each near source from its FP64 stage position (P: the stage's records of
// bodies n_exact.., src: source of each slot, null when slot q holds source q) and the
// tracer's (xt, yt, zt), added to k.  A zero FP64 separation makes the sum NaN, which removes
// the tracer as in the FP64 step.
template <int N>
__device__ __forceinline__ void near_span(const BodyPair* R, int q0, f2 XH, f2 XL, f2 YH, f2 YL, f2 ZH, f2 ZL,
                                          double xt, double yt, double zt, float inv_near, const Body* __restrict__ P,
                                          const int* __restrict__ src, f2& px, f2& py, f2& pz, double& kx,
                                          double& ky, double& kz) {
    for (int u = 0; u < N; ++u) {
        const BodyPair* r = R + u;
        const ulonglong2 q0v = *reinterpret_cast<const ulonglong2*>(r->hx);
        const ulonglong2 q1v = *reinterpret_cast<const ulonglong2*>(r->hz);
        const ulonglong2 q2v = *reinterpret_cast<const ulonglong2*>(r->lx);
        const f2 lz = *reinterpret_cast<const f2*>(r->lz);
        const f2 dX = add2(sub2(q0v.x, XH), sub2(q2v.x, XL));
        const f2 dY = add2(sub2(q0v.y, YH), sub2(q2v.y, YL));
        const f2 dZ = add2(sub2(q1v.x, ZH), sub2(lz, ZL));
        const f2 RR = fma2(dX, dX, fma2(dY, dY, mul2(dZ, dZ)));
        float r0, r1;
        f2_split(RR, r0, r1);
        const float i0 = rsqrt_approx(r0), i1 = rsqrt_approx(r1);
        const bool n0 = i0 > inv_near, n1 = i1 > inv_near;
        const f2 ri = f2_join(n0 ? 0.f : i0, n1 ? 0.f : i1);
        const f2 f = mul2(mul2(q1v.y, ri), mul2(ri, ri));
        px = fma2(f, dX, px); py = fma2(f, dY, py); pz = fma2(f, dZ, pz);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!(h ? n1 : n0)) continue;
            const int q = q0 + 2 * u + h;
            const Body p = P[src ? src[q] : q];
            const double ex = p.x - xt, ey = p.y - yt, ez = p.z - zt;
            const double rr = fma(ez, ez, fma(ey, ey, ex * ex));
            const double f64 = pull64(p.m, rr);
            kx = fma(f64, ex, kx); ky = fma(f64, ey, ky); kz = fma(f64, ez, kz);
        }
    }
}

// Kahan sums across the FP32 spans.  The compensated variant keeps both lanes (its
// float-float spans go to the FP64 acceleration instead, ff_total).  The FP32 forms add
// the span's two lanes (one rounding, against the 16 of each lane's plain sum) and carry one
// FP32 sum per axis: six registers fewer in the loop, which the dusty-ring dust kernel took
// from 8.18 to 8.00 ms.
template <bool F2> struct SpanAcc;
template <> struct SpanAcc<true> {
    f2 S = 0, C = 0;
    __device__ __forceinline__ void add(f2 v) { kahan2(S, C, v); }
    __device__ __forceinline__ double total() const { return f2_total(S, C); }
};
template <> struct SpanAcc<false> {
    float S = 0.f, C = 0.f;
    __device__ __forceinline__ void add(f2 v) {
        float a, b;
        f2_split(v, a, b);
        const float y = __fsub_rn(__fadd_rn(a, b), C);
        const float t = __fadd_rn(S, y);
        C = __fsub_rn(__fsub_rn(t, S), y);
        S = t;
    }
    __device__ __forceinline__ double total() const { return (double)S - (double)C; }
};

}  // namespace
}  // namespace ddx
