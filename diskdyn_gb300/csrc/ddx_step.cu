// RK4 step of the DiskDyn system on sm_103a.
//
// Reference behaviour (src/gpu_functions.cu:71-943, launch sequence src/grid.cu:693-752):
//   massive set : k1x = x; k2x = x + v dt/2; k2r = v + k1v dt/2; k3x = x + k2r dt/2;
//                 k3r = v + k2v dt/2; k4x = x + k3r dt; k4r = v + k3v dt;
//                 kNv = sum_j m_j (x_j - x_i)/r^3 at stage N;  x += dt/6 (v + 2k2r + 2k3r + k4r);
//                 v += dt/6 (k1v + 2k2v + 2k3v + k4v).
//   dust        : the same four stages per tracer, with the star term (gravity reduced by
//                 beta + beta_sw, PR + stellar-wind drag, optional Lorentz force) and the
//                 gravity of massive bodies 1..n_grav-1 taken at their stage positions.
//
// Because k2x depends only on x, v and k3x only on k1v, k4x only on k2v, the four massive
// force evaluations need two dependent passes: pass 1 evaluates A1 (at P1) and A2 (at P2),
// pass 2 evaluates A3 (at P3) and A4 (at P4).  The reference issues 4*(num+1)+4 launches
// per step with CAS atomics; here it is prepare + pass1 + pass2 + dust, deterministic, with
// no atomics.
#include "ddx_launch.cuh"
#include "ddx_internal.cuh"
#include "ddx_f32x2.cuh"

namespace ddx {

// ---------------------------------------------------------------------------------------
// Massive set
// ---------------------------------------------------------------------------------------

// FP32 source k = i - n_exact (body i >= n_exact) into its slot q of the pair records of a
// stage: half q & 1 of record q / 2.  The slots follow the sources' cell order when one
// was made for this step (ms.slot), else q = k.
__device__ __forceinline__ void store_pair_slot(MassiveScratch& ms, int stage, int k, const float4 h,
                                                const float4 l) {
    const int q = ms.slot ? ms.slot[k] : k;
    if (stage == 0 && ms.slot) ms.src[q] = k;     // the inverse, for the FP64 pulls of near sources
    BodyPair* r = ms.PP + (size_t)stage * ms.pcap + (q >> 1);
    const int u = q & 1;
    r->hx[u] = h.x; r->hy[u] = h.y; r->hz[u] = h.z; r->m[u] = h.w;
    r->lx[u] = l.x; r->ly[u] = l.y; r->lz[u] = l.z; r->pad[u] = 0.f;
    float2& pm = ms.PM[(size_t)stage * ms.pcap + (q >> 1)];
    if (u) pm.y = l.w; else pm.x = l.w;           // the mass's low part
}

// Zero-mass, far-away filler for the slots past the last FP32 source, so the dust kernel
// always processes whole spans of kPairSpan records.
__device__ __forceinline__ void store_pair_padding(MassiveScratch& ms, int n_src) {
    const int np = pair_count(n_src);
    for (int stage = 0; stage < 4; ++stage)
        for (int q = n_src; q < 2 * np; ++q) {
            BodyPair* r = ms.PP + (size_t)stage * ms.pcap + (q >> 1);
            const int k = q & 1;
            r->hx[k] = kFarAway; r->hy[k] = kFarAway; r->hz[k] = kFarAway; r->m[k] = 0.f;
            r->lx[k] = 0.f; r->ly[k] = 0.f; r->lz[k] = 0.f; r->pad[k] = 0.f;
            float2& pm = ms.PM[(size_t)stage * ms.pcap + (q >> 1)];
            if (k) pm.y = 0.f; else pm.x = 0.f;
        }
}

// The scratch as the kernels of a step see it: the pair slots in cell order only when the
// step orders its sources (else slot k holds source k).
static MassiveScratch slotted(const MassiveScratch& ms, const StepArgs& a) {
    MassiveScratch m = ms;
    if (!spatial_order_on(a)) m.slot = nullptr;
    return m;
}

// P1 = x, P2 = x + v dt/2 (src/gpu_functions.cu:90-99, 219-230).
__global__ void massive_prepare_kernel(ddx_state s, StepArgs a, MassiveScratch ms, int prec) {
    after_previous();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_grav) return;
    const double x = s.x[i], y = s.y[i], z = s.z[i], m = s.m[i];
    const double vx = s.vx[i], vy = s.vy[i], vz = s.vz[i];
    const double x2 = x + vx * a.dt2, y2 = y + vy * a.dt2, z2 = z + vz * a.dt2;
    ms.P[0 * ms.cap + i] = make_body(x, y, z, m);
    ms.P[1 * ms.cap + i] = make_body(x2, y2, z2, m);
    if (prec != DDX_PREC_FP64) {   // the FP32 records of the mixed and compensated dust kernels
        float4 h, l;
        split_hilo(x, h.x, l.x); split_hilo(y, h.y, l.y); split_hilo(z, h.z, l.z);
        split_hilo(m, h.w, l.w);
        ms.Phi[0 * ms.cap + i] = h; ms.Plo[0 * ms.cap + i] = l;
        if (i >= a.n_exact) store_pair_slot(ms, 0, i - a.n_exact, h, l);
        split_hilo(x2, h.x, l.x); split_hilo(y2, h.y, l.y); split_hilo(z2, h.z, l.z);
        ms.Phi[1 * ms.cap + i] = h; ms.Plo[1 * ms.cap + i] = l;
        if (i >= a.n_exact) store_pair_slot(ms, 1, i - a.n_exact, h, l);
        if (i == 0) store_pair_padding(ms, a.n_grav - a.n_exact);
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void kahan_add(float& S, float& C, float v) {
    const float y = v - C;
    const float t = S + y;
    C = (t - S) - y;
    S = t;
}

// Acceleration of body i from body j (FP64): m_j (x_j - x_i)/r^3; zero for coincident
// bodies, like the reference's f != 0 test (src/gpu_functions.cu:156-172).
__device__ __forceinline__ void pair64(const Body pi, const Body pj, double& ax,
                                       double& ay, double& az) {
    const double dX = pj.x - pi.x, dY = pj.y - pi.y, dZ = pj.z - pi.z;
    const double RR = dX * dX + dY * dY + dZ * dZ;
    if (positive64(RR)) {
        const double f = pull64(pj.m, RR);
        ax = fma(f, dX, ax); ay = fma(f, dY, ay); az = fma(f, dZ, az);
    }
}

// Same in FP32 on hi/lo split positions: the difference (hi_j - hi_i) + (lo_j - lo_i)
// keeps FP32 relative precision in the separation even when |x| >> |x_j - x_i|.  Returns
// true, adding nothing, when the source lies within the near radius (reciprocal distance
// above inv_near): the caller takes that pull in FP64.
__device__ __forceinline__ bool pair32(const float4 hi, const float4 li, const float4 hj,
                                       const float4 lj, float inv_near, float& fx, float& fy, float& fz) {
    const float dX = (hj.x - hi.x) + (lj.x - li.x);
    const float dY = (hj.y - hi.y) + (lj.y - li.y);
    const float dZ = (hj.z - hi.z) + (lj.z - li.z);
    const float RR = fmaf(dX, dX, fmaf(dY, dY, dZ * dZ));
    if (RR > 0.f) {
        const float ri = rsqrtf(RR);
        if (ri > inv_near) return true;
        const float f = hj.w * (ri * (ri * ri));
        fx = fmaf(f, dX, fx); fy = fmaf(f, dY, fy); fz = fmaf(f, dZ, fz);
    }
    return false;
}

// One warp per target body i, lanes stride over the sources, fixed-order butterfly
// reduction (deterministic).  Evaluates the accelerations at two stages sa, sb at once.
// In the mixed path the star's own acceleration and every pull of the star or a planet
// (sources 0..n_exact-1) stay FP64; the pulls of the planetesimals run in FP32 with a
// per-lane Kahan sum.
template <int PREC>
__device__ __forceinline__ void massive_two_stage_accel(const MassiveScratch& ms, int ng, int n_exact, float near_eta,
                                                         int i, int sa, int sb, double a_out[6]) {
    const int lane = threadIdx.x & 31;
    double ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
    const Body pa = ms.P[sa * ms.cap + i];
    const Body pb = ms.P[sb * ms.cap + i];
    if (PREC == DDX_PREC_FP64) {
        for (int j = lane; j < ng; j += 32) {
            if (j == i) continue;
            pair64(pa, ms.P[sa * ms.cap + j], ax, ay, az);
            pair64(pb, ms.P[sb * ms.cap + j], bx, by, bz);
        }
    } else {
        float Sa[3] = {0.f, 0.f, 0.f}, Ca[3] = {0.f, 0.f, 0.f};
        float Sb[3] = {0.f, 0.f, 0.f}, Cb[3] = {0.f, 0.f, 0.f};
        const float4 ha = ms.Phi[sa * ms.cap + i], la = ms.Plo[sa * ms.cap + i];
        const float4 hb = ms.Phi[sb * ms.cap + i], lb = ms.Plo[sb * ms.cap + i];
        const float inv_a = near_inv(near_eta, fmaxf(fabsf(ha.x), fmaxf(fabsf(ha.y), fabsf(ha.z))));
        const float inv_b = near_inv(near_eta, fmaxf(fabsf(hb.x), fmaxf(fabsf(hb.y), fabsf(hb.z))));
        for (int j = lane; j < ng; j += 32) {
            if (j == i) continue;
            if (i == 0 || j < n_exact) {
                pair64(pa, ms.P[sa * ms.cap + j], ax, ay, az);
                pair64(pb, ms.P[sb * ms.cap + j], bx, by, bz);
            } else {
                float fx = 0.f, fy = 0.f, fz = 0.f;
                if (pair32(ha, la, ms.Phi[sa * ms.cap + j], ms.Plo[sa * ms.cap + j], inv_a, fx, fy, fz))
                    pair64(pa, ms.P[sa * ms.cap + j], ax, ay, az);   // within the near radius: FP64
                kahan_add(Sa[0], Ca[0], fx); kahan_add(Sa[1], Ca[1], fy); kahan_add(Sa[2], Ca[2], fz);
                fx = fy = fz = 0.f;
                if (pair32(hb, lb, ms.Phi[sb * ms.cap + j], ms.Plo[sb * ms.cap + j], inv_b, fx, fy, fz))
                    pair64(pb, ms.P[sb * ms.cap + j], bx, by, bz);
                kahan_add(Sb[0], Cb[0], fx); kahan_add(Sb[1], Cb[1], fy); kahan_add(Sb[2], Cb[2], fz);
            }
        }
        ax += (double)Sa[0] - (double)Ca[0]; ay += (double)Sa[1] - (double)Ca[1];
        az += (double)Sa[2] - (double)Ca[2];
        bx += (double)Sb[0] - (double)Cb[0]; by += (double)Sb[1] - (double)Cb[1];
        bz += (double)Sb[2] - (double)Cb[2];
    }
    a_out[0] = warp_sum(ax); a_out[1] = warp_sum(ay); a_out[2] = warp_sum(az);
    a_out[3] = warp_sum(bx); a_out[4] = warp_sum(by); a_out[5] = warp_sum(bz);
}

__device__ __forceinline__ void store_stage_pos(MassiveScratch& ms, int stage, int i, double x,
                                                double y, double z, double m, int prec, int n_exact) {
    ms.P[stage * ms.cap + i] = make_body(x, y, z, m);
    if (prec != DDX_PREC_FP64) {
        float4 h, l;
        split_hilo(x, h.x, l.x); split_hilo(y, h.y, l.y); split_hilo(z, h.z, l.z);
        split_hilo(m, h.w, l.w);
        ms.Phi[stage * ms.cap + i] = h; ms.Plo[stage * ms.cap + i] = l;
        if (i >= n_exact) store_pair_slot(ms, stage, i - n_exact, h, l);
    }
}

// Pass 1: A1 at P1, A2 at P2; then R2, P3, R3, P4 for the target
// (src/gpu_functions.cu:219-230, 350-362, 482-493).
__device__ __forceinline__ void pass1_update(const ddx_state& s, const StepArgs& a, MassiveScratch& ms, int i,
                                             const double acc[6], int prec) {
    const int c = ms.cap;
    double* A = ms.A;
    double* R = ms.R;
    A[(0 * 3 + 0) * c + i] = acc[0]; A[(0 * 3 + 1) * c + i] = acc[1]; A[(0 * 3 + 2) * c + i] = acc[2];
    A[(1 * 3 + 0) * c + i] = acc[3]; A[(1 * 3 + 1) * c + i] = acc[4]; A[(1 * 3 + 2) * c + i] = acc[5];
    const double x = s.x[i], y = s.y[i], z = s.z[i], m = s.m[i];
    const double vx = s.vx[i], vy = s.vy[i], vz = s.vz[i];
    const double k2rx = vx + acc[0] * a.dt2, k2ry = vy + acc[1] * a.dt2, k2rz = vz + acc[2] * a.dt2;
    const double k3x = x + k2rx * a.dt2, k3y = y + k2ry * a.dt2, k3z = z + k2rz * a.dt2;
    const double k3rx = vx + acc[3] * a.dt2, k3ry = vy + acc[4] * a.dt2, k3rz = vz + acc[5] * a.dt2;
    const double k4x = x + k3rx * a.dt, k4y = y + k3ry * a.dt, k4z = z + k3rz * a.dt;
    R[(0 * 3 + 0) * c + i] = k2rx; R[(0 * 3 + 1) * c + i] = k2ry; R[(0 * 3 + 2) * c + i] = k2rz;
    R[(1 * 3 + 0) * c + i] = k3rx; R[(1 * 3 + 1) * c + i] = k3ry; R[(1 * 3 + 2) * c + i] = k3rz;
    store_stage_pos(ms, 2, i, k3x, k3y, k3z, m, prec, a.n_exact);
    store_stage_pos(ms, 3, i, k4x, k4y, k4z, m, prec, a.n_exact);
}

// PREC: the arithmetic of the accelerations; STORE: the precision whose stage records
// pass 1 writes (the compensated step integrates the massive set in FP64 and writes the
// FP32 records its dust kernel reads).
template <int PREC, int STORE = PREC>
__global__ void massive_pass1_kernel(ddx_state s, StepArgs a, MassiveScratch ms) {
    after_previous();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= a.n_grav) return;  // warp-uniform
    double acc[6];
    massive_two_stage_accel<PREC>(ms, a.n_grav, a.n_exact, a.near_eta, i, 0, 1, acc);
    if ((threadIdx.x & 31) != 0) return;
    pass1_update(s, a, ms, i, acc, STORE);
}

// Pass 2: A3 at P3, A4 at P4; R4; final combination (src/gpu_functions.cu:613-625).
// Reads only stage records of other bodies, so updating x, v of the target is safe.
__device__ __forceinline__ void pass2_update(const ddx_state& s, const StepArgs& a, MassiveScratch& ms, int i,
                                             const double acc[6]) {
    const int c = ms.cap;
    double* A = ms.A;
    const double* R = ms.R;
    A[(2 * 3 + 0) * c + i] = acc[0]; A[(2 * 3 + 1) * c + i] = acc[1]; A[(2 * 3 + 2) * c + i] = acc[2];
    A[(3 * 3 + 0) * c + i] = acc[3]; A[(3 * 3 + 1) * c + i] = acc[4]; A[(3 * 3 + 2) * c + i] = acc[5];
    const double vx = s.vx[i], vy = s.vy[i], vz = s.vz[i];
    const double k4rx = vx + acc[0] * a.dt, k4ry = vy + acc[1] * a.dt, k4rz = vz + acc[2] * a.dt;
    const double dt = a.dt6;
    s.x[i] += dt * (vx + 2.0 * R[(0 * 3 + 0) * c + i] + 2.0 * R[(1 * 3 + 0) * c + i] + k4rx);
    s.y[i] += dt * (vy + 2.0 * R[(0 * 3 + 1) * c + i] + 2.0 * R[(1 * 3 + 1) * c + i] + k4ry);
    s.z[i] += dt * (vz + 2.0 * R[(0 * 3 + 2) * c + i] + 2.0 * R[(1 * 3 + 2) * c + i] + k4rz);
    s.vx[i] += dt * (A[(0 * 3 + 0) * c + i] + 2.0 * A[(1 * 3 + 0) * c + i] + 2.0 * acc[0] + acc[3]);
    s.vy[i] += dt * (A[(0 * 3 + 1) * c + i] + 2.0 * A[(1 * 3 + 1) * c + i] + 2.0 * acc[1] + acc[4]);
    s.vz[i] += dt * (A[(0 * 3 + 2) * c + i] + 2.0 * A[(1 * 3 + 2) * c + i] + 2.0 * acc[2] + acc[5]);
}

template <int PREC>
__global__ void massive_pass2_kernel(ddx_state s, StepArgs a, MassiveScratch ms) {
    after_previous();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= a.n_grav) return;
    double acc[6];
    massive_two_stage_accel<PREC>(ms, a.n_grav, a.n_exact, a.near_eta, i, 2, 3, acc);
    if ((threadIdx.x & 31) != 0) return;
    pass2_update(s, a, ms, i, acc);
}

// ---------------------------------------------------------------------------------------
// Mixed massive passes over source slices
// ---------------------------------------------------------------------------------------
// A few thousand targets leave most of the GPU idle when one warp serves one target, so
// the FP32 pulls of the planetesimals are split over source slices: block (target group of
// kSliceThreads, slice k, one of the pass's two stages) stages the slice's pair records in
// shared memory, every thread (two targets) reads each record at once (broadcast) and
// works on both sources of a record with one f32x2 instruction, in plain sums over spans
// of kPairSpan records with a Kahan sum across spans (the dust kernel's scheme).  A
// target's own slot gives RR = 0 and is masked.  The star (target 0) takes the
// planetesimals' pulls in FP64, in an extra row of blocks that spread each slice over a
// whole block (a fixed-order tree sum).  massive_gather_kernel then adds the slices (a
// fixed lane order: deterministic), adds the FP64 pulls of bodies 0..n_exact-1 and applies
// the pass's update.
constexpr int kSliceTile = 256;       // pair records per stage staged at once (16 KiB)
constexpr int kMaxSlices = 64;

__device__ __forceinline__ void pair_f2(const BodyPair& r, f2 XH, f2 XL, f2 YH, f2 YL, f2 ZH, f2 ZL, f2& px,
                                        f2& py, f2& pz) {
    const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(r.hx);   // hx, hy
    const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(r.hz);   // hz, m
    const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(r.lx);   // lx, ly
    const f2 lz = *reinterpret_cast<const f2*>(r.lz);
    const f2 dX = add2(sub2(q0.x, XH), sub2(q2.x, XL));
    const f2 dY = add2(sub2(q0.y, YH), sub2(q2.y, YL));
    const f2 dZ = add2(sub2(q1.x, ZH), sub2(lz, ZL));
    const f2 RR = fma2(dX, dX, fma2(dY, dY, mul2(dZ, dZ)));
    float r0, r1;
    f2_split(RR, r0, r1);
    const f2 ri = f2_join(r0 > 0.f ? rsqrt_approx(r0) : 0.f, r1 > 0.f ? rsqrt_approx(r1) : 0.f);
    const f2 f = mul2(mul2(q1.y, ri), mul2(ri, ri));
    px = fma2(f, dX, px); py = fma2(f, dY, py); pz = fma2(f, dZ, pz);
}

// pair_f2 that also raises mx to the larger reciprocal distance of the two sources (0 for
// a coincident source, the target's own slot included, so it never counts as near).
__device__ __forceinline__ void pair_f2_max(const BodyPair& r, f2 XH, f2 XL, f2 YH, f2 YL, f2 ZH, f2 ZL, f2& px,
                                            f2& py, f2& pz, float& mx) {
    const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(r.hx);   // hx, hy
    const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(r.hz);   // hz, m
    const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(r.lx);   // lx, ly
    const f2 lz = *reinterpret_cast<const f2*>(r.lz);
    const f2 dX = add2(sub2(q0.x, XH), sub2(q2.x, XL));
    const f2 dY = add2(sub2(q0.y, YH), sub2(q2.y, YL));
    const f2 dZ = add2(sub2(q1.x, ZH), sub2(lz, ZL));
    const f2 RR = fma2(dX, dX, fma2(dY, dY, mul2(dZ, dZ)));
    float r0, r1;
    f2_split(RR, r0, r1);
    const float i0 = r0 > 0.f ? rsqrt_approx(r0) : 0.f, i1 = r1 > 0.f ? rsqrt_approx(r1) : 0.f;
    mx = fmax3(mx, i0, i1);
    const f2 ri = f2_join(i0, i1);
    const f2 f = mul2(mul2(q1.y, ri), mul2(ri, ri));
    px = fma2(f, dX, px); py = fma2(f, dY, py); pz = fma2(f, dZ, pz);
}

// One span of kPairSpan pair records (slots q0 ..) summed again for a target with a source
// within the near radius (reciprocal FP32 distance above inv_near): the FP32 partial sum of
// the other sources, with the same operations as pair_f2_max, and the FP64 pull of each near
// source from the FP64 stage records (P: bodies n_exact.. of the stage; src: source of each
// slot, null when slot q holds source q) on the target's FP64 stage position pt, added to n.
// The target's own slot is never near (its reciprocal distance is 0).
__device__ __forceinline__ void near_span_massive(const BodyPair* R, int q0, f2 XH, f2 XL, f2 YH, f2 YL, f2 ZH,
                                                  f2 ZL, float inv_near, const Body pt, const Body* __restrict__ P,
                                                  const int* __restrict__ src, f2& px, f2& py, f2& pz,
                                                  double n[3]) {
    px = 0; py = 0; pz = 0;
    for (int u = 0; u < kPairSpan; ++u) {
        const BodyPair& r = R[u];
        const ulonglong2 q0v = *reinterpret_cast<const ulonglong2*>(r.hx);
        const ulonglong2 q1v = *reinterpret_cast<const ulonglong2*>(r.hz);
        const ulonglong2 q2v = *reinterpret_cast<const ulonglong2*>(r.lx);
        const f2 lz = *reinterpret_cast<const f2*>(r.lz);
        const f2 dX = add2(sub2(q0v.x, XH), sub2(q2v.x, XL));
        const f2 dY = add2(sub2(q0v.y, YH), sub2(q2v.y, YL));
        const f2 dZ = add2(sub2(q1v.x, ZH), sub2(lz, ZL));
        const f2 RR = fma2(dX, dX, fma2(dY, dY, mul2(dZ, dZ)));
        float r0, r1;
        f2_split(RR, r0, r1);
        const float i0 = r0 > 0.f ? rsqrt_approx(r0) : 0.f, i1 = r1 > 0.f ? rsqrt_approx(r1) : 0.f;
        const bool n0 = i0 > inv_near, n1 = i1 > inv_near;
        const f2 ri = f2_join(n0 ? 0.f : i0, n1 ? 0.f : i1);
        const f2 f = mul2(mul2(q1v.y, ri), mul2(ri, ri));
        px = fma2(f, dX, px); py = fma2(f, dY, py); pz = fma2(f, dZ, pz);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!(h ? n1 : n0)) continue;
            const int q = q0 + 2 * u + h;
            pair64(pt, P[src ? src[q] : q], n[0], n[1], n[2]);
        }
    }
}

// Threads of a slice block.  A thread takes two targets at one stage, which share every
// record read: broadcasting a record's 56 bytes to 32 lanes costs the shared-memory pipe 14
// cycles, a target's FP32 operations on it 9 (4,099 bodies: 38 us a pass with one target at
// both stages per thread, 26 us with two at one).
constexpr int kSliceWorkers = kSliceThreads / 2;

// Deterministic block sum of v (fixed tree order); the result in thread 0.
__device__ __forceinline__ double block_sum(double v, double* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int o = kSliceWorkers / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

// One target of a slice block.
struct SliceTarget {
    f2 XH, XL, YH, YL, ZH, ZL;
    f2 S[3], C[3];             // Kahan sums of the spans
    double N[3];               // FP64 pulls of near sources, added to the slice's total
    float inv_near;
};

__global__ void __launch_bounds__(kSliceWorkers)
massive_slice_kernel(StepArgs a, MassiveScratch ms, int sa, int per, int np, double* __restrict__ part) {
    after_previous();
    __shared__ __align__(16) BodyPair tile[kSliceTile];
    const int k = blockIdx.y, st = sa + blockIdx.z;
    const int n_src = a.n_grav - a.n_exact;
    const int npairs = pair_count(n_src);
    const int r0 = k * per, r1 = min(r0 + per, npairs);
    const int c = ms.cap;
    double* const o = part + ((size_t)k * 6 + 3 * blockIdx.z) * np;
    if (blockIdx.x == gridDim.x - 1) {
        // the star's row: the whole block takes the slice's planetesimals in FP64
        const Body ps = ms.P[st * c];
        double d[3] = {0.0, 0.0, 0.0};
        const int q1 = min(2 * r1, n_src);
        for (int q = 2 * r0 + threadIdx.x; q < q1; q += kSliceWorkers)
            pair64(ps, ms.P[st * c + a.n_exact + q], d[0], d[1], d[2]);
        double* red = reinterpret_cast<double*>(&tile[0]);        // 1 KiB of the tile space
        for (int q = 0; q < 3; ++q) {
            const double t = block_sum(d[q], red);
            if (threadIdx.x == 0) o[(size_t)q * np] = t;
        }
        return;
    }
    const int i0 = blockIdx.x * kSliceThreads + threadIdx.x;      // targets i0 and i0 + kSliceWorkers
    SliceTarget t[2];
    bool any = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = i0 + q * kSliceWorkers;
        const bool active = i > 0 && i < a.n_grav;                // the star has its own row
        any = any || active;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
        if (active) { h = ms.Phi[st * c + i]; l = ms.Plo[st * c + i]; }
        t[q].XH = f2_dup(h.x); t[q].XL = f2_dup(l.x); t[q].YH = f2_dup(h.y); t[q].YL = f2_dup(l.y);
        t[q].ZH = f2_dup(h.z); t[q].ZL = f2_dup(l.z);
        // a thread without a target finds nothing near
        t[q].inv_near = active ? near_inv(a.near_eta, fmaxf(fabsf(h.x), fmaxf(fabsf(h.y), fabsf(h.z)))) : INFINITY;
#pragma unroll
        for (int d = 0; d < 3; ++d) t[q].S[d] = t[q].C[d] = 0, t[q].N[d] = 0.0;
    }
    for (int t0 = r0; t0 < r1; t0 += kSliceTile) {
        const int cnt = min(kSliceTile, r1 - t0);          // a multiple of kPairSpan
        __syncthreads();                                   // the previous tile is consumed
        const uint4* g = reinterpret_cast<const uint4*>(ms.PP + (size_t)st * ms.pcap + t0);
        for (int w = threadIdx.x; w < cnt * 4; w += kSliceWorkers) reinterpret_cast<uint4*>(tile)[w] = g[w];
        __syncthreads();
        if (!any) continue;
        for (int u0 = 0; u0 < cnt; u0 += kPairSpan) {
            f2 x[2] = {0, 0}, y[2] = {0, 0}, z[2] = {0, 0};
            float mx[2] = {0.f, 0.f};
#pragma unroll 4
            for (int u = 0; u < kPairSpan; ++u)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    pair_f2_max(tile[u0 + u], t[q].XH, t[q].XL, t[q].YH, t[q].YL, t[q].ZH, t[q].ZL, x[q], y[q], z[q],
                                mx[q]);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (mx[q] > t[q].inv_near)   // rare: a source of this span within the near radius
                    near_span_massive(&tile[u0], 2 * (t0 + u0), t[q].XH, t[q].XL, t[q].YH, t[q].YL, t[q].ZH, t[q].ZL,
                                      t[q].inv_near, ms.P[st * c + i0 + q * kSliceWorkers],
                                      ms.P + (size_t)st * c + a.n_exact, ms.slot ? ms.src : nullptr, x[q], y[q], z[q],
                                      t[q].N);
                kahan2(t[q].S[0], t[q].C[0], x[q]); kahan2(t[q].S[1], t[q].C[1], y[q]); kahan2(t[q].S[2], t[q].C[2], z[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = i0 + q * kSliceWorkers;
        if (!(i > 0 && i < a.n_grav)) continue;
#pragma unroll
        for (int d = 0; d < 3; ++d) o[(size_t)d * np + i] = f2_total(t[q].S[d], t[q].C[d]) + t[q].N[d];
    }
}

// 32 targets per block of 8 warps, a target per lane (coalesced reads of the slice sums).  Warp
// w adds slices w, w + 8, ... , the warps' sums are added in warp order (the same on every
// run), two warps add the FP64 pulls of bodies 0..n_exact-1 at the pass's two stages, and
// warp 0 applies the pass's update (4,099 bodies: 25 us with a warp per target's slices and
// every FP64 pull in warp 0, 9 us so).
constexpr int kGatherTargets = 32;
constexpr int kGatherThreads = 256;

// n_pull: the bodies 0..n_pull-1 whose FP64 pulls the sums leave out; PREC: the precision whose
// stage records pass 1 writes.
template <int PASS, int PREC>
__global__ void __launch_bounds__(kGatherThreads)
massive_gather_kernel(ddx_state s, StepArgs a, MassiveScratch ms, int n_pull, int slices, int np,
                      const double* __restrict__ part) {
    after_previous();
    constexpr int kWarps = kGatherThreads / 32;
    __shared__ double sums[kWarps][6][kGatherTargets];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kGatherTargets + lane;
    double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (i < a.n_grav)
        for (int k = warp; k < slices; k += kWarps)
#pragma unroll
            for (int q = 0; q < 6; ++q) acc[q] += part[((size_t)k * 6 + q) * np + i];
#pragma unroll
    for (int q = 0; q < 6; ++q) sums[warp][q][lane] = acc[q];
    __syncthreads();
    if (warp < 6) {
        double v = sums[0][warp][lane];
        for (int k = 1; k < kWarps; ++k) v += sums[k][warp][lane];
        sums[0][warp][lane] = v;
    }
    __syncthreads();
    if (warp >= 2) return;
    const int c = ms.cap;
    const int st = (PASS == 1 ? 0 : 2) + warp;
    if (i < a.n_grav) {
        double d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) d[q] = sums[0][3 * warp + q][lane];
        const Body p = ms.P[st * c + i];
        for (int j = 0; j < n_pull && j < a.n_grav; ++j)
            if (j != i) pair64(p, ms.P[st * c + j], d[0], d[1], d[2]);
#pragma unroll
        for (int q = 0; q < 3; ++q) sums[0][3 * warp + q][lane] = d[q];
    }
    asm volatile("bar.sync 1, 64;" ::: "memory");          // the two warps
    if (warp != 0 || i >= a.n_grav) return;
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = sums[0][q][lane];
    if (PASS == 1) pass1_update(s, a, ms, i, acc, PREC);
    else pass2_update(s, a, ms, i, acc);
}

// ---------------------------------------------------------------------------------------
// FP64 all-pairs over pairs of bodies
// ---------------------------------------------------------------------------------------
// FP64 issue bounds the all-pairs sums, and a pair's separation and r^-3 serve both of its bodies:
// 20 FP64 operations a pair instead of 32.  A block takes two groups I < J of kPairBlock bodies at one
// of the pass's two stages.  A thread holds a body of I; a warp goes through 32 bodies of J
// in 32 steps, lane l taking body (l + step) mod 32, and the sums of J's bodies move one lane
// with each step, so each ends where it began.  The four warps' sums are added in order.  A
// block I = J takes every body's pulls on its own.  Every block writes sums of its own, row J for the
// bodies of I and row I for those of J, which massive_gather_kernel adds in row order: the same
// on every run.  4,099 bodies: 1460 us for both passes of a step, 2330 us with a warp per body.
constexpr int kPairBlock = 128;
// Bodies from which on it pays (FP64 steps of 2,000 tracers, us with / without: 1,503 bodies 1286 / 1248,
// 2,003 1576 / 1787; below, the blocks are too few), and up to which the sums fit into the scratch that
// every step keeps for the slices (MassiveScratch::part: 7.5 MB; 8,192 bodies would take 25 MB).  Beyond, a
// warp per body as before; larger scratch has not been measured.
constexpr int kPairsFrom = 1664, kPairsTo = 34 * kPairBlock;

__global__ void __launch_bounds__(kPairBlock)
massive_pairs_kernel(StepArgs a, MassiveScratch ms, int sa, int np, double* __restrict__ part) {
    after_previous();
    __shared__ Body src[kPairBlock];
    __shared__ double red[kPairBlock / 32][3][32];
    // blockIdx.x = J (J + 1) / 2 + I, I <= J
    int J = (int)((sqrtf(8.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
    while ((J + 1) * (J + 2) / 2 <= (int)blockIdx.x) ++J;
    while (J * (J + 1) / 2 > (int)blockIdx.x) --J;
    const int I = (int)blockIdx.x - J * (J + 1) / 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Body* const P = ms.P + (size_t)(sa + blockIdx.y) * ms.cap;
    // past the last body, and for one without a position (NaN, a pair of which pair64 leaves out): no mass, and so
    // far away that its pulls are 0 both ways
    auto body = [&](int k) {
        const Body none = make_body(1e150, 1e150, 1e150, 0.0);
        const Body b = k < a.n_grav ? P[k] : none;
        return b.x == b.x && b.y == b.y && b.z == b.z ? b : none;
    };
    const int i = I * kPairBlock + threadIdx.x, j0 = J * kPairBlock;
    const Body p = body(i);
    src[threadIdx.x] = body(j0 + threadIdx.x);
    __syncthreads();
    double* const rowI = part + ((size_t)I * 6 + 3 * blockIdx.y) * np;
    double* const rowJ = part + ((size_t)J * 6 + 3 * blockIdx.y) * np;
    double acc[3] = {0.0, 0.0, 0.0};
    if (I == J) {
#pragma unroll 4
        for (int k = 0; k < kPairBlock; ++k)
            if (k != (int)threadIdx.x) pair64(p, src[k], acc[0], acc[1], acc[2]);
    } else {
        for (int j = 0; j < kPairBlock; j += 32) {
            double b[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
            for (int step = 0; step < 32; ++step) {
                const Body q = src[j + ((lane + step) & 31)];
                const double dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
                const double RR = dx * dx + dy * dy + dz * dz;
                const double f = positive64(RR) ? pull64(1.0, RR) : 0.0, fi = f * q.m, fj = f * p.m;
                acc[0] = fma(fi, dx, acc[0]); acc[1] = fma(fi, dy, acc[1]); acc[2] = fma(fi, dz, acc[2]);
                b[0] = fma(-fj, dx, b[0]); b[1] = fma(-fj, dy, b[1]); b[2] = fma(-fj, dz, b[2]);
#pragma unroll
                for (int c = 0; c < 3; ++c) b[c] = __shfl_sync(0xffffffffu, b[c], (lane + 1) & 31);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) red[warp][c][lane] = b[c];
            __syncthreads();
            if (warp < 3) {
                double t = red[0][warp][lane];
                for (int w = 1; w < kPairBlock / 32; ++w) t += red[w][warp][lane];
                rowI[(size_t)warp * np + j0 + j + lane] = t;
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) rowJ[(size_t)c * np + i] = acc[c];
}

// ---------------------------------------------------------------------------------------
// Dust tracers
// ---------------------------------------------------------------------------------------

// Variants of the dust kernel.
enum DustVariant {
    kDustFP64Exact = 0,  // reference arithmetic expression for expression: m/RR/sqrt(RR)
    kDustFP64 = 1,       // FP64 with rsqrt
};

// Small blocks spread the tracers evenly: FP64 issue bounds the kernel, so the SM with the most
// warps sets its time, and 65,536 tracers in blocks of 256 put 512 of them on two thirds of the
// SMs and 256 on the rest (4,096 planetesimals: 41.1 ms in blocks of 256, 37.5 ms so).
constexpr int kDustThreads = 64;
constexpr int kDustTile = 256;     // sources per shared-memory tile (8 KiB)
// Four lanes share a tracer of the FP64 kernel while that pays for repeating its star term: one
// thread's chain of sources leaves the FP64 pipe waiting (us a step with one / four lanes: star and
// 8 planets, 1,000 tracers 56 / 41, 16,384 tracers 57 / 75; 200 planetesimals, 2,000 tracers
// 518 / 172, 65,536 tracers 1819 / 1750; 4,096 planetesimals, 65,536 tracers 37500 / 34000; 300
// planetesimals, 262,144 tracers 9540 / 10010).
constexpr int kLanesMinSources = 128, kLanesFew = 4864, kLanesMany = 131072;

// FP64 gravity of massive bodies 1..n_grav-1 at stage `st` on every tracer of the block.
// Sources are staged through shared memory tile by tile; every thread of the block takes
// part in the loads and barriers whether or not its tracer is still alive.
// kDustFP64 sums source j into partial sum j mod 4, and adds the four in pairs: with T = 4 lanes
// per tracer each lane has one of them (the butterfly gives every lane the same bits as T = 1).
// Returns false (for the calling thread) on an exact coincidence with a body.
template <int VAR, int T>
__device__ __forceinline__ bool dust_perturb(const MassiveScratch& ms, int ng, int st, bool alive,
                                             double xt, double yt, double zt, double& kx,
                                             double& ky, double& kz, unsigned char* smem) {
    const int nsrc = ng - 1;
    bool ok = true;
    constexpr int kSums = VAR == kDustFP64 && T == 1 ? 4 : 1;
    double s[kSums][3];
#pragma unroll
    for (int q = 0; q < kSums; ++q) s[q][0] = s[q][1] = s[q][2] = 0.0;
    Body* sP = reinterpret_cast<Body*>(smem);
    for (int base = 0; base < nsrc; base += kDustTile) {
        const int cnt = min(kDustTile, nsrc - base);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += blockDim.x)
            sP[k] = ms.P[st * ms.cap + 1 + base + k];
        __syncthreads();
        if (!alive || !ok) continue;
        if (VAR == kDustFP64Exact) {
            // src/gpu_functions.cu:722-735, in order, with its early exit.
            for (int k = 0; k < cnt; ++k) {
                const Body p = sP[k];
                const double dx = xt - p.x, dy = yt - p.y, dz = zt - p.z;
                const double RR = dx * dx + dy * dy + dz * dz;
                if (RR == 0) { ok = false; break; }
                const double f = p.m / RR / sqrt(RR);
                kx += -f * dx; ky += -f * dy; kz += -f * dz;
            }
        } else {
            auto add = [&](int k, double (&a)[3]) {
                const Body p = sP[k];
                const double dx = p.x - xt, dy = p.y - yt, dz = p.z - zt;
                const double f = pull64(p.m, fma(dz, dz, fma(dy, dy, dx * dx)));
                a[0] = fma(f, dx, a[0]); a[1] = fma(f, dy, a[1]); a[2] = fma(f, dz, a[2]);
            };
            if (T == 1) {
                int k = 0;
                for (; k + 4 <= cnt; k += 4)
#pragma unroll
                    for (int q = 0; q < 4; ++q) add(k + q, s[q % kSums]);
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (k + q < cnt) add(k + q, s[q % kSums]);
            } else {
#pragma unroll 4
                for (int k = threadIdx.x & (T - 1); k < cnt; k += T) add(k, s[0]);
            }
        }
    }
    if (VAR == kDustFP64) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double t = s[0][c];
            if (T == 1) {
                t = (s[0][c] + s[1 % kSums][c]) + (s[2 % kSums][c] + s[3 % kSums][c]);
            } else {
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                t += __shfl_xor_sync(0xffffffffu, t, 2);
            }
            (c == 0 ? kx : c == 1 ? ky : kz) += t;
        }
        if (alive && !(finite64(kx) && finite64(ky) && finite64(kz))) ok = false;
    }
    return ok;
}

// Full RK4 of one dust tracer per thread, or per T = 4 lanes (src/gpu_functions.cu:627-943).
template <int VAR, int T>
__global__ void __launch_bounds__(kDustThreads, VAR == kDustFP64 ? 8 : 1)
dust_rk4_kernel(ddx_state s, StepArgs a, MassiveScratch ms, const SizeBin* __restrict__ bins) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / T;
    const int ng = a.n_grav;
    const int t = ng + i;
    bool alive = false;
    double x = 0, y = 0, z = 0, vx = 0, vy = 0, vz = 0, m = 1.0;
    float bet = 0.f, betsw = 0.f, qe = 0.f;
    if (i < a.n_dust) {
        alive = (s.N[t] != 0.0);
        if (alive) {
            x = s.x[t]; y = s.y[t]; z = s.z[t];
            vx = s.vx[t]; vy = s.vy[t]; vz = s.vz[t];
            m = s.m[t];
            const int id = s.id[t];
            if (id >= 0 && id < a.n_grid) {
                const SizeBin b = bins[id];
                bet = b.beta; betsw = b.betasw; qe = b.q;
            }
        }
    }
    const StarCoef star = star_coef(ms.P[0].m, bet, betsw, qe, m, a);
    const double dt = a.dt, dt2 = a.dt / 2.0, dt6 = a.dt / 6.0;
    double k1vx = 0, k1vy = 0, k1vz = 0, k2vx = 0, k2vy = 0, k2vz = 0;
    double k3vx = 0, k3vy = 0, k3vz = 0, k4vx = 0, k4vy = 0, k4vz = 0;
    double k2rx = 0, k2ry = 0, k2rz = 0, k3rx = 0, k3ry = 0, k3rz = 0;
    double k4rx = 0, k4ry = 0, k4rz = 0;
    int removed = 0;  // 1: sublimated (stage kept in removed_stage), 2: coincidence
    int removed_stage = -1;

#pragma unroll 1
    for (int st = 0; st < 4; ++st) {
        double xt, yt, zt, rx, ry, rz;
        if (st == 0)      { xt = x; yt = y; zt = z; rx = vx; ry = vy; rz = vz; }
        else if (st == 1) {
            k2rx = vx + k1vx * dt2; k2ry = vy + k1vy * dt2; k2rz = vz + k1vz * dt2;
            xt = x + vx * dt2; yt = y + vy * dt2; zt = z + vz * dt2;
            rx = k2rx; ry = k2ry; rz = k2rz;
        } else if (st == 2) {
            k3rx = vx + k2vx * dt2; k3ry = vy + k2vy * dt2; k3rz = vz + k2vz * dt2;
            xt = x + k2rx * dt2; yt = y + k2ry * dt2; zt = z + k2rz * dt2;
            rx = k3rx; ry = k3ry; rz = k3rz;
        } else {
            k4rx = vx + k3vx * dt; k4ry = vy + k3vy * dt; k4rz = vz + k3vz * dt;
            xt = x + k3rx * dt; yt = y + k3ry * dt; zt = z + k3rz * dt;
            rx = k4rx; ry = k4ry; rz = k4rz;
        }
        double kx = 0, ky = 0, kz = 0;
        if (alive) {
            const Body ps = ms.P[st * ms.cap + 0];
            const double dx = xt - ps.x, dy = yt - ps.y, dz = zt - ps.z;
            const bool outside = VAR == kDustFP64Exact
                                     ? star_term(dx, dy, dz, rx, ry, rz, ps.m, bet, betsw, qe, m, a, kx, ky, kz)
                                     : star_term(dx, dy, dz, rx, ry, rz, star, a, kx, ky, kz);
            if (!outside) { alive = false; removed = 1; removed_stage = st; }
        }
        if (!dust_perturb<VAR, T>(ms, ng, st, alive, xt, yt, zt, kx, ky, kz, smem)) {
            alive = false; removed = 2; removed_stage = st;
        }
        if (st == 0)      { k1vx = kx; k1vy = ky; k1vz = kz; }
        else if (st == 1) { k2vx = kx; k2vy = ky; k2vz = kz; }
        else if (st == 2) { k3vx = kx; k3vy = ky; k3vz = kz; }
        else              { k4vx = kx; k4vy = ky; k4vz = kz; }
    }
    if (i >= a.n_dust || (T > 1 && (threadIdx.x & (T - 1)))) return;
    if (removed) {
        // src/gpu_functions.cu:878 zeroes N[i] (i is the dust-relative index) on a stage-4
        // sublimation and leaves the grain alive; DDX_MODE_REFERENCE reproduces it.
        if (removed == 1 && removed_stage == 3 && a.mode == DDX_MODE_REFERENCE) s.N[i] = 0;
        else s.N[t] = 0;
        return;
    }
    if (!alive) return;
    x += dt6 * (vx + 2.0 * (k2rx + k3rx) + k4rx);
    y += dt6 * (vy + 2.0 * (k2ry + k3ry) + k4ry);
    z += dt6 * (vz + 2.0 * (k2rz + k3rz) + k4rz);
    vx += dt6 * (k1vx + 2.0 * (k2vx + k3vx) + k4vx);
    vy += dt6 * (k1vy + 2.0 * (k2vy + k3vy) + k4vy);
    vz += dt6 * (k1vz + 2.0 * (k2vz + k3vz) + k4vz);
    s.x[t] = x; s.y[t] = y; s.z[t] = z;
    s.vx[t] = vx; s.vy[t] = vy; s.vz[t] = vz;
}

// ---------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------

cudaError_t launch_massive_prepare(const ddx_state& s, const StepArgs& a, MassiveScratch& ms,
                                   int precision, cudaStream_t st) {
    // the FP32 sources' pair slots in cell order, from their positions at the start of the step
    const bool ordered = precision != DDX_PREC_FP64 && ms.slot && spatial_order_on(a);
    if (ordered) {
        const cudaError_t e =
            order_bodies(s, a.n_exact, a.n_grav - a.n_exact, false, ms.src_order, nullptr, ms.slot,
                         precision == DDX_PREC_MIXED, st);
        if (e != cudaSuccess) return e;
    }
    const int threads = 128;
    const int blocks = (a.n_grav + threads - 1) / threads;
    launch_with(ordered, massive_prepare_kernel, blocks, threads, 0, st, s, a, slotted(ms, a), precision);
    return cudaGetLastError();
}

int sm_count() {
    static int cached[128] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 128) return 152;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 152;
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {
// The sliced mixed pass: slice sums, then their gather with the pass's update.
// Slice sums are stored [slice][component][np] with np = n_grav rounded up to a block.
int slice_stride(int n_grav) { return (n_grav + kSliceThreads - 1) / kSliceThreads * kSliceThreads; }

bool sliced_fits(const StepArgs& a, const MassiveScratch& ms) {
    return ms.part && ms.part_words >= (long long)massive_slices(a.n_grav, a.n_exact) * 6 * slice_stride(a.n_grav);
}

template <int PASS>
cudaError_t launch_sliced(const ddx_state& s, const StepArgs& a, MassiveScratch& ms, cudaStream_t st) {
    const int spans = pair_count(a.n_grav - a.n_exact) / kPairSpan;
    const int S = spans > 0 ? massive_slices(a.n_grav, a.n_exact) : 0;    // no planetesimals: no slices
    const int np = slice_stride(a.n_grav);
    if (S > 0) {
        const int per = (spans + S - 1) / S * kPairSpan;
        const dim3 grid((a.n_grav + kSliceThreads - 1) / kSliceThreads + 1, S, 2);   // + the star's row; two stages
        launch_with(a.n_grav <= kOverlapPasses, massive_slice_kernel, grid, kSliceWorkers, 0, st, a, slotted(ms, a),
                    PASS == 1 ? 0 : 2, per, np, ms.part);
    }
    launch_after(massive_gather_kernel<PASS, DDX_PREC_MIXED>, (a.n_grav + kGatherTargets - 1) / kGatherTargets,
                 kGatherThreads, 0, st, s, a, slotted(ms, a), a.n_exact, S, np, ms.part);
    return cudaGetLastError();
}

// The FP64 all-pairs pass over pairs of bodies (FP64 and compensated steps).
bool pairs_fit(const StepArgs& a, const MassiveScratch& ms) {
    const long long nb = (a.n_grav + kPairBlock - 1) / kPairBlock;
    return a.n_grav >= kPairsFrom && a.n_grav <= kPairsTo && ms.part && ms.part_words >= 6 * nb * nb * kPairBlock;
}

template <int PASS>
cudaError_t launch_pairs(const ddx_state& s, const StepArgs& a, MassiveScratch& ms, int precision, cudaStream_t st) {
    const int nb = (a.n_grav + kPairBlock - 1) / kPairBlock, np = nb * kPairBlock;
    launch_first(massive_pairs_kernel, dim3(nb * (nb + 1) / 2, 2), kPairBlock, 0, st, a, ms, PASS == 1 ? 0 : 2, np, ms.part);
    launch_after(precision == DDX_PREC_FP64 ? massive_gather_kernel<PASS, DDX_PREC_FP64>
                                            : massive_gather_kernel<PASS, DDX_PREC_MIXED>,
                 (a.n_grav + kGatherTargets - 1) / kGatherTargets, kGatherThreads, 0, st, s, a,
                 precision == DDX_PREC_FP64 ? ms : slotted(ms, a), 0, nb, np, ms.part);
    return cudaGetLastError();
}
}  // namespace

int massive_slices(int n_grav, int n_exact) {
    const int groups = (n_grav + kSliceThreads - 1) / kSliceThreads;
    const int spans = pair_count(n_grav - n_exact) / kPairSpan;
    int S = (slice_blocks_per_sm(n_grav) * sm_count() + groups - 1) / groups;
    if (S > kMaxSlices) S = kMaxSlices;
    if (S > spans) S = spans;
    return S < 1 ? 1 : S;
}

// The bound grows with the groups, so the bound at the capacity covers every smaller system.
long long massive_part_words(int cap) { return massive_part_words_for(cap, sm_count()); }

cudaError_t launch_massive_pass1(const ddx_state& s, const StepArgs& a, MassiveScratch& ms,
                                 int precision, cudaStream_t st) {
    if (precision == DDX_PREC_MIXED && sliced_fits(a, ms)) return launch_sliced<1>(s, a, ms, st);
    if (precision != DDX_PREC_MIXED && pairs_fit(a, ms)) return launch_pairs<1>(s, a, ms, precision, st);
    const int threads = 128;  // 4 targets per block
    const int blocks = (a.n_grav * 32 + threads - 1) / threads;
    if (precision == DDX_PREC_COMPENSATED)   // the massive set in FP64
        launch_with(a.n_grav <= kOverlapPasses, (massive_pass1_kernel<DDX_PREC_FP64, DDX_PREC_MIXED>), blocks,
                    threads, 0, st, s, a, slotted(ms, a));
    else if (precision == DDX_PREC_MIXED)
        launch_with(a.n_grav <= kOverlapPasses, massive_pass1_kernel<DDX_PREC_MIXED>, blocks, threads, 0, st, s, a,
                    slotted(ms, a));
    else launch_with(a.n_grav <= kOverlapPasses, massive_pass1_kernel<DDX_PREC_FP64>, blocks, threads, 0, st, s, a, ms);
    return cudaGetLastError();
}

cudaError_t launch_massive_pass2(const ddx_state& s, const StepArgs& a, MassiveScratch& ms,
                                 int precision, cudaStream_t st) {
    if (precision == DDX_PREC_MIXED && sliced_fits(a, ms)) return launch_sliced<2>(s, a, ms, st);
    if (precision != DDX_PREC_MIXED && pairs_fit(a, ms)) return launch_pairs<2>(s, a, ms, precision, st);
    const int threads = 128;
    const int blocks = (a.n_grav * 32 + threads - 1) / threads;
    if (precision == DDX_PREC_COMPENSATED)
        launch_with(a.n_grav <= kOverlapPasses, massive_pass2_kernel<DDX_PREC_FP64>, blocks, threads, 0, st, s, a, ms);
    else if (precision == DDX_PREC_MIXED)
        launch_with(a.n_grav <= kOverlapPasses, massive_pass2_kernel<DDX_PREC_MIXED>, blocks, threads, 0, st, s, a,
                    slotted(ms, a));
    else launch_with(a.n_grav <= kOverlapPasses, massive_pass2_kernel<DDX_PREC_FP64>, blocks, threads, 0, st, s, a, ms);
    return cudaGetLastError();
}

int dust_block_threads(int n_dust) {
    static int sm_count[128] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 128) return 256;
    if (sm_count[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
        sm_count[dev] = n;
    }
    int threads = 256;
    while (threads > 64 && (n_dust + threads - 1) / threads < 2 * sm_count[dev]) threads /= 2;
    return threads;
}

cudaError_t launch_dust(const ddx_state& s, const StepArgs& a, const MassiveScratch& ms,
                        const SizeBin* bins, int precision, cudaStream_t st) {
    if (a.n_dust <= 0) return cudaSuccess;
    const int threads = kDustThreads;
    const bool overlap = a.n_grav <= kOverlapDust && !a.after_event;
    const size_t smem = (size_t)kDustTile * 32;
    if (precision == DDX_PREC_MIXED || precision == DDX_PREC_COMPENSATED) {
        return launch_dust_mixed(s, a, ms, bins, precision, st);
    } else if (a.mode == DDX_MODE_REFERENCE) {
        launch_with(overlap, (dust_rk4_kernel<kDustFP64Exact, 1>), (a.n_dust + threads - 1) / threads, threads, smem,
                    st, s, a, ms, bins);
    } else if (a.n_dust <= (a.n_grav > kLanesMinSources ? kLanesMany : kLanesFew)) {
        const int blocks = (int)((4LL * a.n_dust + threads - 1) / threads);
        launch_with(overlap, (dust_rk4_kernel<kDustFP64, 4>), blocks, threads, smem, st, s, a, ms, bins);
    } else {
        launch_with(overlap, (dust_rk4_kernel<kDustFP64, 1>), (a.n_dust + threads - 1) / threads, threads, smem, st,
                    s, a, ms, bins);
    }
    return cudaGetLastError();
}

}  // namespace ddx
