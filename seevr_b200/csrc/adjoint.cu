// adjoint.cu — reverse mode of one physics substep, for gradients of a
// rollout with respect to initial positions, orientations, velocities,
// angular velocities and friction coefficients.
//
// The substep is gravity (physics.comp:418-428), contacts from MPR
// (physics.comp:171-399, 475-491), the PGS solve (500-583) and integration
// (586-604).  Its adjoint, run once per substep in reverse order with the
// state restored from a checkpoint:
//   1. the contacts are recomputed by the regular kernels, the narrowphase
//      taping which hull vertices support each contact's final portal;
//   2. per solver bundle (one warp), the PGS sweep is recomputed in the
//      reference order, recording the inputs of every contact update;
//   3. integration, the PGS sweep (unrolled, reverse order), the contact
//      constants (effective mass, bias, friction coefficient, lever arms),
//      the contact normal, depth and point (as functions of the taped
//      support points), rotation matrices and gravity are differentiated by
//      hand, statement by statement.
// Contact selection (AABBs, broadphase, which pairs touch, MPR's discrete
// portal choices) and the clamps max(., 0), min(., .) and the friction test
// are piecewise constant: the adjoint follows the branches the forward took.
//
// Precision: every forward quantity is recomputed in FP32 with the forward's
// arithmetic, so branch decisions and values are the forward's own; the
// reverse-mode arithmetic on them runs in FP64 (type d3 below).  The PGS
// sweep's per-iteration sensitivities nearly cancel (later iterations undo
// most of an earlier impulse), so FP32 accumulation loses digits, most
// visibly in the friction gradient, while FP64 keeps the result to the
// FP32 forward's own accuracy.
//
// Parallelism: one block per solver bundle, two lanes per contact (or for
// several), in the bundle solver's dataflow order (solver.cu): every body counts
// its updates, and a contact's update runs when both its dynamic bodies have had
// the ones before it; in reverse, the ones after it.  Each contact's constants and
// gradients stay in its lanes' registers through the sweep, velocities and their
// gradients in shared memory.  What a sweep adds to a body besides its velocities'
// gradients (position, rotation, friction) is kept per contact side and summed at
// the end, dynamic bodies by contact rank, fixed bodies (which contacts that run
// together share) in contact order, so the result is deterministic.
// A bundle's time is its longest chain, and a reverse update's is its FP64 work:
// about 4,000 cycles with two lanes, 5,500 with one.  Measured for 1,024 scenes of
// 65 bodies at 30 iterations: 472 us per substep (603 us with one lane per
// contact; 1,000 us with a warp per bundle going level by level, all of this in
// global memory behind four dependent loads).
#include "adjoint.cuh"

#include <algorithm>

#include "solver.cuh"

namespace seevr {
namespace {

// ---- FP64 vectors for the reverse pass (operators only on d3, so an FP32
// f3 can never enter a derivative expression without an explicit D()) ----
struct d3 {
    double x, y, z;
};
struct dm3 {
    d3 c0, c1, c2;
};
__device__ __forceinline__ d3 D(f3 a) { return d3{a.x, a.y, a.z}; }
__device__ __forceinline__ dm3 DM(const m3& m) { return dm3{D(m.c0), D(m.c1), D(m.c2)}; }
__device__ __forceinline__ d3 dz() { return d3{0.0, 0.0, 0.0}; }
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return d3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return d3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator-(d3 a) { return d3{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ d3 operator*(double s, d3 a) { return d3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ d3& operator+=(d3& a, d3 b) {
    a = a + b;
    return a;
}
// s a + b, each component rounded once
__device__ __forceinline__ d3 dfma(double s, d3 a, d3 b) {
    return d3{fma(s, a.x, b.x), fma(s, a.y, b.y), fma(s, a.z, b.z)};
}
__device__ __forceinline__ double ddot(d3 a, d3 b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ d3 dcross(d3 a, d3 b) {
    return d3{fma(a.y, b.z, -(a.z * b.y)), fma(a.z, b.x, -(a.x * b.z)), fma(a.x, b.y, -(a.y * b.x))};
}
// a x b + c
__device__ __forceinline__ d3 dcross_add(d3 a, d3 b, d3 c) {
    return d3{fma(-a.z, b.y, fma(a.y, b.z, c.x)), fma(-a.x, b.z, fma(a.z, b.x, c.y)),
              fma(-a.y, b.x, fma(a.x, b.y, c.z))};
}
__device__ __forceinline__ d3 dhad(d3 a, d3 b) { return d3{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ d3 dmul(const dm3& m, d3 v) {
    return dfma(v.z, m.c2, dfma(v.y, m.c1, v.x * m.c0));
}
__device__ __forceinline__ d3 dmulT(const dm3& m, d3 v) {
    return d3{ddot(m.c0, v), ddot(m.c1, v), ddot(m.c2, v)};
}
__device__ __forceinline__ dm3 dm3zero() { return dm3{dz(), dz(), dz()}; }
__device__ __forceinline__ d3 ldd3(const double* p, uint32_t i) {
    return d3{p[size_t(i) * 3], p[size_t(i) * 3 + 1], p[size_t(i) * 3 + 2]};
}
__device__ __forceinline__ void std3(double* p, uint32_t i, d3 v) {
    p[size_t(i) * 3] = v.x;
    p[size_t(i) * 3 + 1] = v.y;
    p[size_t(i) * 3 + 2] = v.z;
}
// y = R (I ⊙ (Rᵀ x)): accumulates dL/dR into gR (columns) and returns dL/dx
// (the map is symmetric in x).
__device__ __forceinline__ d3 inv_I_bwd(const dm3& R, d3 I, d3 x, d3 gy, dm3& gR) {
    const d3 u = dhad(I, dmulT(R, x));
    const d3 gw = dhad(I, dmulT(R, gy));
    gR.c0 = dfma(u.x, gy, dfma(gw.x, x, gR.c0));
    gR.c1 = dfma(u.y, gy, dfma(gw.y, x, gR.c1));
    gR.c2 = dfma(u.z, gy, dfma(gw.z, x, gR.c2));
    return dmul(R, gw);
}

// dL/d(x,y,z,w) of quat_to_mat (physics.comp:74-81) from dL/dR by columns
__device__ __forceinline__ void quat_bwd(double x, double y, double z, double w, const double* g,
                                         double out[4]) {
    out[0] = 2.0 * (g[1] * y + g[2] * z + g[3] * y - 2.0 * g[4] * x + g[5] * w + g[6] * z -
                    g[7] * w - 2.0 * g[8] * x);
    out[1] = 2.0 * (-2.0 * g[0] * y + g[1] * x - g[2] * w + g[3] * x + g[5] * z + g[6] * w +
                    g[7] * z - 2.0 * g[8] * y);
    out[2] = 2.0 * (-2.0 * g[0] * z + g[1] * w + g[2] * x - g[3] * w - 2.0 * g[4] * z + g[5] * y +
                    g[6] * x + g[7] * y);
    out[3] = 2.0 * (g[1] * z - g[2] * y - g[3] * z + g[5] * x + g[6] * y - g[7] * x);
}

// Gradients of a contact's constants.
struct CGrad {
    d3 n, ra, rb;
    double bias, kn, mu;
};
__device__ __forceinline__ CGrad ld_grad(const double* p, size_t c) {
    const double* q = p + c * 12;
    return CGrad{d3{q[0], q[1], q[2]}, d3{q[3], q[4], q[5]}, d3{q[6], q[7], q[8]}, q[9], q[10],
                 q[11]};
}
// A contact takes two lanes here: the even one holds body a's half of its record
// and of every update, the odd one body b's; they exchange contact-point
// velocities, shares of the tangential mass and gradients of shared quantities by
// shuffles.  (Most bundles hold fewer contacts than a warp has lanes, and an
// update's time is its instruction count.)
struct HalfRec {
    f3 n, r, I;
    float bias, kn, rk, mu, m, msum;  // rk = 1 / kn, 0 when kn is out of div_by's range
    m3 R;
};
__device__ __forceinline__ HalfRec load_half(const float4* rec, uint32_t side) {
    const float4 a = rec[0], b = rec[1];
    rec += 2 + 4 * side;
    const float4 c = rec[0], d = rec[1], e = rec[2], f = rec[3];
    HalfRec h;
    h.n = mk(a.x, a.y, a.z);
    h.bias = a.w;
    h.kn = b.x;
    h.rk = b.y;
    h.mu = b.z;
    h.msum = b.w;
    h.r = mk(c.x, c.y, c.z);
    h.R = m3{mk(c.w, d.x, d.y), mk(d.z, d.w, e.x), mk(e.y, e.z, e.w)};
    h.I = mk(f.x, f.y, f.z);
    h.m = f.w;
    return h;
}
// One update of the lane pair's contact: solve_core's operations in solve_core's
// order.  kBuiltin: with the built-in square root and divisions; else the result
// tells whether every argument was in the branch-free ones' ranges.  All lanes of
// the warp call it.
template <bool kBuiltin>
__device__ __forceinline__ bool update_half(const HalfRec& h, uint32_t side, f3& v, f3& om,
                                            float& lam) {
    const unsigned full = 0xFFFFFFFFu;
    // impulses act on a with -, on b with +, friction the other way round: the
    // sign rides through products and sums, which it does not round differently
    const float sg = side ? 1.0f : -1.0f;
    auto slip = [&](f3 u) {  // u_b - u_a
        const f3 o = mk(__shfl_xor_sync(full, u.x, 1), __shfl_xor_sync(full, u.y, 1),
                        __shfl_xor_sync(full, u.z, 1));
        return side ? sub(u, o) : sub(o, u);
    };
    const float num = -dot(slip(add(v, cross(om, h.r))), h.n) + h.bias;
    float d = kBuiltin ? num / h.kn : div_by(num, h.kn, h.rk);
    const float ln = gmax(lam + d, 0.0f);
    d = ln - lam;
    lam = ln;
    f3 imp = scale(sg, scale(d, h.n));
    v = add(v, scale(h.m, imp));
    om = add(om, apply_inv_I(h.R, h.I, cross(h.r, imp)));
    // Coulomb friction along the current slip direction
    const f3 dv = slip(add(v, cross(om, h.r)));
    const f3 vt = sub(dv, scale(dot(dv, h.n), h.n));
    const float len2 = dot(vt, vt);
    const float rs = rsqrt_approx(len2);
    const float len = kBuiltin ? sqrtf(len2) : root_of(len2, rs);
    // (1e-6)^2 lies in root_of's range; below it only the comparison matters
    const bool still = len2 < kRootMin;
    const bool slips = kBuiltin ? len > 1e-6f : !still && len > 1e-6f;
    f3 td;
    if (kBuiltin) {
        td = divs(vt, len);
    } else {
        const float rl = recip_of(len, rcp_approx(len));
        td = mk(div_by(vt.x, len, rl), div_by(vt.y, len, rl), div_by(vt.z, len, rl));
    }
    const f3 rt = cross(h.r, td);
    const float kq = dot(rt, apply_inv_I(h.R, h.I, rt)), ko = __shfl_xor_sync(full, kq, 1);
    const float kt = h.msum + (side ? ko : kq) + (side ? kq : ko);
    const float dl = gmin(kBuiltin ? len / kt : div_by(len, kt, recip_of(kt, rcp_approx(kt))),
                          h.mu * ln);
    imp = scale(-sg, scale(dl, td));
    const f3 v2 = add(v, scale(h.m, imp)), w2 = add(om, apply_inv_I(h.R, h.I, cross(h.r, imp)));
    if (slips) {
        v = v2;
        om = w2;
    }
    if (kBuiltin) return true;
    // a NaN fails every comparison; the slip's components are at most len
    const uint32_t key = min(min(size_key(vt.x), size_key(vt.y)), size_key(vt.z));
    return size_key(num) >= kNumMinKey && fabsf(num) <= kNumMax &&
           (still || (len2 <= kRootMax && key >= kNumMinKey && kt >= kDivMin && kt <= kDivMax));
}

// The update with the built-in operations, for the arguments outside the ranges.
__device__ __noinline__ void half_builtin(const HalfRec* h, uint32_t side, float* state) {
    f3 v = mk(state[0], state[1], state[2]), om = mk(state[3], state[4], state[5]);
    update_half<true>(*h, side, v, om, state[6]);
    state[0] = v.x; state[1] = v.y; state[2] = v.z;
    state[3] = om.x; state[4] = om.y; state[5] = om.z;
}

// update_half, redone with the built-in operations by a warp where a lane that
// `counts` has an argument outside the ranges.
__device__ __forceinline__ void forward_half(const HalfRec& h, uint32_t side, bool counts, f3& v, f3& om,
                                       float& lam) {
    f3 v2 = v, w2 = om;
    float l2 = lam;
    const bool ok = update_half<false>(h, side, v2, w2, l2) && h.rk != 0.0f;
    if (__any_sync(0xFFFFFFFFu, counts && !ok)) {
        const HalfRec copy = h;
        float state[7] = {v.x, v.y, v.z, om.x, om.y, om.z, lam};
        half_builtin(&copy, side, state);
        v2 = mk(state[0], state[1], state[2]);
        w2 = mk(state[3], state[4], state[5]);
        l2 = state[6];
    }
    v = v2;
    om = w2;
    lam = l2;
}

// The forward intermediates of one update from its inputs, FP32, the forward's
// arithmetic (update_half): the same values and branches.  Of the calling lane's
// body where a vector belongs to one.  All lanes of the warp call.
struct Mid {
    f3 dvn, imp, x, w1, dv, vt, td, rt;
    float d0, s1, l1, d, dn, s, kt, dt;
    bool slips, take2;
};
template <bool kBuiltin>
__device__ __forceinline__ bool mid_half(const HalfRec& h, uint32_t side, f3 v, f3 om, float lam,
                                         Mid& m) {
    const unsigned full = 0xFFFFFFFFu;
    const float sg = side ? 1.0f : -1.0f;
    auto slip = [&](f3 u) {  // u_b - u_a
        const f3 o = mk(__shfl_xor_sync(full, u.x, 1), __shfl_xor_sync(full, u.y, 1),
                        __shfl_xor_sync(full, u.z, 1));
        return side ? sub(u, o) : sub(o, u);
    };
    m.dvn = slip(add(v, cross(om, h.r)));
    const float num = -dot(m.dvn, h.n) + h.bias;
    m.d0 = kBuiltin ? num / h.kn : div_by(num, h.kn, h.rk);
    m.s1 = lam + m.d0;
    m.l1 = gmax(m.s1, 0.0f);
    m.d = m.l1 - lam;
    m.imp = scale(sg, scale(m.d, h.n));
    m.x = cross(h.r, m.imp);
    m.w1 = add(om, apply_inv_I(h.R, h.I, m.x));
    m.dv = slip(add(add(v, scale(h.m, m.imp)), cross(m.w1, h.r)));
    m.dn = dot(m.dv, h.n);
    m.vt = sub(m.dv, scale(m.dn, h.n));
    const float len2 = dot(m.vt, m.vt);
    const float rs = rsqrt_approx(len2);
    const bool still = len2 < kRootMin;
    m.s = kBuiltin ? sqrtf(len2) : root_of(len2, rs);
    m.slips = kBuiltin ? m.s > 1e-6f : !still && m.s > 1e-6f;
    if (kBuiltin) {
        m.td = divs(m.vt, m.s);
    } else {
        const float rl = recip_of(m.s, rcp_approx(m.s));
        m.td = mk(div_by(m.vt.x, m.s, rl), div_by(m.vt.y, m.s, rl), div_by(m.vt.z, m.s, rl));
    }
    m.rt = cross(h.r, m.td);
    const float kq = dot(m.rt, apply_inv_I(h.R, h.I, m.rt)), ko = __shfl_xor_sync(full, kq, 1);
    m.kt = h.msum + (side ? ko : kq) + (side ? kq : ko);
    const float q1 = kBuiltin ? m.s / m.kt : div_by(m.s, m.kt, recip_of(m.kt, rcp_approx(m.kt)));
    const float q2 = h.mu * m.l1;
    m.take2 = q2 < q1;  // GLSL min(q1, q2)
    m.dt = m.take2 ? q2 : q1;
    if (kBuiltin) return true;
    const uint32_t key = min(min(size_key(m.vt.x), size_key(m.vt.y)), size_key(m.vt.z));
    return h.rk != 0.0f && size_key(num) >= kNumMinKey && fabsf(num) <= kNumMax &&
           (still || (len2 <= kRootMax && key >= kNumMinKey && m.kt >= kDivMin && m.kt <= kDivMax));
}
__device__ __noinline__ void mid_builtin(const HalfRec* h, uint32_t side, const float* in, Mid* m) {
    mid_half<true>(*h, side, mk(in[0], in[1], in[2]), mk(in[3], in[4], in[5]), in[6], *m);
}

// What the reverse sweep carries for a contact: gradients of its constants (r: the
// calling lane's lever arm; the shared ones alike in both lanes), of its impulse
// and of the lane's body's rotation.
struct Carry {
    d3 n, r;
    double bias, kn, mu, lam;
    dm3 R;
};

// The sum of both lanes' vectors.
__device__ __forceinline__ d3 both(d3 v) {
    const unsigned full = 0xFFFFFFFFu;
    return v + d3{__shfl_xor_sync(full, v.x, 1), __shfl_xor_sync(full, v.y, 1),
                  __shfl_xor_sync(full, v.z, 1)};
}

// Reverse of an update from its inputs (v, om, lam).  On entry Gv, Gw hold
// dL/d(the lane's body's velocities after the update) and y.lam dL/d(λ after); on
// return dL/d(before).  fixed: the body's outputs are discarded.  counts: whether
// the lane pair's contact is updated at all (the others compute along).
__device__ __forceinline__ void reverse_half(const HalfRec& h, uint32_t side, bool counts, f3 v,
                                             f3 om, float lam, bool fixed, d3& Gv, d3& Gw, Carry& y) {
    Mid m;
    const bool ok = mid_half<false>(h, side, v, om, lam, m);
    if (__any_sync(0xFFFFFFFFu, counts && !ok)) {
        const HalfRec hc = h;
        const float in[7] = {v.x, v.y, v.z, om.x, om.y, om.z, lam};
        Mid mc;
        mid_builtin(&hc, side, in, &mc);
        m = mc;
    }
    // the reverse pass, FP64; impulses act on b with sg = +, on a with -
    const double sg = side ? 1.0 : -1.0;
    const dm3 R = DM(h.R);
    const d3 I = D(h.I), n = D(h.n), r = D(h.r);
    const double im = h.m;
    d3 gv1 = fixed ? dz() : Gv, gw1 = fixed ? dz() : Gw;
    double g_l1 = y.lam;
    d3 g_vt = dz();
    if (__any_sync(0xFFFFFFFFu, counts && m.slips)) {
        const bool on = m.slips;
        const double sd = on ? double(m.s) : 1.0, inv_s = 1.0 / sd;
        const float dtf = on ? m.dt : 0.0f;
        const d3 td = on ? D(m.td) : dz(), rt = on ? D(m.rt) : dz();
        // v2 = v1 + m it; w2 = w1 + A(r x it); it = -sg dt td
        const f3 itf = on ? scale(side ? -1.0f : 1.0f, scale(dtf, m.td)) : mk(0.f, 0.f, 0.f);
        const d3 it = D(itf);
        const d3 g_x2 = inv_I_bwd(R, I, D(cross(h.r, itf)), on ? gw1 : dz(), y.R);
        y.r = dcross_add(it, g_x2, y.r);
        const d3 g_it = both(-sg * dfma(im, gv1, dcross(g_x2, r)));
        const double g_dt = ddot(g_it, td);
        d3 g_td = double(dtf) * g_it;
        double g_kt = 0.0, g_s = 0.0;
        const double g_q1 = m.take2 || !on ? 0.0 : g_dt, g_q2 = m.take2 && on ? g_dt : 0.0;
        y.mu = fma(g_q2, double(m.l1), y.mu);
        g_l1 = fma(g_q2, double(h.mu), g_l1);
        const double inv_kt = 1.0 / (on ? double(m.kt) : 1.0);
        g_s = g_q1 * inv_kt;
        g_kt = -g_s * sd * inv_kt;
        // kt = ... + rt·A(rt) of both: d/drt = 2 A(rt)
        const d3 g_rt = 2.0 * inv_I_bwd(R, I, rt, g_kt * rt, y.R);
        // rt = r x td
        y.r = dcross_add(td, g_rt, y.r);
        g_td += both(dcross(g_rt, r));
        // td = vt / s; s = |vt|
        const d3 vt = D(m.vt);
        g_s = fma(-ddot(g_td, vt) * inv_s, inv_s, g_s);
        g_vt = on ? dfma(g_s * inv_s, vt, inv_s * g_td) : dz();
    }
    // vt = dv - dn n; dn = dv·n
    const double g_dn = -ddot(g_vt, n);
    y.n = dfma(-double(m.dn), g_vt, dfma(g_dn, D(m.dv), y.n));
    // dv = u1_b - u1_a; u1 = v1 + w1 x r
    const d3 g_u1 = sg * dfma(g_dn, n, g_vt);
    gv1 += g_u1;
    gw1 = dcross_add(r, g_u1, gw1);
    y.r = dcross_add(g_u1, D(m.w1), y.r);
    // v1 = v + m imp; w1 = w + A(x); x = r x imp; imp = sg d n
    const d3 imp = D(m.imp);
    const d3 g_x = inv_I_bwd(R, I, D(m.x), gw1, y.R);
    y.r = dcross_add(imp, g_x, y.r);
    const d3 g_imp = both(sg * dfma(im, gv1, dcross(g_x, r)));
    const double g_d = ddot(g_imp, n);
    y.n = dfma(double(m.d), g_imp, y.n);
    // d = l1 - lam; l1 = max(s1, 0); s1 = lam + d0
    g_l1 += g_d;
    const double g_s1 = m.s1 < 0.f ? 0.0 : g_l1;
    y.lam = g_s1 - g_d;
    // d0 = (-vn + bias) / kn
    const double q = g_s1 / double(h.kn);
    y.bias += q;
    y.kn = fma(-q, double(m.d0), y.kn);
    // vn = dvn·n; dvn = u_b - u_a; u = v + w x r; dL/dvn = -q
    y.n = dfma(-q, D(m.dvn), y.n);
    const d3 g_u = (-sg * q) * n;
    gv1 += g_u;
    gw1 = dcross_add(r, g_u, gw1);
    y.r = dcross_add(g_u, D(om), y.r);
    // a fixed body's state persists: its incoming gradient passes through
    Gv = fixed ? Gv + gv1 : gv1;
    Gw = fixed ? Gw + gw1 : gw1;
}

__device__ __forceinline__ f3 hull_vert(const World& w, uint32_t vs, uint32_t i) {
    return i == kNone ? mk(0.f, 0.f, 0.f) : ld3(w.hull, vs + i);
}

// dL/d (positions, rotations) of one contact's normal, depth and point,
// through the taped supporting vertices (physics.comp:224-247, 346-365,
// 376-387).  The support points are recomputed in FP32 as the narrowphase
// computed them; the derivatives are FP64.
__device__ void contact_geom_bwd(const World& w, const Consts& k, const AdjScratch& a, uint32_t c,
                                 uint32_t ba, uint32_t bb, d3 g_n, double g_pen, d3 g_cp,
                                 d3& gpA, d3& gpB, dm3& gRA, dm3& gRB) {
    const uint4 t0 = a.ctape[size_t(c) * 2], t1 = a.ctape[size_t(c) * 2 + 1];
    const f3 pAf = ld3(w.pos, ba), pBf = ld3(w.pos, bb);
    const m3 RAf = quat_to_mat(w.quat, ba), RBf = quat_to_mat(w.quat, bb);
    const uint32_t vsA = w.hull_range[size_t(ba) * 2], vsB = w.hull_range[size_t(bb) * 2];
    f3 hA[4], hB[4], saf[4], sbf[4], vf[4];
    d3 gsa[4], gsb[4], gv[4];
    const uint32_t ia[4] = {kNone, t0.y, t0.w, t1.y};
    const uint32_t ib[4] = {kNone, t0.z, t1.x, t1.z};
    for (int i = 0; i < 4; ++i) {
        hA[i] = hull_vert(w, vsA, ia[i]);
        hB[i] = hull_vert(w, vsB, ib[i]);
        saf[i] = add(pAf, mul(RAf, hA[i]));
        sbf[i] = add(pBf, mul(RBf, hB[i]));
        vf[i] = sub(saf[i], sbf[i]);
        gsa[i] = gsb[i] = gv[i] = dz();
    }
    gpA = dz();
    gpB = dz();
    if (t0.x == 2u) {  // segment case: depth = |v1|, n = v1/|v1|, cp = (s1a + s1b)/2
        const d3 v1 = D(vf[1]);
        const double l = sqrt(ddot(v1, v1));
        const d3 n = (1.0 / l) * v1;
        d3 g1 = g_pen * n;
        g1 += (1.0 / l) * (g_n - ddot(n, g_n) * n);
        gsa[1] = 0.5 * g_cp + g1;
        gsb[1] = 0.5 * g_cp - g1;
    } else {  // portal: n = normalize((v2-v1)x(v3-v1)), depth = n·v1, cp = find_pos
        f3 v0f = sub(pAf, pBf);
        if (fabsf(v0f.x) < k.eps && fabsf(v0f.y) < k.eps && fabsf(v0f.z) < k.eps)
            v0f.x += 10.0f * k.eps;
        vf[0] = v0f;
        saf[0] = pAf;
        sbf[0] = pBf;
        d3 v[4], sa[4], sb[4];
        for (int i = 0; i < 4; ++i) {
            v[i] = D(vf[i]);
            sa[i] = D(saf[i]);
            sb[i] = D(sbf[i]);
        }
        const d3 e1 = v[2] - v[1], e2 = v[3] - v[1];
        const d3 cr = dcross(e1, e2);
        const double cl = sqrt(ddot(cr, cr));
        const d3 n = (1.0 / cl) * cr;
        d3 g_nn = g_n;
        g_nn += g_pen * v[1];
        gv[1] += g_pen * n;
        // contact point: the forward's fallback test (FP32, find_pos)
        const float fsum = dot(cross(vf[1], vf[2]), vf[3]) + -dot(cross(vf[0], vf[2]), vf[3]) +
                           dot(cross(vf[0], vf[1]), vf[3]) + -dot(cross(vf[0], vf[1]), vf[2]);
        const bool fallback = fabsf(fsum) < k.eps;
        double b[4];
        if (!fallback) {
            b[0] = ddot(dcross(v[1], v[2]), v[3]);
            b[1] = -ddot(dcross(v[0], v[2]), v[3]);
            b[2] = ddot(dcross(v[0], v[1]), v[3]);
            b[3] = -ddot(dcross(v[0], v[1]), v[2]);
        } else {
            b[0] = 0.0;
            b[1] = ddot(dcross(v[2], v[3]), n);
            b[2] = ddot(dcross(v[3], v[1]), n);
            b[3] = ddot(dcross(v[1], v[2]), n);
        }
        const double sum = b[0] + b[1] + b[2] + b[3];
        d3 P = dz();
        for (int i = 0; i < 4; ++i) P += b[i] * (sa[i] + sb[i]);
        const d3 gP = (0.5 / sum) * g_cp;
        const double g_sum = -0.5 / (sum * sum) * ddot(g_cp, P);
        double gb[4];
        for (int i = 0; i < 4; ++i) {
            gb[i] = ddot(gP, sa[i]) + ddot(gP, sb[i]) + g_sum;
            gsa[i] += b[i] * gP;
            gsb[i] += b[i] * gP;
        }
        if (!fallback) {
            // triple products [a,b,c] = (a x b)·c: d/da = b x c, d/db = c x a, d/dc = a x b
            gv[1] += gb[0] * dcross(v[2], v[3]);
            gv[2] += gb[0] * dcross(v[3], v[1]);
            gv[3] += gb[0] * dcross(v[1], v[2]);
            gv[0] += (-gb[1]) * dcross(v[2], v[3]);
            gv[2] += (-gb[1]) * dcross(v[3], v[0]);
            gv[3] += (-gb[1]) * dcross(v[0], v[2]);
            gv[0] += gb[2] * dcross(v[1], v[3]);
            gv[1] += gb[2] * dcross(v[3], v[0]);
            gv[3] += gb[2] * dcross(v[0], v[1]);
            gv[0] += (-gb[3]) * dcross(v[1], v[2]);
            gv[1] += (-gb[3]) * dcross(v[2], v[0]);
            gv[2] += (-gb[3]) * dcross(v[0], v[1]);
        } else {
            // b1 = (v2 x v3)·n, b2 = (v3 x v1)·n, b3 = (v1 x v2)·n
            gv[2] += gb[1] * dcross(v[3], n);
            gv[3] += gb[1] * dcross(n, v[2]);
            g_nn += gb[1] * dcross(v[2], v[3]);
            gv[3] += gb[2] * dcross(v[1], n);
            gv[1] += gb[2] * dcross(n, v[3]);
            g_nn += gb[2] * dcross(v[3], v[1]);
            gv[1] += gb[3] * dcross(v[2], n);
            gv[2] += gb[3] * dcross(n, v[1]);
            g_nn += gb[3] * dcross(v[1], v[2]);
        }
        // n = cr / |cr|; cr = e1 x e2
        const d3 g_cr = (1.0 / cl) * (g_nn - ddot(n, g_nn) * n);
        const d3 g_e1 = dcross(e2, g_cr), g_e2 = dcross(g_cr, e1);
        gv[2] += g_e1;
        gv[3] += g_e2;
        gv[1] = gv[1] - (g_e1 + g_e2);
        // v0 = pA - pB; s0a = pA; s0b = pB
        gpA += gv[0] + gsa[0];
        gpB += gsb[0] - gv[0];
        for (int i = 1; i < 4; ++i) {
            gsa[i] += gv[i];
            gsb[i] = gsb[i] - gv[i];
        }
    }
    // s_ia = pA + RA h_ia; s_ib = pB + RB h_ib (i = 1..3)
    gRA = dm3zero();
    gRB = dm3zero();
    for (int i = 1; i < 4; ++i) {
        gpA += gsa[i];
        gpB += gsb[i];
        const d3 ha = D(hA[i]), hb = D(hB[i]);
        gRA.c0 += ha.x * gsa[i];
        gRA.c1 += ha.y * gsa[i];
        gRA.c2 += ha.z * gsa[i];
        gRB.c0 += hb.x * gsb[i];
        gRB.c1 += hb.y * gsb[i];
        gRB.c2 += hb.z * gsb[i];
    }
}

// A contact side's slot of gradients to its body: v3 w3 p3 R9 friction1.
constexpr uint32_t kFixStride = 20;
__device__ __forceinline__ double* side_slot(const AdjScratch& a, size_t c, uint32_t side) {
    return a.fix + (c * 2 + side) * kFixStride;
}
__device__ __forceinline__ void put3(double* f, d3 v) {
    f[0] = v.x;
    f[1] = v.y;
    f[2] = v.z;
}
__device__ __forceinline__ d3 get3(const double* f) { return d3{f[0], f[1], f[2]}; }
__device__ __forceinline__ void putR(double* f, const dm3& g) {
    put3(f + 9, g.c0);
    put3(f + 12, g.c1);
    put3(f + 15, g.c2);
}
__device__ __forceinline__ dm3 getR(const double* f) { return dm3{get3(f + 9), get3(f + 12), get3(f + 15)}; }

// A contact side: bundle-local body, and its rank among the body's contacts with
// the flags (kFixed: infinite mass, orders nothing; kNoStore: not written back;
// kSkip: both bodies' masses infinite, the contact is not solved).
constexpr uint32_t kRankMask = 0x0FFFFFFFu, kFixed = 1u << 31, kNoStore = 1u << 30, kSkip = 1u << 29;
static_assert(kRankMask < kSkip, "rank field overlaps the flags");

// One bundle's working arrays: shared memory, or global for large bundles.
struct AdjBodies {
    float4* v;       // velocity during the recomputed sweep
    float4* w;       // angular velocity
    double* g;       // [6 n] running gradients of both
    uint32_t* count;  // updates each body has had
};
__host__ __device__ constexpr size_t adj_body_bytes() { return 2 * sizeof(float4) + 6 * sizeof(double) + 4; }

// A lane pair's contacts i, i + width, ... in sequence order, forward or backward.
struct AdjArgs {
    uint32_t c0, nc, side, slot, width, iters;
    uint32_t* left;  // pairs that are not done
};

// The contact side's flags and rank, body and degree.
struct Place {
    uint32_t l, z, deg;
};
__device__ __forceinline__ Place place_of(const AdjScratch& a, size_t c, uint32_t side) {
    const uint4 x = a.side[c];
    const uint2 d = a.degree[c];
    return Place{side ? x.y : x.x, side ? x.w : x.z, side ? d.y : d.x};
}
// Whether the pair starting at slot owns a contact that is solved.
__device__ __forceinline__ bool owns_any(const AdjScratch& a, const AdjArgs& f) {
    bool any = false;
    for (uint32_t j = f.slot; j < f.nc; j += f.width) any |= !(a.side[f.c0 + j].z & kSkip);
    return any && f.iters > 0;
}
__device__ __forceinline__ bool pair_ready(bool mine) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, mine);
    return ((m >> (threadIdx.x & 30u)) & 3u) == 3u;
}

// The PGS sweep recomputed in dataflow order, the inputs of every update taped
// ([iteration][13][contact]).
__device__ void adjoint_forward(const Scratch& s, const AdjScratch& a, const AdjArgs& f,
                                const AdjBodies& B) {
    const unsigned full = 0xFFFFFFFFu;
    const bool several = f.nc > f.width;
    uint32_t i = f.slot, it = 0;
    bool live = owns_any(a, f);
    HalfRec h{};
    Place x{0u, kFixed | kNoStore, 0u};
    float lam = 0.0f;
    auto arm = [&] {
        h = load_half(s.s_rec + size_t(f.c0 + i) * kRecWords, f.side);
        x = place_of(a, f.c0 + i, f.side);
        lam = several && it > 0 ? a.lam[f.c0 + i] : 0.0f;
    };
    // on to the pair's next contact that is solved
    auto step = [&] {
        do {
            i += f.width;
            if (i >= f.nc) {
                i = f.slot;
                live = ++it < f.iters;
            }
        } while (live && (a.side[f.c0 + i].z & kSkip));
        if (live) arm();
    };
    if (live) {
        if (a.side[f.c0 + i].z & kSkip) step();
        else arm();
        if (live && f.side == 0) atomicAdd(f.left, 1u);
    }
    float* tape = a.tape + size_t(f.c0) * f.iters * 13;
    __syncthreads();
    // the first unfinished update of the sequence is ready in every round
    for (uint64_t round = 0, cap = uint64_t(f.iters) * f.nc; round <= cap; ++round) {
        const float4 v4 = B.v[x.l], w4 = B.w[x.l];
        const uint32_t want = x.deg * it + (x.z & kRankMask);
        const bool ready = pair_ready(live && ((x.z & (kFixed | kNoStore)) || B.count[x.l] == want));
        const uint32_t left = *f.left;
        __syncthreads();  // every read of the round before its writes
        if (left == 0u) break;
        if (__any_sync(full, ready)) {
            f3 v = mk(v4.x, v4.y, v4.z), om = mk(w4.x, w4.y, w4.z);
            float ln = lam;
            forward_half(h, f.side, ready, v, om, ln);
            if (ready) {
                float* t = tape + (size_t(it) * 13 + 6 * f.side) * f.nc + i;
                const float in[6] = {v4.x, v4.y, v4.z, w4.x, w4.y, w4.z};
#pragma unroll
                for (uint32_t q = 0; q < 6; ++q) t[size_t(q) * f.nc] = in[q];
                if (f.side == 0) t[size_t(12) * f.nc] = lam;
                lam = ln;
                if (!(x.z & (kFixed | kNoStore))) {
                    B.v[x.l] = make_float4(v.x, v.y, v.z, 0.0f);
                    B.w[x.l] = make_float4(om.x, om.y, om.z, 0.0f);
                    B.count[x.l] = want + 1u;
                }
                if (several) {
                    a.lam[f.c0 + i] = lam;  // both lanes: each reads back its own write
                    step();
                } else {
                    live = ++it < f.iters;
                }
                if (!live && f.side == 0) atomicSub(f.left, 1u);
            }
        }
        __syncthreads();
    }
}

// The sweep reversed: updates in reverse order, each when the later ones at its
// dynamic bodies are done.  Leaves, per contact, the gradients of its constants
// (a.gc) and by side those of its body's rotation, and of the velocities of a
// fixed body (side slots).
__device__ void adjoint_reverse(const Scratch& s, const AdjScratch& a, const AdjArgs& f,
                                const AdjBodies& B) {
    const unsigned full = 0xFFFFFFFFu;
    const bool several = f.nc > f.width;
    // the pair's last contact of the sequence first
    const uint32_t last = f.slot < f.nc ? f.slot + (f.nc - 1 - f.slot) / f.width * f.width : f.slot;
    uint32_t i = last, it = 0;  // it: iterations before the last
    bool live = owns_any(a, f);
    HalfRec h{};
    Place x{0u, kFixed | kNoStore, 0u};
    Carry y{};
    d3 fv = dz(), fw = dz();  // gradient of a fixed body's velocities
    float in[7] = {};
    const float* tape = a.tape + size_t(f.c0) * f.iters * 13;
    auto inputs = [&](uint32_t back) {
        const float* t = tape + size_t(f.iters - 1 - back) * 13 * f.nc + i;
#pragma unroll
        for (uint32_t q = 0; q < 6; ++q) in[q] = t[size_t(6 * f.side + q) * f.nc];
        in[6] = t[size_t(12) * f.nc];
    };
    auto arm = [&] {
        const size_t c = f.c0 + i;
        h = load_half(s.s_rec + c * kRecWords, f.side);
        x = place_of(a, c, f.side);
        y = Carry{};
        fv = fw = dz();
        if (several && it > 0) {
            const double* q = a.gc + c * 12;
            y.n = get3(q);
            y.r = get3(q + 3 + 3 * f.side);
            y.bias = q[9];
            y.kn = q[10];
            y.mu = q[11];
            y.lam = a.glam[c];
            const double* o = side_slot(a, c, f.side);
            y.R = getR(o);
            fv = get3(o);
            fw = get3(o + 3);
        }
        inputs(it);
    };
    // (a dynamic side's slot starts with zero velocity gradients: fv, fw)
    auto save = [&] {
        const size_t c = f.c0 + i;
        double* q = a.gc + c * 12;
        put3(q + 3 + 3 * f.side, y.r);
        if (several || f.side == 0) {  // several: each lane reads back its own write
            put3(q, y.n);
            q[9] = y.bias;
            q[10] = y.kn;
            q[11] = y.mu;
            a.glam[c] = y.lam;
        }
        double* o = side_slot(a, c, f.side);
        putR(o, y.R);
        put3(o, fv);
        put3(o + 3, fw);
    };
    auto step = [&] {
        do {
            if (i >= f.width) {
                i -= f.width;
            } else {
                i = last;
                live = ++it < f.iters;
            }
        } while (live && (a.side[f.c0 + i].z & kSkip));
        if (live) arm();
    };
    if (f.iters == 0)
        for (i = f.slot; i < f.nc; i += f.width) save();  // nothing to reverse
    if (live) {
        if (a.side[f.c0 + i].z & kSkip) step();
        else arm();
        if (live && f.side == 0) atomicAdd(f.left, 1u);
    }
    __syncthreads();
    for (uint64_t round = 0, cap = uint64_t(f.iters) * f.nc; round <= cap; ++round) {
        const uint32_t want = x.deg * it + (x.deg - 1u - (x.z & kRankMask));
        const bool ready = pair_ready(live && ((x.z & (kFixed | kNoStore)) || B.count[x.l] == want));
        d3 Gv = dz(), Gw = dz();
        if (live && !(x.z & kFixed)) {
            Gv = get3(B.g + size_t(x.l) * 6);
            Gw = get3(B.g + size_t(x.l) * 6 + 3);
        }
        const uint32_t left = *f.left;
        __syncthreads();
        if (left == 0u) break;
        if (__any_sync(full, ready)) {
            const f3 v = mk(in[0], in[1], in[2]), om = mk(in[3], in[4], in[5]);
            const float lam = in[6];
            // the next update's inputs, beside this one
            if (ready && !several && it + 1 < f.iters) inputs(it + 1);
            Carry y2 = y;
            reverse_half(h, f.side, ready, v, om, lam, (x.z & kFixed) != 0u, Gv, Gw, y2);
            if (ready) {
                y = y2;
                if (x.z & kFixed) {
                    fv += Gv;
                    fw += Gw;
                } else if (!(x.z & kNoStore)) {
                    put3(B.g + size_t(x.l) * 6, Gv);
                    put3(B.g + size_t(x.l) * 6 + 3, Gw);
                    B.count[x.l] = want + 1u;
                }
                if (several) {
                    save();
                    step();
                } else {
                    live = ++it < f.iters;
                    if (!live) save();
                }
                if (!live && f.side == 0) atomicSub(f.left, 1u);
            }
        }
        __syncthreads();
    }
}

// Contact c's constants and geometry reversed; adds its sides' gradients to their
// slots.
__device__ void adjoint_contact(const World& w, const Consts& k, const Scratch& s,
                                const AdjScratch& a, uint32_t c, float dt) {
    const uint32_t ga = w.c_a[c], gb = w.c_b[c];
    const uint32_t ba = w.geom_body[ga], bb = w.geom_body[gb];
    const Rec h = load_rec(s.s_rec + size_t(c) * kRecWords);
    CGrad gc = ld_grad(a.gc, c);
    double *fa = side_slot(a, c, 0), *fb = side_slot(a, c, 1);
    dm3 gRa = getR(fa), gRb = getR(fb);
    const dm3 RA = DM(h.a.R), RB = DM(h.b.R);
    const d3 IA = D(h.a.I), IB = D(h.b.I), n = D(h.n), ra = D(h.a.r), rb = D(h.b.r);
    // kn = ima + imb + ran·A(ran) + rbn·B(rbn); ran = ra x n
    const d3 ran = D(cross(h.a.r, h.n)), rbn = D(cross(h.b.r, h.n));
    const d3 g_ran = 2.0 * inv_I_bwd(RA, IA, ran, gc.kn * ran, gRa);
    const d3 g_rbn = 2.0 * inv_I_bwd(RB, IB, rbn, gc.kn * rbn, gRb);
    gc.ra = dcross_add(n, g_ran, gc.ra);
    gc.rb = dcross_add(n, g_rbn, gc.rb);
    gc.n = dcross_add(g_ran, ra, dcross_add(g_rbn, rb, gc.n));
    // bias = baum max(pen - slop, 0)/dt + e max(-vn0, 0)
    const float pen = w.c_pen[c];
    const double g_pen = (pen - k.slop < 0.f) ? 0.0 : gc.bias * double(k.baumgarte) / double(dt);
    const float e = gmax(w.restitution[ga], w.restitution[gb]);
    const f3 oa = ld3(w.omega, ba), ob = ld3(w.omega, bb);
    const f3 va0 = add(ld3(w.vel, ba), cross(oa, h.a.r));
    const f3 vb0 = add(ld3(w.vel, bb), cross(ob, h.b.r));
    const float vn0 = dot(sub(vb0, va0), h.n);
    const double g_vn0 = (-vn0 < 0.f) ? 0.0 : -double(e) * gc.bias;
    gc.n = dfma(g_vn0, D(sub(vb0, va0)), gc.n);
    const d3 g_ub0 = g_vn0 * n, g_ua0 = -g_ub0;
    gc.ra = dcross_add(g_ua0, D(oa), gc.ra);
    gc.rb = dcross_add(g_ub0, D(ob), gc.rb);
    // mu = sqrt(fa fb)
    double gfa = 0.0, gfb = 0.0;
    if (h.mu > 0.f) {
        const double qa = w.friction[ga], qb = w.friction[gb], mu = h.mu;
        gfa = gc.mu * qb / (2.0 * mu);
        gfb = gc.mu * qa / (2.0 * mu);
    }
    // ra = cp - pos_a; rb = cp - pos_b; the contact point, normal and depth
    // through the taped support vertices
    d3 gpA, gpB;
    dm3 gRA, gRB;
    contact_geom_bwd(w, k, a, c, ba, bb, gc.n, g_pen, gc.ra + gc.rb, gpA, gpB, gRA, gRB);
    put3(fa, get3(fa) + g_ua0);
    put3(fa + 3, dcross_add(ra, g_ua0, get3(fa + 3)));
    put3(fa + 6, gpA - gc.ra);
    putR(fa, dm3{gRa.c0 + gRA.c0, gRa.c1 + gRA.c1, gRa.c2 + gRA.c2});
    fa[18] = gfa;
    put3(fb, get3(fb) + g_ub0);
    put3(fb + 3, dcross_add(rb, g_ub0, get3(fb + 3)));
    put3(fb + 6, gpB - gc.rb);
    putR(fb, dm3{gRb.c0 + gRB.c0, gRb.c1 + gRB.c1, gRb.c2 + gRB.c2});
    fb[18] = gfb;
}

template <uint32_t W>
__global__ void __launch_bounds__(32 * W)
    k_adjoint(World w, Consts k, Scratch s, AdjScratch a, Grads g, float dt, uint32_t nbmax) {
    constexpr uint32_t kThreads = 32 * W;
    extern __shared__ double smd[];
    __shared__ uint32_t sh_left, sh_deg;
    if (halted(w.status)) return;  // the recomputed contacts are not valid
    const uint32_t t = threadIdx.x, lane = t & 31u, wid = t >> 5, bundle = blockIdx.x;
    const uint32_t b0 = w.bundle_off[bundle], nb = w.bundle_off[bundle + 1] - b0;
    const uint32_t c0 = first_contact(w, s, b0), nc = first_contact(w, s, b0 + nb) - c0;
    if (nb == 0) return;
    const bool in_smem = nb <= nbmax;
    AdjBodies B;
    B.g = in_smem ? smd : a.gvw + size_t(b0) * 6;
    B.v = in_smem ? reinterpret_cast<float4*>(smd + 6 * nbmax) : a.body4 + size_t(b0) * 2;
    B.w = B.v + (in_smem ? nbmax : nb);
    B.count = in_smem ? reinterpret_cast<uint32_t*>(B.w + nbmax) : a.last + b0;

    // ---- working velocities (post-gravity), contact sides ----
    for (uint32_t i = t; i < nb; i += kThreads) {
        const f3 v = ld3(w.vel, b0 + i), o = ld3(w.omega, b0 + i);
        B.v[i] = make_float4(v.x, v.y, v.z, 0.0f);
        B.w[i] = make_float4(o.x, o.y, o.z, 0.0f);
        B.count[i] = 0;
    }
    for (uint32_t i = t; i < nc; i += kThreads) {
        const uint32_t c = c0 + i, ba = w.geom_body[w.c_a[c]], bb = w.geom_body[w.c_b[c]];
        const float ma = w.inv_mass[ba], mb = w.inv_mass[bb];
        const f3 Ia = ld3(w.inv_inertia, ba), Ib = ld3(w.inv_inertia, bb);
        uint4 x{ba - b0, bb - b0, 0u, 0u};
        if (ma == 0.0f && Ia.x == 0.0f && Ia.y == 0.0f && Ia.z == 0.0f) x.z = kFixed;
        if (mb == 0.0f && Ib.x == 0.0f && Ib.y == 0.0f && Ib.z == 0.0f) x.w = kFixed;
        if (ma == 0.0f && mb == 0.0f) {  // physics.comp:531
            x.z |= kSkip | kNoStore;
            x.w |= kSkip | kNoStore;
        } else if (ba == bb) {
            x.z |= kNoStore;  // both sides one body: b is written last, one count
        }
        a.side[c] = x;
        const f3 va = ld3(w.vel, ba), oa = ld3(w.omega, ba), vb = ld3(w.vel, bb), ob = ld3(w.omega, bb);
        make_rec(w, k, c, ba, bb, va, oa, vb, ob, dt, s.s_rec + size_t(c) * kRecWords);
    }
    if (t == 0) sh_left = sh_deg = 0;
    __syncthreads();
    // ---- ranks in contact order by one warp; the counts end as degrees ----
    if (wid == 0) {
        uint32_t* words = reinterpret_cast<uint32_t*>(a.side + c0);  // x y z w per contact
        for (uint32_t e0 = 0; e0 < 2 * nc; e0 += 32) {
            const uint32_t e = e0 + lane;
            uint32_t* x = words + size_t(e >> 1) * 4 + (e & 1u);  // body; flags two words on
            const bool counts = e < 2 * nc && !(x[2] & (kFixed | kNoStore));
            const uint32_t body = counts ? x[0] : 0x80000000u | lane;
            const unsigned m = __match_any_sync(0xFFFFFFFFu, body);
            if (counts) x[2] |= B.count[body] + __popc(m & ((1u << lane) - 1u));
            __syncwarp();
            if (counts && lane == uint32_t(__ffs(m)) - 1u) B.count[body] += __popc(m);
            __syncwarp();
        }
    }
    __syncthreads();
    for (uint32_t i = t; i < nc; i += kThreads) {
        const uint4 x = a.side[c0 + i];
        const uint2 d{x.z & (kFixed | kNoStore) ? 0u : B.count[x.x], x.w & (kFixed | kNoStore) ? 0u : B.count[x.y]};
        a.degree[c0 + i] = d;
        atomicMax(&sh_deg, max(d.x, d.y));
    }
    __syncthreads();
    for (uint32_t i = t; i < nb; i += kThreads) B.count[i] = 0;
    __syncthreads();

    const AdjArgs f{c0, nc, t & 1u, t >> 1, kThreads / 2, k.pgs_iterations, &sh_left};
    adjoint_forward(s, a, f, B);
    __syncthreads();

    // ---- integration (physics.comp:586-604), reversed ----
    for (uint32_t i = t; i < nb; i += kThreads) {
        const uint32_t b = b0 + i;
        const d3 Gp1 = ldd3(g.pos, b);
        d3 Gv = ldd3(g.vel, b), Gw = ldd3(g.omega, b);
        const double Gq1[4] = {g.quat[size_t(b) * 4], g.quat[size_t(b) * 4 + 1],
                               g.quat[size_t(b) * 4 + 2], g.quat[size_t(b) * 4 + 3]};
        double Gq[4] = {Gq1[0], Gq1[1], Gq1[2], Gq1[3]};
        if (w.inv_mass[b] > 0.0f) {
            Gv += double(dt) * Gp1;  // pos += vel dt
            const float4 o = B.w[i];
            const float ox = o.x, oy = o.y, oz = o.z;
            const float qx = w.quat[size_t(b) * 4], qy = w.quat[size_t(b) * 4 + 1],
                        qz = w.quat[size_t(b) * 4 + 2], qw = w.quat[size_t(b) * 4 + 3];
            const float dx = ox * qw + oy * qz - oz * qy;
            const float dy = -ox * qz + oy * qw + oz * qx;
            const float dzq = ox * qy - oy * qx + oz * qw;
            const float dw = -ox * qx - oy * qy - oz * qz;
            const float ux = qx + 0.5f * dx * dt, uy = qy + 0.5f * dy * dt,
                        uz = qz + 0.5f * dzq * dt, uw = qw + 0.5f * dw * dt;
            const float l = sqrtf(ux * ux + uy * uy + uz * uz + uw * uw);
            double gu[4] = {Gq1[0], Gq1[1], Gq1[2], Gq1[3]};
            if (l > 1e-8f) {  // q' = u / |u|
                const double ld = l;
                const double nq[4] = {ux / ld, uy / ld, uz / ld, uw / ld};
                const double dp = nq[0] * Gq1[0] + nq[1] * Gq1[1] + nq[2] * Gq1[2] + nq[3] * Gq1[3];
                for (int j = 0; j < 4; ++j) gu[j] = (Gq1[j] - nq[j] * dp) / ld;
            }
            const double hdt = 0.5 * double(dt);
            const double gdx = hdt * gu[0], gdy = hdt * gu[1], gdz = hdt * gu[2], gdw = hdt * gu[3];
            const double Ox = ox, Oy = oy, Oz = oz, Qx = qx, Qy = qy, Qz = qz, Qw = qw;
            Gq[0] = gu[0] + gdy * Oz - gdz * Oy - gdw * Ox;
            Gq[1] = gu[1] - gdx * Oz + gdz * Ox - gdw * Oy;
            Gq[2] = gu[2] + gdx * Oy - gdy * Ox - gdw * Oz;
            Gq[3] = gu[3] + gdx * Ox + gdy * Oy + gdz * Oz;
            Gw.x += gdx * Qw - gdy * Qz + gdz * Qy - gdw * Qx;
            Gw.y += gdx * Qz + gdy * Qw - gdz * Qx - gdw * Qy;
            Gw.z += -gdx * Qy + gdy * Qx + gdz * Qw - gdw * Qz;
        }
        put3(B.g + size_t(i) * 6, Gv);
        put3(B.g + size_t(i) * 6 + 3, Gw);
        for (int j = 0; j < 4; ++j) a.gq[size_t(b) * 4 + j] = Gq[j];
        std3(a.gp, b, Gp1);
        for (int j = 0; j < 9; ++j) a.gR[size_t(b) * 9 + j] = 0.0;
        B.count[i] = 0;
    }
    if (t == 0) sh_left = 0;
    __syncthreads();

    adjoint_reverse(s, a, f, B);
    __syncthreads();

    // ---- contact constants and contact geometry, reversed ----
    for (uint32_t i = t; i < nc; i += kThreads)
        if (!(a.side[c0 + i].z & kSkip)) adjoint_contact(w, k, s, a, c0 + i, dt);
    __syncthreads();

    // ---- the sides' gradients summed at their bodies: dynamic ones a rank at a
    // time (contacts of one rank touch different bodies), fixed ones in contact
    // order, a lane per component ----
    const uint32_t maxdeg = sh_deg;
    for (uint32_t r = 0; r < maxdeg; ++r) {
        for (uint32_t e = t; e < 2 * nc; e += kThreads) {
            const uint32_t c = c0 + (e >> 1), side = e & 1u;
            const uint4 x = a.side[c];
            const uint32_t z = side ? x.w : x.z, l = side ? x.y : x.x;
            if ((z & (kFixed | kNoStore)) || (z & kRankMask) != r) continue;
            const double* o = side_slot(a, c, side);
            for (int q = 0; q < 6; ++q) B.g[size_t(l) * 6 + q] += o[q];
            double* p = a.gp + size_t(b0 + l) * 3;
            for (int q = 0; q < 3; ++q) p[q] += o[6 + q];
            double* R = a.gR + size_t(b0 + l) * 9;
            for (int q = 0; q < 9; ++q) R[q] += o[9 + q];
            g.friction[side ? w.c_b[c] : w.c_a[c]] += o[18];
        }
        __syncthreads();
    }
    if (wid == 0) {
        uint32_t cur = kNone, geom = kNone;  // the body and geom whose sums the lanes hold
        double sum = 0.0, fr = 0.0;
        double* at = nullptr;
        for (uint32_t e0 = 0; e0 < 2 * nc; e0 += 32) {
            const uint32_t e = min(e0 + lane, 2 * nc - 1), c = c0 + (e >> 1), side = e & 1u;
            const uint4 x = a.side[c];
            const uint32_t z = side ? x.w : x.z, l = side ? x.y : x.x;
            const uint32_t gi = side ? w.c_b[c] : w.c_a[c];
            // fixed bodies, and the side of a body that touches itself
            unsigned m = __ballot_sync(0xFFFFFFFFu, e0 + lane < 2 * nc && !(z & kSkip) &&
                                                        (z & (kFixed | kNoStore)) != 0u);
            while (m) {
                const uint32_t q = uint32_t(__ffs(m)) - 1u;
                m &= m - 1u;
                const uint32_t body = __shfl_sync(0xFFFFFFFFu, l, q), gq = __shfl_sync(0xFFFFFFFFu, gi, q);
                const double val = lane < 19u ? side_slot(a, c0 + ((e0 + q) >> 1), (e0 + q) & 1u)[lane] : 0.0;
                if (body != cur) {
                    if (at) *at = sum;
                    cur = body;
                    at = lane < 6u    ? B.g + size_t(body) * 6 + lane
                         : lane < 9u  ? a.gp + size_t(b0 + body) * 3 + lane - 6
                         : lane < 18u ? a.gR + size_t(b0 + body) * 9 + lane - 9
                                      : nullptr;
                    if (at) sum = *at;
                }
                if (gq != geom) {
                    if (lane == 18u && geom != kNone) g.friction[geom] = fr;
                    geom = gq;
                    if (lane == 18u) fr = g.friction[geom];
                }
                sum += val;
                fr += val;
            }
        }
        if (at) *at = sum;
        if (lane == 18u && geom != kNone) g.friction[geom] = fr;
    }
    __syncthreads();

    // ---- rotations -> quaternions, gravity (physics.comp:418-428), reversed
    for (uint32_t i = t; i < nb; i += kThreads) {
        const uint32_t b = b0 + i;
        double gq[4];
        quat_bwd(w.quat[size_t(b) * 4], w.quat[size_t(b) * 4 + 1], w.quat[size_t(b) * 4 + 2],
                 w.quat[size_t(b) * 4 + 3], a.gR + size_t(b) * 9, gq);
        for (int j = 0; j < 4; ++j) g.quat[size_t(b) * 4 + j] = a.gq[size_t(b) * 4 + j] + gq[j];
        d3 Gv = get3(B.g + size_t(i) * 6), Gw = get3(B.g + size_t(i) * 6 + 3);
        if (w.inv_mass[b] > 0.0f) {
            Gv = double(k.lin_damp) * Gv;
            Gw = double(k.ang_damp) * Gw;
        }
        std3(g.vel, b, Gv);
        std3(g.omega, b, Gw);
        std3(g.pos, b, ldd3(a.gp, b));
    }
}

constexpr uint32_t kAdjSmemBodies = 1024;

}  // namespace

cudaError_t init_adjoint() {
    const int bytes = int(kAdjSmemBodies * adj_body_bytes());
    for (const void* f : {reinterpret_cast<const void*>(k_adjoint<1>),
                          reinterpret_cast<const void*>(k_adjoint<2>),
                          reinterpret_cast<const void*>(k_adjoint<4>),
                          reinterpret_cast<const void*>(k_adjoint<8>)}) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Two lanes for every contact of the largest bundle where it holds about a quarter
// contact per body; larger ones give each pair several.
int launch_adjoint(const World& w, const Consts& k, const Scratch& s, const AdjScratch& a,
                   const Grads& g, float dt, uint32_t max_bundle, cudaStream_t st) {
    if (w.nbundles == 0) return 0;
    const uint32_t nbmax = max_bundle <= kAdjSmemBodies ? std::max(max_bundle, 1u) : 0u;
    const size_t smem = nbmax * adj_body_bytes();
    if (max_bundle <= 128) k_adjoint<1><<<w.nbundles, 32, smem, st>>>(w, k, s, a, g, dt, nbmax);
    else if (max_bundle <= 192) k_adjoint<2><<<w.nbundles, 64, smem, st>>>(w, k, s, a, g, dt, nbmax);
    else if (max_bundle <= 256) k_adjoint<4><<<w.nbundles, 128, smem, st>>>(w, k, s, a, g, dt, nbmax);
    else k_adjoint<8><<<w.nbundles, 256, smem, st>>>(w, k, s, a, g, dt, nbmax);
    return 1;
}

}  // namespace seevr
