// solver.cuh — one PGS contact update (physics.comp:525-580): over a view of
// the body state (solve_core: the island solvers), and over a contact's record
// with the branch-free divisions (update: the bundle solver and the adjoint).
#pragma once
#include "common.cuh"

namespace seevr {

struct BodyView {
    float* v;           // [n*3]
    float* w;           // [n*3]
    const float* R;     // [n*9]
    const float* invI;  // [n*3]
    const float* invm;  // [n]
};

__device__ __forceinline__ bool is_fixed(const BodyView& B, uint32_t i) {
    return B.invm[i] == 0.0f && B.invI[i * 3] == 0.0f && B.invI[i * 3 + 1] == 0.0f &&
           B.invI[i * 3 + 2] == 0.0f;
}

// One normal + friction update of contact c (physics.comp:525-580), given
// the two bodies' constant data; v, w: velocities and angular velocities,
// indexed by la / lb; a fixed body's velocities are not written.
__device__ __forceinline__ void solve_core(float* V, float* W, uint32_t la, uint32_t lb, bool fixed_a,
                                           bool fixed_b, float ima, float imb, const m3& Ra,
                                           const m3& Rb, f3 Ia, f3 Ib, f3 n, f3 ra, f3 rb,
                                           float bias, float kn, float mu, float* lam) {
    f3 va = ld3(V, la), wa = ld3(W, la), vb = ld3(V, lb), wb = ld3(W, lb);
    f3 ua = add(va, cross(wa, ra)), ub = add(vb, cross(wb, rb));
    const float vn = dot(sub(ub, ua), n);
    float d_ln = (-vn + bias) / kn;
    const float old_ln = *lam;
    const float new_ln = gmax(old_ln + d_ln, 0.0f);
    d_ln = new_ln - old_ln;
    *lam = new_ln;
    const f3 imp = scale(d_ln, n);
    va = sub(va, scale(ima, imp));
    vb = add(vb, scale(imb, imp));
    wa = sub(wa, apply_inv_I(Ra, Ia, cross(ra, imp)));
    wb = add(wb, apply_inv_I(Rb, Ib, cross(rb, imp)));
    // Coulomb friction along the current slip direction
    ua = add(va, cross(wa, ra));
    ub = add(vb, cross(wb, rb));
    const f3 dv = sub(ub, ua);
    const f3 vt = sub(dv, scale(dot(dv, n), n));
    const float vt_len = length(vt);
    if (vt_len > 1e-6f) {
        const f3 td = divs(vt, vt_len);
        const f3 rat = cross(ra, td), rbt = cross(rb, td);
        const float kt = ima + imb + dot(rat, apply_inv_I(Ra, Ia, rat)) + dot(rbt, apply_inv_I(Rb, Ib, rbt));
        const float d_lt = gmin(vt_len / kt, mu * new_ln);
        const f3 it = scale(d_lt, td);
        va = add(va, scale(ima, it));
        vb = sub(vb, scale(imb, it));
        wa = add(wa, apply_inv_I(Ra, Ia, cross(ra, it)));
        wb = sub(wb, apply_inv_I(Rb, Ib, cross(rb, it)));
    }
    if (!fixed_a) {
        st3(V, la, va);
        st3(W, la, wa);
    }
    if (!fixed_b) {
        st3(V, lb, vb);
        st3(W, lb, wb);
    }
}

__device__ __forceinline__ void solve_one(const BodyView& B, uint32_t la, uint32_t lb, f3 n, f3 ra,
                                          f3 rb, float bias, float kn, float mu, float* lam) {
    solve_core(B.v, B.w, la, lb, is_fixed(B, la), is_fixed(B, lb), B.invm[la], B.invm[lb],
               ld_m3(B.R, la), ld_m3(B.R, lb), ld3(B.invI, la), ld3(B.invI, lb), n, ra, rb, bias,
               kn, mu, lam);
}

// ---- updates by record ---------------------------------------------------------
// What an update of a contact reads besides the velocities (physics.comp:504-521,
// 533-546); kRecWords float4 in memory.
struct Side {
    f3 r, I;
    m3 R;
    float m;
};
struct Rec {
    f3 n;
    float bias, kn, rk, mu, msum;  // rk = 1 / kn, 0 when kn is out of div_by's range
    Side a, b;
};
// (Words `stride` apart: 1 in lists of whole records.)
__device__ __forceinline__ Side load_side(const float4* p, uint32_t stride) {
    const float4 c = p[0], d = p[stride], e = p[2 * stride], f = p[3 * stride];
    return Side{mk(c.x, c.y, c.z), mk(f.x, f.y, f.z),
                m3{mk(c.w, d.x, d.y), mk(d.z, d.w, e.x), mk(e.y, e.z, e.w)}, f.w};
}
__device__ __forceinline__ void store_side(float4* p, uint32_t stride, const Side& s) {
    p[0] = make_float4(s.r.x, s.r.y, s.r.z, s.R.c0.x);
    p[stride] = make_float4(s.R.c0.y, s.R.c0.z, s.R.c1.x, s.R.c1.y);
    p[2 * stride] = make_float4(s.R.c1.z, s.R.c2.x, s.R.c2.y, s.R.c2.z);
    p[3 * stride] = make_float4(s.I.x, s.I.y, s.I.z, s.m);
}
__device__ __forceinline__ Rec load_rec(const float4* p, uint32_t stride = 1) {
    const float4 a = p[0], b = p[stride];
    return Rec{mk(a.x, a.y, a.z), a.w, b.x, b.y, b.z, b.w, load_side(p + 2 * stride, stride),
               load_side(p + 6 * stride, stride)};
}

// Contact c's record: the constants, computed from the pre-solve velocities
// (va, wa, vb, wb), and both bodies' data.  The rotation matrices are those
// quat_to_mat gives at every update of the sweep, built once.
__device__ __forceinline__ void make_rec(const World& w, const Consts& k, uint32_t c, uint32_t a,
                                         uint32_t b, f3 va, f3 wa, f3 vb, f3 wb, float dt,
                                         float4* out, uint32_t stride = 1) {
    const uint32_t ga = w.c_a[c], gb = w.c_b[c];
    const f3 n = ld3(w.c_normal, c), cp = ld3(w.c_pos, c);
    const Side A{sub(cp, ld3(w.pos, a)), ld3(w.inv_inertia, a), quat_to_mat(w.quat, a), w.inv_mass[a]};
    const Side B{sub(cp, ld3(w.pos, b)), ld3(w.inv_inertia, b), quat_to_mat(w.quat, b), w.inv_mass[b]};
    const f3 ua = add(va, cross(wa, A.r)), ub = add(vb, cross(wb, B.r));
    const float vn = dot(sub(ub, ua), n);
    const float e = gmax(w.restitution[ga], w.restitution[gb]);
    const float bias = k.baumgarte * gmax(w.c_pen[c] - k.slop, 0.0f) / dt + e * gmax(-vn, 0.0f);
    const f3 ran = cross(A.r, n), rbn = cross(B.r, n);
    const float msum = A.m + B.m;
    const float kn = msum + dot(ran, apply_inv_I(A.R, A.I, ran)) + dot(rbn, apply_inv_I(B.R, B.I, rbn));
    const float rk = kn >= kDivMin && kn <= kDivMax ? recip_of(kn, rcp_approx(kn)) : 0.0f;
    out[0] = make_float4(n.x, n.y, n.z, bias);
    out[stride] = make_float4(kn, rk, sqrtf(w.friction[ga] * w.friction[gb]), msum);
    store_side(out + 2 * stride, stride, A);
    store_side(out + 6 * stride, stride, B);
}

// One update (solve_core's operations in solve_core's order).  kBuiltin: with the
// built-in square root and divisions; else the result tells whether every
// argument was in the branch-free ones' ranges.
template <bool kBuiltin>
__device__ __forceinline__ bool update_core(const Rec& h, f3& va, f3& wa, f3& vb, f3& wb, float& lam) {
    const Side &A = h.a, &B = h.b;
    f3 ua = add(va, cross(wa, A.r)), ub = add(vb, cross(wb, B.r));
    const float num = -dot(sub(ub, ua), h.n) + h.bias;
    float d = kBuiltin ? num / h.kn : div_by(num, h.kn, h.rk);
    const float ln = gmax(lam + d, 0.0f);
    d = ln - lam;
    lam = ln;
    const f3 imp = scale(d, h.n);
    va = sub(va, scale(A.m, imp));
    vb = add(vb, scale(B.m, imp));
    wa = sub(wa, apply_inv_I(A.R, A.I, cross(A.r, imp)));
    wb = add(wb, apply_inv_I(B.R, B.I, cross(B.r, imp)));
    // Coulomb friction along the current slip direction
    ua = add(va, cross(wa, A.r));
    ub = add(vb, cross(wb, B.r));
    const f3 dv = sub(ub, ua);
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
    const f3 rat = cross(A.r, td), rbt = cross(B.r, td);
    const float kt = h.msum + dot(rat, apply_inv_I(A.R, A.I, rat)) + dot(rbt, apply_inv_I(B.R, B.I, rbt));
    const float dl = gmin(kBuiltin ? len / kt : div_by(len, kt, recip_of(kt, rcp_approx(kt))),
                          h.mu * ln);
    const f3 it = scale(dl, td);
    const f3 va2 = add(va, scale(A.m, it)), vb2 = sub(vb, scale(B.m, it));
    const f3 wa2 = add(wa, apply_inv_I(A.R, A.I, cross(A.r, it)));
    const f3 wb2 = sub(wb, apply_inv_I(B.R, B.I, cross(B.r, it)));
    if (slips) {
        va = va2;
        vb = vb2;
        wa = wa2;
        wb = wb2;
    }
    if (kBuiltin) return true;
    // a NaN fails every comparison; the slip's components are at most len
    const uint32_t key = min(min(size_key(vt.x), size_key(vt.y)), size_key(vt.z));
    return h.rk != 0.0f && size_key(num) >= kNumMinKey && fabsf(num) <= kNumMax &&
           (still || (len2 <= kRootMax && key >= kNumMinKey && kt >= kDivMin && kt <= kDivMax));
}

// A contact's velocities and impulse during the solve.
struct State {
    f3 va, wa, vb, wb;
    float lam;
};
static __device__ __noinline__ void update_builtin(const Rec* h, State* x) {
    update_core<true>(*h, x->va, x->wa, x->vb, x->wb, x->lam);
}
// The update of the lanes that count (the others' result is not used).
__device__ __forceinline__ State update(const Rec& h, bool counts, const State& x) {
    State y = x;
    const bool ok = update_core<false>(h, y.va, y.wa, y.vb, y.wb, y.lam);
    if (counts && !ok) {
        const Rec copy = h;
        State z = x;
        update_builtin(&copy, &z);
        y = z;
    }
    return y;
}

}  // namespace seevr
