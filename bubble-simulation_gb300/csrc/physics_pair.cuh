// Device-side physics of two lattice cells at once (fast arithmetic, FP32).
//
// The fast bag forms (plain, MIXED, perturbation), gamma law and thermal
// potential of physics.cuh on pairs of cells: every quantity is a float2 whose halves belong to two different
// cells, so the paired FP32 instructions of sm_100+ (two IEEE operations per
// issue slot) carry the whole solver, with no exchange between the halves.
// The formulas are those of the shaders cited in physics.cuh; every rounding
// is explicit, so each call site computes the same bits.
//
// The rarely needed parts -- primitive recovery above gamma = 3 or at the
// pressure floor (with the FP64 recovery of the MIXED and perturbation forms
// and the |Z| cap) and the velocity clamp of a face state -- are decided by one
// test per pair.
#pragma once

#include "physics.cuh"

namespace bubble {
namespace dev {

// A 4-vector of each of two cells: component pairs.
struct P4 {
    float2 x, y, z, w;
};

BUBBLE_DEV P4 pair_of(const float4 &a, const float4 &b) {
    return P4{make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
}
BUBBLE_DEV float4 pair_a(const P4 &q) { return make_float4(q.x.x, q.x.y, q.y.x, q.y.y); }
BUBBLE_DEV float4 pair_b(const P4 &q) { return make_float4(q.z.x, q.z.y, q.w.x, q.w.y); }

BUBBLE_DEV float2 rcp2(float2 a) { return make_float2(rcp_approx(a.x), rcp_approx(a.y)); }
BUBBLE_DEV float2 sqrt2(float2 a) { return make_float2(sqrt_approx(a.x), sqrt_approx(a.y)); }
BUBBLE_DEV float2 max2(float2 a, float s) { return make_float2(fmaxf(a.x, s), fmaxf(a.y, s)); }
BUBBLE_DEV float2 dot3_2(float2 x, float2 y, float2 z) { return p_fma(z, z, p_fma(y, y, p_mul(x, x))); }

// min(|a|, |b|) with the product of the signs; the other operand, or (KEEP_NAN) NaN,
// where one is NaN
template <bool KEEP_NAN = false>
BUBBLE_DEV float min_xorsign(float a, float b) {
    float r;
    if constexpr (KEEP_NAN) asm("min.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    else asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// the smaller, the larger of both, NaN if either is
BUBBLE_DEV float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
BUBBLE_DEV float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Half of the MC-limited slope (limit_slope): 0 unless dm and dp have one
// sign, else min(|dm + dp| / 4, |dm|, |dp|) with it.  The signed minimum
// min(|dm|, |dp|) sign(dm dp), floored at 0, is 0 exactly when the signs
// differ, so no comparison is needed: three instructions per value.  0 also
// beside a cell that is NaN, so NaN spreads no further than the stencil.
BUBBLE_DEV float half_slope(float dm, float dp, float quarter_sum) {
    return min_xorsign(quarter_sum, fmaxf(min_xorsign<true>(dm, dp), 0.0f));
}
BUBBLE_DEV float2 half_slope2(float2 qm, float2 q, float2 qp) {
    const float2 dm = p_sub(q, qm), dp = p_sub(qp, q);
    const float2 h = p_mul(p_add(dm, dp), bc2(0.25f));
    return make_float2(half_slope(dm.x, dp.x, h.x), half_slope(dm.y, dp.y, h.y));
}

// The two face states of a pair along one axis (face_states<FAST>): lo = q -
// s/2, hi = q + s/2, pressure floored; the velocity clamp is hll_pair's.
BUBBLE_DEV void face_states_pair(const P4 &qm, const P4 &q, const P4 &qp, float p_floor, P4 &lo, P4 &hi) {
    const float2 sx = half_slope2(qm.x, q.x, qp.x), sy = half_slope2(qm.y, q.y, qp.y);
    const float2 sz = half_slope2(qm.z, q.z, qp.z), sw = half_slope2(qm.w, q.w, qp.w);
    lo = P4{p_sub(q.x, sx), p_sub(q.y, sy), p_sub(q.z, sz), max2(p_sub(q.w, sw), p_floor)};
    hi = P4{p_add(q.x, sx), p_add(q.y, sy), p_add(q.z, sz), max2(p_add(q.w, sw), p_floor)};
}

// ---------------------------------------------------------------------------
//  Thermal potential: temperature of two cells
// ---------------------------------------------------------------------------
// thermal_temperature of one cell: eight bounded steps.  Out of line: only
// where the short iteration below did not converge.
static __device__ __noinline__ float temperature_slow(float p, float phi, float th_k, float th_g, float th_h, float th_lo,
                                               float p_floor) {
    LatticeParams<float> P{};
    P.th_k = th_k;
    P.th_g = th_g;
    P.th_h = th_h;
    P.th_lo = th_lo;
    P.p_floor = p_floor;
    return thermal_temperature<float, true>(p, phi, P);
}

// The phi-dependent constants of p(T) = k T^4 - b T^2 + h T (b = gamma phi^2 / 2, h = A phi^3 / 3).
struct ThermalPair {
    float2 phi, b, h;
};
BUBBLE_DEV ThermalPair thermal_pair(float2 phi, const LatticeParams<float> &P) {
    const float2 f2 = p_mul(phi, phi);
    return ThermalPair{phi, p_mul(bc2(0.5f * P.th_g), f2), p_mul(bc2(P.th_h), p_mul(f2, phi))};
}
// dp/dT = T (4k T^2 - 2b) + h
BUBBLE_DEV float2 thermal_dp(float2 t, float2 t2, const ThermalPair &f, const LatticeParams<float> &P) {
    return p_fma(t, p_fma(bc2(4.0f * P.th_k), t2, p_mul(bc2(-2.0f), f.b)), f.h);
}
// One Newton step of p(T) = p; returns the step.
BUBBLE_DEV float2 thermal_step(float2 &t, float2 p, const ThermalPair &f, const LatticeParams<float> &P) {
    const float2 t2 = p_mul(t, t);
    const float2 g = p_fma(p_fma(bc2(P.th_k), t2, p_mul(bc2(-1.0f), f.b)), t2, p_sub(p_mul(f.h, t), p));
    const float2 d = p_mul(g, rcp2(thermal_dp(t, t2, f, P)));
    t = p_sub(t, d);
    return d;
}
// eos_temperature(p, phi).  Newton's steps converge quadratically from the phi
// = 0 root: where the first is below 1e-4 T its successor is below rounding
// (all of the symmetric phase); otherwise three more follow, and a cell whose
// last step is still above 2e-4 T takes the bounded iteration.  So does a cell
// that left the branch T >= lo |phi|.  The early step can end off it only for A
// below 1.5 gamma lo, where the phi = 0 root itself solves p(T, phi) = p at T = 2
// A phi / (3 gamma) < lo phi (for A >= 1.6 gamma lo a first step from off the
// branch is above 2e-2 T); only there is it tested (96^3 step 177.7 us, 181
// tested always).  Values accepted early are within 1.1e-7 T of the root, later
// ones within 2.2e-7, as the bounded iteration's are (FP32 rounding against 64
// bits, T from the branch limit to 1.3 T_ref, -0.3 <= phi/phi_b <= 1.2 and the
// validated gamma and A).  Each half is decided on its own values, so a pair's
// halves do not affect each other.
BUBBLE_DEV float2 temperature_pair(float2 p, const ThermalPair &f, const LatticeParams<float> &P) {
    const float2 t0 = sqrt2(sqrt2(p_mul(p, bc2(P.th_ik))));
    float2 t1 = t0;
    const float2 d1 = thermal_step(t1, p, f, P);
    const float lx = P.th_lo * fabsf(f.phi.x), ly = P.th_lo * fabsf(f.phi.y);
    bool cx = fabsf(d1.x) <= 1e-4f * t1.x, cy = fabsf(d1.y) <= 1e-4f * t1.y;
    if (P.th_a < 1.6f * P.th_g * P.th_lo) {
        cx = cx && t1.x >= lx;
        cy = cy && t1.y >= ly;
    }
    if (cx && cy) return t1;
    float2 t = t1;
    thermal_step(t, p, f, P);
    thermal_step(t, p, f, P);
    const float2 d = thermal_step(t, p, f, P);
    if (!cx && !(fabsf(d.x) <= 2e-4f * t.x && t.x >= lx))
        t.x = temperature_slow(p.x, f.phi.x, P.th_k, P.th_g, P.th_h, P.th_lo, P.p_floor);
    if (!cy && !(fabsf(d.y) <= 2e-4f * t.y && t.y >= ly))
        t.y = temperature_slow(p.y, f.phi.y, P.th_k, P.th_g, P.th_h, P.th_lo, P.p_floor);
    return make_float2(cx ? t1.x : t.x, cy ? t1.y : t.y);
}

// ---------------------------------------------------------------------------
//  Primitive recovery
// ---------------------------------------------------------------------------
// One cell through the scalar recovery (|Z| cap, FP64 above gamma = 3,
// velocity clamp).  Out of line: rarely taken and long.
// c0, c1 are e_bg and p_bg, or eos_c2 and eos_e0 of the gamma law.
template <int FORM>
__device__ __noinline__ V4<float> recover_slow(V4<float> u, float e_floor, float z_max, float p_floor, float c0,
                                               float c1) {
    LatticeParams<float> P{};
    P.e_floor = e_floor;
    P.z_max = z_max;
    P.p_floor = p_floor;
    if constexpr (FORM == kGamma) {
        P.eos_c2 = c0;
        P.eos_e0 = c1;
    } else {
        P.e_bg = c0;
        P.p_bg = c1;
    }
    return recover_sanitised<float, true, FORM>(u, P, 0.0f, z_max * z_max);
}

// The same for the thermal potential, whose recovery depends on phi.
static __device__ __noinline__ V4<float> recover_slow_thermal(V4<float> u, float phi, float e_floor, float z_max,
                                                       float p_floor, float th_k, float th_g, float th_h,
                                                       float th_i2a, float a_rad) {
    LatticeParams<float> P{};
    P.e_floor = e_floor;
    P.z_max = z_max;
    P.p_floor = p_floor;
    P.th_k = th_k;
    P.th_g = th_g;
    P.th_h = th_h;
    P.th_i2a = th_i2a;
    P.a_rad = a_rad;
    return recover_sanitised<float, true, kThermal>(u, P, phi, z_max * z_max);
}

// sanitise(recover(u)) of two cells in two parts, so independent work can be
// scheduled between them: recover_pair evaluates both cells by the formulas
// that hold below gamma = 3 and above the pressure floor, which it does not
// apply; recover_fix sends a cell whose |v|^2 came out above 8/9 (gamma > 3)
// or NaN, or whose p is below the floor or NaN, through the scalar recovery.  Together
// they cover every cell whose |Z| exceeds z_max E: the uncapped p of the bag
// forms and the gamma law is then below the floor, NaN, or so small that |v|^2
// is above 8/9 (where the floor is comparable to E, |v| alone can stay below);
// the thermal potential tests |Z| itself.
template <int FORM>
BUBBLE_DEV P4 recover_pair(const V4<float> &ua, const V4<float> &ub, float2 phi, const LatticeParams<float> &P) {
    const float2 de = max2(make_float2(ua.x, ub.x), P.e_floor);
    const float2 zx = make_float2(ua.y, ub.y), zy = make_float2(ua.z, ub.z), zz = make_float2(ua.w, ub.w);
    const float2 z2 = dot3_2(zx, zy, zz);
    if constexpr (FORM == kGamma) {
        // with s = E + p the closure is s^2 - B s + c2 Z^2 = 0, B = E + c2 (E -
        // e0), whose larger root the Newton steps of prim_from_cons_gamma
        // approach; p = c2 (E - e0 - Z^2 / s) keeps p's digits.  No real root
        // (NaN) and a p below the floor both go through recover_fix.  For B <= 0
        // the root is all cancellation, a few units of B's last place of either
        // sign; held at 0 it gives p = -inf or NaN, and a positive one gives p
        // below c2 (E - e0) < 0.
        const float2 x = p_sub(de, bc2(P.eos_e0));
        const float2 b = p_fma(bc2(P.eos_c2), x, de);
        const float2 sq = sqrt2(p_fma(b, b, p_mul(bc2(-4.0f * P.eos_c2), z2)));
        const float2 s = max2(p_mul(bc2(0.5f), p_add(b, sq)), 0.0f);
        const float2 p = p_mul(bc2(P.eos_c2), p_sub(x, p_mul(z2, rcp2(s))));
        const float2 inv = rcp2(p_add(de, p));
        return P4{p_mul(zx, inv), p_mul(zy, inv), p_mul(zz, inv), p};
    }
    if constexpr (FORM == kThermal) {
        // Newton on f(p) = p - p(T(e), phi) from the Z = 0 root, e = E - Z^2 / (E
        // + p): three steps; a cell whose last step is above 2e-4 p, or whose |Z|
        // is beyond the cap (cold cells have p > e there and |v| below the
        // threshold), gets v out of range, which sends it to recover_fix
        const ThermalPair f = thermal_pair(phi, P);
        const float2 a4 = bc2(4.0f * P.a_rad), b2 = p_mul(f.b, f.b);
        float2 p, dp = make_float2(0.0f, 0.0f), e = de, isp = dp;
#pragma unroll
        for (int it = 0; it <= 3; ++it) {
            if (it > 0) {
                isp = rcp2(p_add(de, p));
                e = p_sub(de, p_mul(z2, isp));
            }
            const float2 x = p_mul(p_add(f.b, sqrt2(p_fma(a4, e, b2))), bc2(P.th_i2a));
            const float2 t = sqrt2(x);
            const float2 pt = p_fma(p_sub(p_mul(bc2(P.th_k), x), f.b), x, p_mul(f.h, t));  // p(T(e), phi)
            if (it == 0) {
                p = max2(pt, P.p_floor);
            } else {
                const float2 dpt = thermal_dp(t, x, f, P);
                const float2 det = max2(p_mul(t, p_fma(a4, x, p_mul(bc2(-2.0f), f.b))), 1e-30f);
                float2 c2 = p_mul(dpt, rcp2(det));
                c2 = make_float2(fminf(fmaxf(c2.x, 1e-4f), 1.0f), fminf(fmaxf(c2.y, 1e-4f), 1.0f));
                const float2 d = p_fma(p_mul(c2, p_mul(z2, bc2(-1.0f))), p_mul(isp, isp), bc2(1.0f));
                dp = p_mul(p_sub(p, pt), rcp2(d));
                p = max2(p_sub(p, dp), P.p_floor);
            }
        }
        const float2 inv = rcp2(p_add(de, p));
        P4 q{p_mul(zx, inv), p_mul(zy, inv), p_mul(zz, inv), p};
        const float2 over = p_fma(p_mul(bc2(-P.z_max * P.z_max), de), de, z2);
        if (!(fabsf(dp.x) <= 2e-4f * p.x && over.x <= 0.0f)) q.x.x = 2.0f;
        if (!(fabsf(dp.y) <= 2e-4f * p.y && over.y <= 0.0f)) q.x.y = 2.0f;
        return q;
    }
    const float2 e = FORM == kPert ? p_add(bc2(P.e_bg), de) : de;
    const float2 sq = sqrt2(p_fma(p_mul(bc2(4.0f), e), e, p_mul(bc2(-3.0f), z2)));
    float2 p, s;
    if constexpr (FORM == kPert) {
        const float2 t = p_mul(z2, rcp2(p_fma(bc2(2.0f), e, sq)));
        p = p_fma(de, bc2((float)(1.0 / 3.0)), p_mul(t, bc2(-1.0f)));
        s = p_add(p_add(e, bc2(P.p_bg)), p);
    } else {
        p = p_mul(p_fma(e, e, p_mul(z2, bc2(-1.0f))), rcp2(p_add(e, sq)));
        s = p_add(e, p);
    }
    const float2 inv = rcp2(s);
    return P4{p_mul(zx, inv), p_mul(zy, inv), p_mul(zz, inv), p};
}
template <int FORM>
BUBBLE_DEV void recover_fix(P4 &q, const V4<float> *ua, const V4<float> *ub, float2 phi,
                            const LatticeParams<float> &P) {
    const float2 v2 = dot3_2(q.x, q.y, q.z);
    constexpr float kFast = 8.0f / 9.0f;
    const bool fast = !(max_nan(v2.x, v2.y) <= kFast);
    // the thermal form floors p and marks the cells itself
    const auto low = [&] { return FORM != kThermal && !(min_nan(q.w.x, q.w.y) >= P.p_floor); };
    // One branch or two, by what measured faster (us per step, one and two): plain
    // 32^3 17.15 and 17.27, 48^3 22.9 and 23.05, 128^3 159.4 and 160.0; mixed 256^3
    // 1129.5 and 1119.0, perturbation 1158.1 and 1157.2.
    constexpr bool kOneBranch = FORM == kPlain || FORM == kGamma;
    if (kOneBranch ? fast | low() : fast || low()) {
        auto slow = [&](const V4<float> *u, float f) {
            if constexpr (FORM == kThermal)
                return recover_slow_thermal(*u, f, P.e_floor, P.z_max, P.p_floor, P.th_k, P.th_g, P.th_h, P.th_i2a,
                                            P.a_rad);
            else
                return recover_slow<FORM>(*u, P.e_floor, P.z_max, P.p_floor, FORM == kGamma ? P.eos_c2 : P.e_bg,
                                          FORM == kGamma ? P.eos_e0 : P.p_bg);
        };
        if (!(v2.x <= kFast) || !(q.w.x >= P.p_floor)) {
            const V4<float> r = slow(ua, phi.x);
            q.x.x = r.x;
            q.y.x = r.y;
            q.z.x = r.z;
            q.w.x = r.w;
        }
        if (!(v2.y <= kFast) || !(q.w.y >= P.p_floor)) {
            const V4<float> r = slow(ub, phi.y);
            q.x.y = r.x;
            q.y.y = r.y;
            q.z.y = r.z;
            q.w.y = r.w;
        }
    }
}

// ---------------------------------------------------------------------------
//  HLL face flux of two faces along one axis
// ---------------------------------------------------------------------------
struct PairSide {
    P4 u, f;         // conserved state and flux along the axis
    float2 nlm, lp;  // minus the lower wave speed, the upper wave speed
};

// With c_s^2 = 1/3, D = 3 - v^2 and T = D - 2 vd^2 the wave speeds
// (2 vd -+ sqrt((1 - v^2) T)) / D are those of face_side: numerator and
// denominator scaled by 3.
template <int AXIS, int FORM>
BUBBLE_DEV PairSide pair_side(const P4 &q, float2 v2, float2 phi, const LatticeParams<float> &P) {
    PairSide s;
    const float2 vd = AXIS == 0 ? q.x : (AXIS == 1 ? q.y : q.z);
    const float2 p = q.w;
    const float2 om = p_sub(bc2(1.0f), v2);
    const float2 pf = FORM == kPert ? p_add(bc2(P.p_bg), p) : p;  // the full pressure
    float2 cs2 = om, enth = om;  // thermal: c_s^2 and the enthalpy density at T(p, phi)
    if constexpr (FORM == kThermal) {
        const ThermalPair f = thermal_pair(phi, P);
        const float2 t = temperature_pair(p, f, P), t2 = p_mul(t, t);
        enth = p_fma(p_sub(p_mul(bc2(P.a_rad), t2), f.b), t2, p);
        const float2 de = max2(p_mul(t, p_fma(bc2(4.0f * P.a_rad), t2, p_mul(bc2(-2.0f), f.b))), 1e-30f);
        cs2 = p_mul(thermal_dp(t, t2, f, P), rcp2(de));
        cs2 = make_float2(fminf(fmaxf(cs2.x, 1e-4f), 1.0f), fminf(fmaxf(cs2.y, 1e-4f), 1.0f));
    }
    const float2 w = p_mul(FORM == kThermal ? enth : FORM == kGamma ? p_fma(bc2(P.eos_k), p, bc2(P.eos_e0)) : p_mul(bc2(4.0f), pf), rcp2(om));
    s.u.x = FORM == kPert ? p_fma(w, v2, p_mul(bc2(3.0f), p)) : p_sub(w, p);
    s.u.y = p_mul(w, q.x);
    s.u.z = p_mul(w, q.y);
    s.u.w = p_mul(w, q.z);
    if constexpr (FORM == kThermal) {
        const float2 d = p_fma(v2, p_mul(cs2, bc2(-1.0f)), bc2(1.0f));
        const float2 inv = rcp2(d);
        const float2 tv = p_mul(vd, p_sub(cs2, bc2(1.0f)));
        const float2 sq = sqrt2(p_mul(cs2, p_mul(om, p_fma(tv, vd, d))));
        s.nlm = p_mul(p_add(sq, tv), inv);
        s.lp = p_mul(p_sub(sq, tv), inv);
    } else if constexpr (FORM == kGamma) {
        // the same with c_s^2 = c2, unscaled: D = 1 - c2 v^2, T = D - (1 - c2) vd^2
        const float2 d = p_fma(v2, bc2(-P.eos_c2), bc2(1.0f));
        const float2 inv = rcp2(d);
        const float2 tv = p_mul(vd, bc2(P.eos_c2 - 1.0f));
        const float2 sq = p_mul(bc2(P.eos_cs), sqrt2(p_mul(om, p_fma(tv, vd, d))));
        s.nlm = p_mul(p_add(sq, tv), inv);
        s.lp = p_mul(p_sub(sq, tv), inv);
    } else {
        const float2 d = p_sub(bc2(3.0f), v2);
        const float2 inv = rcp2(d);
        const float2 tv = p_mul(vd, bc2(-2.0f));
        const float2 sq = sqrt2(p_mul(om, p_fma(tv, vd, d)));
        s.nlm = p_mul(p_add(sq, tv), inv);
        s.lp = p_mul(p_sub(sq, tv), inv);
    }
    s.f.x = p_mul(w, vd);
    s.f.y = AXIS == 0 ? p_fma(s.u.y, vd, p) : p_mul(s.u.y, vd);
    s.f.z = AXIS == 1 ? p_fma(s.u.z, vd, p) : p_mul(s.u.z, vd);
    s.f.w = AXIS == 2 ? p_fma(s.u.w, vd, p) : p_mul(s.u.w, vd);
    return s;
}

// |v|^2 of a pair whose x and y components may be exchanged: the same bits
// either way.
BUBBLE_DEV float2 speed2(const P4 &q, bool exchanged) {
    return dot3_2(exchanged ? q.y : q.x, exchanged ? q.x : q.y, q.z);
}

// The velocity half of sanitise on the halves of a pair beyond the cap.
BUBBLE_DEV void clamp_pair(P4 &q, float2 &v2, float zmax2, bool exchanged) {
    float2 f;
    f.x = v2.x > zmax2 ? __fsqrt_rn(__fdiv_rn(zmax2, v2.x)) : 1.0f;
    f.y = v2.y > zmax2 ? __fsqrt_rn(__fdiv_rn(zmax2, v2.y)) : 1.0f;
    q.x = p_mul(q.x, f);
    q.y = p_mul(q.y, f);
    q.z = p_mul(q.z, f);
    v2 = speed2(q, exchanged);
    v2 = make_float2(fminf(v2.x, zmax2), fminf(v2.y, zmax2));
}

// One side of a face pair and its |v|^2.  `exchanged`: q holds (vy, vx, vz,
// p), for a y face taken as AXIS 0; the flux is then (E, Zy, Zx, Zz) with the
// bits of AXIS 1.
// fl, fr: the field in the two sides' own cells, read by the thermal form only.
struct FacePair {
    P4 l, r;
    float2 vl, vr, fl, fr;
};
BUBBLE_DEV FacePair face_pair(const P4 &l, const P4 &r, float2 fl, float2 fr, bool exchanged = false) {
    return FacePair{l, r, speed2(l, exchanged), speed2(r, exchanged), fl, fr};
}
// Whether a speed of a face pair is beyond the cap or NaN.
BUBBLE_DEV bool needs_clamp(const FacePair &f, float zmax2) {
    return !(max_nan(max_nan(f.vl.x, f.vl.y), max_nan(f.vr.x, f.vr.y)) <= zmax2);
}
// The velocity clamps of such a pair; |v|^2 of a NaN velocity is the cap's, so
// the components that are not NaN keep finite fluxes.
BUBBLE_DEV void clamp_face(FacePair &f, float zmax2, bool exchanged = false) {
    clamp_pair(f.l, f.vl, zmax2, exchanged);
    clamp_pair(f.r, f.vr, zmax2, exchanged);
}

template <int AXIS, int FORM>
BUBBLE_DEV P4 hll_pair(const FacePair &f, const LatticeParams<float> &P) {
    const PairSide L = pair_side<AXIS, FORM>(f.l, f.vl, f.fl, P);
    const PairSide R = pair_side<AXIS, FORM>(f.r, f.vr, f.fr, P);
    const float2 ns = make_float2(fmaxf(fmaxf(L.nlm.x, R.nlm.x), 0.0f), fmaxf(fmaxf(L.nlm.y, R.nlm.y), 0.0f));
    const float2 sx = make_float2(fmaxf(fmaxf(L.lp.x, R.lp.x), 0.0f), fmaxf(fmaxf(L.lp.y, R.lp.y), 0.0f));
    // (s_max f_L - s_min f_R + s_min s_max (u_R - u_L)) / (s_max - s_min)
    const float2 inv = rcp2(p_add(ns, sx));
    const float2 ca = p_mul(sx, inv), cb = p_mul(ns, inv);
    const float2 cc = p_mul(ns, ca);
    return P4{p_fma(ca, L.f.x, p_fma(cb, R.f.x, p_mul(cc, p_sub(L.u.x, R.u.x)))),
              p_fma(ca, L.f.y, p_fma(cb, R.f.y, p_mul(cc, p_sub(L.u.y, R.u.y)))),
              p_fma(ca, L.f.z, p_fma(cb, R.f.z, p_mul(cc, p_sub(L.u.z, R.u.z)))),
              p_fma(ca, L.f.w, p_fma(cb, R.f.w, p_mul(cc, p_sub(L.u.w, R.u.w))))};
}

}  // namespace dev
}  // namespace bubble
