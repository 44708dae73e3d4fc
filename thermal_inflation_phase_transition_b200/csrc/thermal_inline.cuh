// The thermal one-loop V' evaluated per site, as the reference's inline form
// _vprime_inline (R:2201-2266) that rk2_fused_single_pass (R:2339-2647) calls
// or (form 1) as Vprime_field (R:1435-1485) that rk2_step / rk2_step_fused call:
//   V' = lam phi^3 - mphi^2 phi + T^4/(2 pi^2) (cb dJ_B(x_b) dx_b/dphi + cf dJ_F(x_f) dx_f/dphi),
//   x_b = sqrt(mB^2 + gb^2 phi^2/2 + (gb^2/4 + 2 gg^2/3) T^2) / T,
//   x_f = sqrt(gf^2 phi^2/2 + gfg^2 T^2/6) / T,
// dJ from the cubic splines on the uniform grid x_min + i h: inline form x
// clamped to [x_min, xhi], xhi = x_min + h nseg - 1e-12, segment
// trunc((x - x_min) * (1/h)); field form x below x_min raised to x_min, x above
// x_min + h nseg lowered to x_min + h nseg - 1e-12, segment trunc((x - x_min) / h);
// the segment clamped to [0, nseg-1] in both.
// FP64.
#pragma once

#include "gauss64.cuh"
#include "tipt.h"

namespace tipt {

// Per-launch constants (computed on the host from tipt_thermal and T).
struct ThermalSite {
    const double* spline;  // [8][nseg]: dx^3, dx^2, dx, 1 coefficients of dJ_B, then dJ_F
    int nseg;
    int field_form;        // 1: the Vprime_field / cubic_eval_uniform clamp and segment rule
    double lam, mphi_sq, bms, gb2, gf2, gfg2, coef_b, coeff_b, coeff_f;
    double x_min, h, inv_hy, xhi, xtop;
    double T, T2, pref;
    // what the per-site evaluation needs of them: 1/T; the arguments' squares times T^2,
    // mass + half coupling * phi^2, and (half coupling / T) of the slopes
    double inv_T, mass_b, half_b, slope_b, mass_f, half_f, slope_f;
    double far_b, far_f;     // half coupling / (T^2 1e-20): the slopes where x < 1e-20
    double sq_lo, sq_hi;     // squares whose x needs no clamp
};

inline ThermalSite thermal_site(const tipt_thermal& t, double T) {
    ThermalSite s;
    s.spline = t.spline;
    s.nseg = t.nseg;
    s.lam = t.lam;
    s.mphi_sq = t.mphi * t.mphi;
    s.bms = t.boson_mass_sq;
    s.gb2 = t.boson_coupling * t.boson_coupling;
    const double gg2 = t.boson_gauge_coupling * t.boson_gauge_coupling;
    s.gf2 = t.fermion_coupling * t.fermion_coupling;
    s.gfg2 = t.fermion_gauge_coupling * t.fermion_gauge_coupling;
    s.coef_b = 0.25 * s.gb2 + (2.0 / 3.0) * gg2;  // R:2376
    s.coeff_b = t.coeff_b;
    s.coeff_f = t.coeff_f;
    s.x_min = t.x_min;
    s.h = t.h;
    s.inv_hy = 1.0 / t.h;                       // R:452
    s.xhi = t.x_min + t.h * t.nseg - 1e-12;     // R:453
    s.xtop = t.x_min + t.h * t.nseg;            // R:1467-1468
    s.field_form = t.form == 1;
    s.T = T;
    s.T2 = T * T;
    s.pref = s.T2 * s.T2 / (2.0 * 3.141592653589793 * 3.141592653589793);
    s.inv_T = 1.0 / T;
    s.mass_b = s.bms + s.coef_b * s.T2;
    s.half_b = 0.5 * s.gb2;
    s.slope_b = s.half_b / T;
    s.mass_f = (1.0 / 6.0) * s.gfg2 * s.T2;
    s.half_f = 0.5 * s.gf2;
    s.slope_f = s.half_f / T;
    s.far_b = s.half_b / (s.T2 * 1e-20);
    s.far_f = s.half_f / (s.T2 * 1e-20);
    // x in (max(x_min, 1e-20), x_top) with room for rounding; none when T is not a
    // normal positive number, or when x_min < 0: the room, relative to x_top, may then be
    // smaller than the rounding of x - x_min, and the segment has to be clamped
    const double lo = t.x_min > 1e-20 ? t.x_min : 1e-20, hi = s.xhi < s.xtop ? s.xhi : s.xtop;
    s.sq_lo = (lo * T) * (lo * T) * (1.0 + 1e-12);
    s.sq_hi = (hi * T) * (hi * T) * (1.0 - 1e-12);
    if (!(s.sq_lo >= 1e-300 && s.sq_hi <= 1e300 && T > 0.0 && t.x_min >= 0.0))
        s.sq_lo = 1.0, s.sq_hi = 0.0;
    return s;
}

// The cubic of segment si at xc.
__device__ __forceinline__ double thermal_cubic(const double* c, const ThermalSite& s, int si, double xc) {
    const double d = __dsub_rn(xc, __fma_rn((double)si, s.h, s.x_min));
    c += si;
    return __fma_rn(__fma_rn(__fma_rn(__ldg(c), d, __ldg(c + s.nseg)), d, __ldg(c + 2 * s.nseg)), d,
                    __ldg(c + 3 * s.nseg));
}
// (x - x_min) / h; the field form's quotient from the reciprocal and its remainder
__device__ __forceinline__ double thermal_pos(const ThermalSite& s, double x) {
    const double a = __dsub_rn(x, s.x_min), q = __dmul_rn(a, s.inv_hy);
    return s.field_form ? __fma_rn(__fma_rn(-q, s.h, a), s.inv_hy, q) : q;
}

// One species: dJ(x) dx/dphi for x = sqrt(sq) / T (0 where sq is not positive), dx/dphi =
// half phi / (T^2 max(x, 1e-20)) (R:2228-2262), dJ's segment by truncation.  x and the
// slope (half / T) phi / sqrt(sq) come from one reciprocal square root, x with the
// quotient's remainder added back.  Squares outside [sq_lo, sq_hi] (and NaN) take the
// form with every clamp: below 1e-300 they count as 0, above 1e300 as that; a NaN x
// takes segment 0 and gives NaN.
__device__ __forceinline__ double thermal_term(const double* c, const ThermalSite& s, double sq,
                                               double slope, double far, double ph) {
    double y, r, dj;
    if (sq >= s.sq_lo && sq <= s.sq_hi) {
        rsqrt_sqrt<true>(sq, y, r);
        const double q = __dmul_rn(r, s.inv_T);
        const double x = __fma_rn(__fma_rn(-q, s.T, r), s.inv_T, q);
        dj = thermal_cubic(c, s, (int)thermal_pos(s, x), x);
        y = __dmul_rn(slope, y);
    } else {
        const bool pos = sq >= 1e-300;
        rsqrt_sqrt<true>(pos ? fmin(sq, 1e300) : 1.0, y, r);
        const double q = __dmul_rn(r, s.inv_T);
        const double x = pos ? __fma_rn(__fma_rn(-q, s.T, r), s.inv_T, q) : 0.0;
        const double top = s.field_form ? s.xtop : s.xhi;
        // R:1464-1473 (field form: above x_top lowered to x_top - 1e-12), R:2238-2248
        const double xc = x < s.x_min ? s.x_min
                                      : (x > top ? (s.field_form ? s.xtop - 1e-12 : s.xhi) : x);
        const int si = (int)thermal_pos(s, xc);
        dj = thermal_cubic(c, s, si < 0 ? 0 : (si >= s.nseg ? s.nseg - 1 : si), xc);
        y = x >= 1e-20 ? __dmul_rn(slope, y) : far;
    }
    return __dmul_rn(dj, __dmul_rn(y, ph));
}

// What it costs bounds the thermal stages: two square roots and four divisions in FP64
// per evaluation in the reference's form, none here.  Every operation is an explicit
// round-to-nearest intrinsic (the kernels that call it give the same bits).  256^3
// float32, rk2_fused_single_pass (two halves, two evaluations a site each): 1254 us in
// the reference's form, 894 us here (694 -> 596 instructions a site from the clamps
// off the common path).
__device__ __forceinline__ double thermal_vprime_inline(const ThermalSite& s, double ph) {
    const double p2 = __dmul_rn(ph, ph);
    const double b = thermal_term(s.spline, s, __fma_rn(s.half_b, p2, s.mass_b), s.slope_b, s.far_b, ph);
    const double f = thermal_term(s.spline + 4 * s.nseg, s, __fma_rn(s.half_f, p2, s.mass_f), s.slope_f,
                                  s.far_f, ph);
    const double poly = __dmul_rn(ph, __fma_rn(s.lam, p2, -s.mphi_sq));
    return __fma_rn(s.pref, __fma_rn(s.coeff_b, b, __dmul_rn(s.coeff_f, f)), poly);
}

}  // namespace tipt
