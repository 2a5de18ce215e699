// FP64 HLL / HLL3 face fluxes with the correctly rounded
// straight-line division and root of exact64.cuh.
//
// The values and their order are those of euler_math.cuh (and so the
// reference's); only the way a quotient or root is computed differs, and
// it gives the same bits while the operands lie in the ranges tested here.
// A face outside them (vacuum, overflow, NaN, values below 2^-700
// that are not zero) reports it, and the caller evaluates the plain form.
//
// Why the tests suffice.  With both densities and pressures in
// [2^-60, 2^60) and gamma - 1 at least 2^-20: (gamma-1)(E - m.m/(2 rho)) = p,
// a difference rounded in the 53rd place, bounds E by 2^133, |m| and velocities
// by 2^97 and speeds by 2^98; normal momenta are 0 or at least 2^-700, so velocities, their Roe sums (a sum of doubles is 0 or at least
// the last place of its smallest operand) and every denominator below stay
// far from over- and underflow.  The kinetic energy m.m/(2 rho) may be
// subnormal, but only where it is lost against E whatever its last bits.
// The remaining numerators and denominators are tested one by one.
//
// Measured on a B200, ms per RK3 step with the compiler's operators and with
// these: KH 1024^2 0.370 and 0.279 (32 x 16 tiles), KH 128^3 1.14 and 0.84,
// Sod with 1,024 cells, a thousandth of that per step, 16.8 and 10.2 us.
#pragma once

#include "euler_math.cuh"
#include "exact64.cuh"

namespace als {

// What a face's straight-line evaluation leaves for the decision on it.
struct QuickFace {
    double pl, pr, vl, vr;   // pressures and normal velocities of the two sides
    double w;                // wave speed
    int hl, hr;              // high words of the two signal speeds
    bool base;               // both sides inside the tested ranges
    bool star;               // and sL < 0 < sR with every quotient in range: F holds the flux
};

// The face flux along D between ul and ur (face_flux of euler_math.cuh),
// without a branch: F is the star-state flux, which face_settle replaces
// where another one is due.
template<int NSD, int FLUX, int D>
__device__ __forceinline__ void face_quick(const double* ul, const double* ur, double gamma,
    double* F, QuickFace& Q) {
    constexpr int NV = NSD + 2;
    const double rl = ul[0], rr = ur[0];
    const double yl = rcp64(rl), yr = rcp64(rr);
    double dl = ul[1] * ul[1], dr = ur[1] * ur[1];
#pragma unroll
    for (int k = 1; k < NSD; ++k) {
        dl = dl + ul[1 + k] * ul[1 + k];
        dr = dr + ur[1 + k] * ur[1 + k];
    }
    const double pl = (gamma - 1.0) * (ul[NSD + 1] - quot64(0.5 * dl, rl, yl));
    const double pr = (gamma - 1.0) * (ur[NSD + 1] - quot64(0.5 * dr, rr, yr));
    const double vl = quot64(ul[1 + D], rl, yl);
    const double vr = quot64(ur[1 + D], rr, yr);
    // speeds: HLL3.hpp:120-160, HLL.hpp:51-116 (without the correction)
    const double cl = sqrt64(quot64(gamma * pl, rl, yl));
    const double cr = sqrt64(quot64(gamma * pr, rr, yr));
    const double wl = sqrt64(rl), wr = sqrt64(rr);
    const double ws = wl + wr, yw = rcp64(ws);
    const double rho = (rl + rr) * 0.5, yrho = rcp64(rho);
    const double v = quot64(wl * vl + wr * vr, ws, yw);
    const double p = quot64(wl * pl + wr * pr, ws, yw);
    const double cs = sqrt64(quot64(gamma * p, rho, yrho));
    double al, ar;
    if (FLUX == FLUX_HLL3) {
        const double dv = vl - vr;
        const double correct = 0.5 * (dv > 0.0 ? dv : 0.0);
        al = vl + correct - cl;
        ar = vr - correct + cr;
    } else {
        al = vl - cl;
        ar = vr + cr;
    }
    const double bl = v - cs, br = v + cs;
    const double sL = al < bl ? al : bl;
    const double sR = ar > br ? ar : br;

    // densities and pressures in [2^-60, 2^60), normal momenta 0 or not tiny,
    // an ordinary adiabatic exponent: gamma - 1 in [2^-20, 2^10)
    int lo = min(min(__double2hiint(rl), __double2hiint(rr)),
        min(__double2hiint(pl), __double2hiint(pr)));
    const int top = max(max(__double2hiint(rl), __double2hiint(rr)),
        max(__double2hiint(pl), __double2hiint(pr)));
    unsigned key = min(numerator_key(ul[1 + D]), numerator_key(ur[1 + D]));
    const int g1 = __double2hiint(gamma - 1.0);
    Q.base = top < hi_pow2(60) && lo >= hi_pow2(-60) && key >= unsigned(hi_pow2(-700)) - 1u &&
        g1 >= hi_pow2(-20) && g1 < hi_pow2(10);
    Q.pl = pl;
    Q.pr = pr;
    Q.vl = vl;
    Q.vr = vr;
    const double ml = fabs(sL), mr = fabs(sR);
    Q.w = ml > mr ? ml : mr;
    Q.hl = __double2hiint(sL);
    Q.hr = __double2hiint(sR);

    // the star state, whatever the signs of the speeds
    if (FLUX == FLUX_HLL) {
        const double den = sR - sL, y = rcp64(den);
        lo = min(lo, __double2hiint(den));
        const double ss = sR * sL;
        double fl[NV], fr[NV];
        fl[0] = ul[1 + D];
        fr[0] = ur[1 + D];
#pragma unroll
        for (int k = 0; k < NSD; ++k) {
            fl[1 + k] = ul[1 + k] * vl;
            fr[1 + k] = ur[1 + k] * vr;
        }
        fl[1 + D] = fl[1 + D] + pl;
        fr[1 + D] = fr[1 + D] + pr;
        fl[NV - 1] = (ul[NV - 1] + pl) * vl;
        fr[NV - 1] = (ur[NV - 1] + pr) * vr;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const double num = sR * fl[k] - sL * fr[k] + ss * (ur[k] - ul[k]);
            key = min(key, numerator_key(num));
            F[k] = quot64(num, den, y);
        }
    } else {
        const double ql = vl - sL, qr = vr - sR;
        const double aa = qr * rr - ql * rl;
        const int as = __double2hiint(aa) & int(0x80000000u);
        const double pa = fabs(aa), ya = rcp64(pa);
        lo = min(lo, __double2hiint(pa));
        const double sm = quot64(flip_sign(ur[1 + D] * qr - ul[1 + D] * ql + pr - pl, as), pa, ya);
        double us[NSD];
#pragma unroll
        for (int k = 0; k < NSD; ++k) {
            if (k == D) {
                us[k] = sm;
            } else {
                const double num = ur[1 + k] * vr - ul[1 + k] * vl - sR * ur[1 + k] + sL * ul[1 + k];
                key = min(key, numerator_key(num));
                us[k] = quot64(flip_sign(num, as), pa, ya);
            }
        }
        // the side of the contact the face lies on; its denominator
        // sm - s is positive on the left and negative on the right
        const bool left = sm >= 0.0;
        const int ss = left ? 0 : int(0x80000000u);
        const double s = left ? sL : sR;
        const double q = left ? ql : qr;
        const double pp = left ? pl : pr;
        const double vv = left ? vl : vr;
        double c[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            c[k] = left ? ul[k] : ur[k];
        }
        const double den = fabs(sm - s), y = rcp64(den);
        lo = min(lo, __double2hiint(den));
        const double n0 = c[0] * q;
        const double ps = pp + c[0] * (vv - sm) * q;
        const double ne = q * c[NV - 1] + pp * vv - ps * sm;
        key = min(key, min(numerator_key(n0), numerator_key(ne)));
        double mid[NV];
        mid[0] = quot64(flip_sign(n0, ss), den, y);
#pragma unroll
        for (int k = 0; k < NSD; ++k) {
            mid[1 + k] = us[k] * mid[0];
        }
        mid[NV - 1] = quot64(flip_sign(ne, ss), den, y);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double f = k == 0 ? c[1 + D] : (k == NV - 1 ? (c[NV - 1] + pp) * vv : c[k] * vv);
            if (k == 1 + D) {
                f = f + pp;
            }
            F[k] = f + s * (mid[k] - c[k]);
        }
    }
    // finite speeds here: the high words decide the signs, zeros excluded
    Q.star = Q.base && unsigned(Q.hl) > 0x80000000u && Q.hr > 0 && lo >= hi_pow2(-60) &&
        key >= unsigned(hi_pow2(-700)) - 1u;
}

// The plain form out of line: u holds the left and the right state.
template<int NSD, int FLUX, int D>
__device__ __noinline__ double face_flux_plain(const double* u, double gamma, double* F) {
    return face_flux<double, NSD, FLUX, D>(u, u + NSD + 2, gamma, F);
}

// The flux and wave speed of a face whose star state does not apply: the
// upwind point flux of a supersonic face, or the plain form.
template<int NSD, int FLUX, int D>
__device__ __forceinline__ void face_settle(const double* ul, const double* ur, double gamma,
    double* F, QuickFace& Q) {
    constexpr int NV = NSD + 2;
    if (Q.star) {
        return;
    }
    const bool left = Q.hl > 0;
    if (Q.base && (left || unsigned(Q.hr) > 0x80000000u)) {
        const double p = left ? Q.pl : Q.pr;
        const double v = left ? Q.vl : Q.vr;
        const double E = left ? ul[NV - 1] : ur[NV - 1];
        F[0] = left ? ul[1 + D] : ur[1 + D];
#pragma unroll
        for (int k = 0; k < NSD; ++k) {
            F[1 + k] = (left ? ul[1 + k] : ur[1 + k]) * v;
        }
        F[1 + D] = F[1 + D] + p;
        F[NV - 1] = (E + p) * v;
        return;
    }
    double u[2 * NV], f[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        u[v] = ul[v];
        u[NV + v] = ur[v];
    }
    Q.w = face_flux_plain<NSD, FLUX, D>(u, gamma, f);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        F[v] = f[v];
    }
}

// Whether a face has a straight-line form.
template<class R, int FLUX>
__host__ __device__ constexpr bool quick_face() {
    return sizeof(R) == 8 && (FLUX == FLUX_HLL || FLUX == FLUX_HLL3);
}

// face_flux with the straight-line form where there is one, and FP32 with the
// flushing reciprocals and roots where the face allows them.
template<class R, int NSD, int FLUX, int D>
__device__ __forceinline__ R face_flux_best(const R* ul, const R* ur, R gamma, R* F) {
    if constexpr (quick_face<R, FLUX>()) {
        QuickFace Q;
        face_quick<NSD, FLUX, D>(ul, ur, gamma, F, Q);
        face_settle<NSD, FLUX, D>(ul, ur, gamma, F, Q);
        return Q.w;
    } else if constexpr (fast_recip<R>() && (FLUX == FLUX_HLL || FLUX == FLUX_HLL3)) {
        FaceState<R, NSD> L, Rt;
        make_state<R, NSD, D, true>(ul, gamma, L);
        make_state<R, NSD, D, true>(ur, gamma, Rt);
        return flux_between<R, NSD, FLUX, D, true>(L, Rt, gamma, F);
    } else {
        return face_flux<R, NSD, FLUX, D>(ul, ur, gamma, F);
    }
}

} // namespace als
