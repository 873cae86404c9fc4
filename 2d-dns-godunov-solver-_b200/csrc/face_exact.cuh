// The FP64 face and cell formulas with every division and square root
// correctly rounded in straight-line code (exact_math.cuh).
//
// Each function evaluates the formulas of physics.cuh so that every result
// rounds as there -- regrouped only where that is exact: multiplications by
// powers of two moved or folded into an fma, selects for branches, quotients
// over one divisor sharing its reciprocal -- and returns whether all its
// operands were in the range for which that holds.  Where they were not
// (exact zeros in a density, values near underflow at the head of a
// disturbance, infinities, NaN, a negative pressure) the caller evaluates
// the formulas as they stand in physics.cuh.
#pragma once

#include "exact_math.cuh"
#include "physics.cuh"

namespace gd2d {

// Numerators and divisors of one side's limiter for the four variables: u
// the cell's values, o the outer difference, c the central one; s the face's
// uL^2 + uR^2 and eh half the cell's (K HX)^3 (Venkatakrishnan).  The
// reconstruction is u + sign/2 times the quotient.
__device__ __forceinline__ void venkat_terms(double o, double c, double e, double &n, double &d) {
    const double oc = o * c;
    const bool opposite = oc < 0.0;
    const double cb = opposite ? 0.0 : c;
    const double c2 = cb * cb, oo = o * o;
    d = fma(2.0, oo, c2) + (opposite ? 0.0 : oc) + e;
    n = fma(2.0, oo * cb, (c2 + e) * o);
}
__device__ __forceinline__ void minmod_terms(double x, double y, double ksi, double &n, double &d) {
    const double p = x * y;
    n = p > 0.0 ? copysign(2.0 * p, x) : 0.0;
    d = fabs(x) + fabs(y) + ksi;
}
__device__ __forceinline__ void vanleer_terms(double a, double b, double ksi, double &n, double &d) {
    const double p = a * b, s = a + b + ksi;
    n = p > 0.0 ? copysign(2.0 * p, s) : 0.0;
    d = fabs(s);
}
__device__ __forceinline__ void vanalbada_terms(double a, double b, double ksi, double &n, double &d) {
    const double aa = a * a, bb = b * b;
    n = a * (bb + ksi) + b * (aa + ksi);
    d = aa + bb + 2.0 * ksi;
}

// Limited states of both sides of a face.  x: outer difference, y: central
// difference in the argument order of the caller's limiter kind.  One row of
// four quotients a side: eight at once would hold 32 registers of operands.
template <bool VENKAT>
__device__ __forceinline__ bool limited_side(int kind, double ksi, const double *u, const double *x, const double *y,
                                             const double *e, double half, double *up) {
    double n[4], d[4];
    if (VENKAT) {
#pragma unroll
        for (int v = 0; v < 4; ++v) venkat_terms(x[v], y[v], e[v], n[v], d[v]);
        // a velocity component that is zero all around has no quotient
#pragma unroll
        for (int v = 1; v < 3; ++v) d[v] = d[v] == 0.0 ? 1.0 : d[v];
    } else if (kind == LIM_MINMOD) {
#pragma unroll
        for (int v = 0; v < 4; ++v) minmod_terms(x[v], y[v], ksi, n[v], d[v]);
    } else if (kind == LIM_VANLEER) {
#pragma unroll
        for (int v = 0; v < 4; ++v) vanleer_terms(x[v], y[v], ksi, n[v], d[v]);
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v) vanalbada_terms(x[v], y[v], ksi, n[v], d[v]);
    }
    Divisors<-600, 200> r(d[0]);
    r.add(d[1]);
    r.add(d[2]);
    r.add(d[3]);
    Numerators t(n[1]);
    t.add(n[2]);
#pragma unroll
    for (int v = 0; v < 4; ++v) up[v] = fma(half, div_rn(n[v], d[v]), u[v]);
    // the reconstructed density and pressure are above 2^-150 (tested by the
    // caller), so that a quotient too small to be rounded right is lost in
    // the sum; a velocity may be as small as the quotient
    return r.ok() && t.ok();
}

// flux_ausm_plus (physics.cuh) with rg1 = 1/(gamma-1) correctly rounded.
// The caller tests the densities and pressures.
__device__ __forceinline__ bool ausm_plus_exact(const double *L, const double *R, double nx, double ny, double side,
                                                double gm1, double rg1, double g2, double *flux) {
    const double rhoL = L[0], UL = L[1], VL = L[2], PL = L[3];
    const double rhoR = R[0], UR = R[1], VR = R[2], PR = R[3];
    const double prL = div_rn(PL, rhoL), prR = div_rn(PR, rhoR);
    const double htL = fma(0.5, UL * UL + VL * VL, prL + div_by(prL, gm1, rg1));
    const double htR = fma(0.5, UR * UR + VR * VR, prR + div_by(prR, gm1, rg1));
    const double xL = g2 * htL, xR = g2 * htR;
    InRange<-400, 400> hr(xL);
    hr.add(xR);
    const double sL = sqrt_rn(xL), sR = sqrt_rn(xR);
    const double vnL = UL * nx + VL * ny, vnR = UR * nx + VR * ny;
    // s min(1, s/|vn|): the quotient counts only where |vn| > s
    const double wL = fabs(vnL) > sL ? fabs(vnL) : sL, wR = fabs(vnR) > sR ? fabs(vnR) : sR;
    const double aL = sL * div_rn(sL, wL), aR = sR * div_rn(sR, wR);
    const double a12 = aR < aL ? aR : aL;
    Divisors<-700, 200> dr(rhoL);
    dr.add(rhoR);
    dr.add(wL);
    dr.add(wR);
    dr.add(a12);
    const bool ok = hr.ok() && dr.ok();
    const double ya = rcp_rn(a12);
    const double ML = div_by(vnL, a12, ya), MR = div_by(vnR, a12, ya);
    const bool superL = fabs(ML) >= 1.0, superR = fabs(MR) >= 1.0;
    const double qL = ML * ML - 1.0, qR = MR * MR - 1.0;
    const double sqL = (ML + 1.0) * (ML + 1.0), sqR = (MR - 1.0) * (MR - 1.0);
    const double mpl = superL ? (ML > 0.0 ? ML : 0.0) : 0.125 * fma(2.0, sqL, qL * qL);
    const double mmi = superR ? (MR > 0.0 ? 0.0 : MR) : -0.125 * fma(2.0, sqR, qR * qR);
    const double m_dot12 = mpl + mmi;
    const double al = 3.0 / 16.0;
    const double ppl = superL ? (ML > 0.0 ? 1.0 : 0.0) : fma(0.25, sqL * (2.0 - ML), al * ML * qL * qL);
    const double pmi = superR ? (MR > 0.0 ? 0.0 : 1.0) : fma(0.25, sqR * (2.0 + MR), -(al * MR * qR * qR));
    const double p12 = ppl * PL + pmi * PR;
    const bool out = m_dot12 > 0.0;
    const double mL = (out ? m_dot12 : 0.0) * rhoL, mR = (out ? 0.0 : m_dot12) * rhoR;
    flux[0] = -(a12 * (mL + mR) + 0.0) * side;
    flux[1] = -(a12 * (mL * UL + mR * UR) + p12 * nx) * side;
    flux[2] = -(a12 * (mL * VL + mR * VR) + p12 * ny) * side;
    flux[3] = -(a12 * (mL * htL + mR * htR) + 0.0) * side;
    return ok;
}

// flux_roe (physics.cuh).  The caller tests the densities and pressures.
__device__ __forceinline__ bool roe_exact(const double *L, const double *R, double nx, double ny, double side,
                                          double gam, double gm1, double rgm1, double *flux) {
    const double rhoL = L[0], uL = L[1], vL = L[2], pL = L[3];
    const double rhoR = R[0], uR = R[1], vR = R[2], pR = R[3];
    const double mx = -ny, my = nx;
    const double unL = uL * nx + vL * ny, umL = uL * mx + vL * my;
    const double unR = uR * nx + vR * ny, umR = uR * mx + vR * my;
    const double yL = rcp_rn(rhoL);
    const double aL2 = div_by(gam * pL, rhoL, yL), aR2 = div_rn(gam * pR, rhoR), RT2 = div_by(rhoR, rhoL, yL);
    InRange<-400, 400> r(aL2);
    r.add(aR2);
    r.add(RT2);
    const double aL = sqrt_rn(aL2), aR = sqrt_rn(aR2), RT = sqrt_rn(RT2);
    const double HL = div_by(aL * aL, gm1, rgm1) + 0.5 * (uL * uL + vL * vL);
    const double HR = div_by(aR * aR, gm1, rgm1) + 0.5 * (uR * uR + vR * vR);
    const double rho = RT * rhoL, w = 1.0 + RT, yw = rcp_rn(w);
    // (a numerator too small for its quotient to round right is a velocity
    // lost beside the sound speed in all that follows but the products with
    // u and v themselves, so it is tested)
    const double un_ = uL + RT * uR, vn_ = vL + RT * vR;
    const double u = div_by(un_, w, yw), v = div_by(vn_, w, yw), H = div_by(HL + RT * HR, w, yw);
    const double a2 = gm1 * (H - 0.5 * (u * u + v * v));
    r.add(a2);
    r.add(HL);
    r.add(HR);
    const double a = sqrt_rn(a2);
    const double un = u * nx + v * ny, um = u * mx + v * my;
    const double drho = rhoR - rhoL, dp = pR - pL, dun = unR - unL, dum = umR - umL;
    const double aa = a * a, yaa = rcp_rn(aa);
    const double n1 = dp - rho * a * dun, n4 = dp + rho * a * dun;
    // 2 a a is twice a a, and so are their reciprocals one half
    const double LdU1 = div_by(n1, 2.0 * aa, 0.5 * yaa), LdU2 = rho * dum, LdU3 = drho - div_by(dp, aa, yaa);
    const double LdU4 = div_by(n4, 2.0 * aa, 0.5 * yaa);
    Divisors<-400, 200> d(rhoL);
    d.add(rhoR);
    d.add(w);
    d.add(aa);
    Numerators t(n1);
    t.add(n4);
    t.add(dp);
    t.add(un_);
    t.add(vn_);
    double ws1 = fabs(un - a), ws4 = fabs(un + a);
    const double ws2 = fabs(un);
    const double dws = 1.0 / 5.0, rdws = 1.0 / dws;
    Numerators tw(ws1);
    tw.add(ws4);
    if (ws1 < dws) ws1 = 0.5 * (div_by(ws1 * ws1, dws, rdws) + dws);
    if (ws4 < dws) ws4 = 0.5 * (div_by(ws4 * ws4, dws, rdws) + dws);
    const double w1 = ws1 * LdU1, w2 = ws2 * LdU2, w3 = ws2 * LdU3, w4 = ws4 * LdU4;
    const double d1 = ((0.0 + w1 * 1.0) + w2 * 0.0) + w3 * 1.0 + w4 * 1.0;
    const double d2 = ((0.0 + w1 * (u - a * nx)) + w2 * mx) + w3 * u + w4 * (u + a * nx);
    const double d3 = ((0.0 + w1 * (v - a * ny)) + w2 * my) + w3 * v + w4 * (v + a * ny);
    const double d4 = ((0.0 + w1 * (H - un * a)) + w2 * um) + w3 * (0.5 * (u * u + v * v)) + w4 * (H + un * a);
    const double mL = rhoL * unL, mR = rhoR * unR;
    flux[0] = -0.5 * (mL + mR - d1) * side;
    flux[1] = -0.5 * ((mL * uL + pL * nx) + (mR * uR + pR * nx) - d2) * side;
    flux[2] = -0.5 * ((mL * vL + pL * ny) + (mR * vR + pR * ny) - d3) * side;
    flux[3] = -0.5 * (mL * HL + mR * HR - d4) * side;
    return r.ok() && d.ok() && t.ok() && tw.ok();
}

// computeInterfaceSlope (computeslope2d.jl:3-136) from the face's states in
// registers: the cell's own values uL, the neighbour's (or ghost) uR, the
// node values uDn, uUp; ehL, ehR half of (K HX)^3 of the two cells.
template <int FLUX>
__device__ __forceinline__ bool face_flux_exact(const FaceCase &P, const double *uL, const double *uDn,
                                                const double *uR, const double *uUp, double ehL, double ehR,
                                                double nx, double ny, double side, double *f) {
    double A[4], B[4];
    bool ok = P.exact_rows != 0;
    const int kind = P.limiter;
    if (kind == LIM_VENKAT) {
        double o[4], c[4], s[4], e[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            c[v] = uR[v] - uL[v];
            o[v] = uL[v] - uDn[v];
            s[v] = uL[v] * uL[v] + uR[v] * uR[v];
            e[v] = ehL * s[v];
        }
        ok &= limited_side<true>(kind, 0.0, uL, o, c, e, 0.5, A);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            c[v] = -c[v];
            o[v] = uR[v] - uUp[v];
            e[v] = ehR * s[v];
        }
        ok &= limited_side<true>(kind, 0.0, uR, o, c, e, 0.5, B);
    } else if (kind == LIM_NONE) {
#pragma unroll
        for (int v = 0; v < 4; ++v) { A[v] = uL[v]; B[v] = uR[v]; }
    } else {
        double o[4], c[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            c[v] = uR[v] - uL[v];
            o[v] = uL[v] - uDn[v];
        }
        ok &= limited_side<false>(kind, P.ksi, uL, o, c, nullptr, 0.5, A);
#pragma unroll
        for (int v = 0; v < 4; ++v) o[v] = uUp[v] - uR[v];
        ok &= limited_side<false>(kind, P.ksi, uR, c, o, nullptr, -0.5, B);
    }
    InRange<-150, 200> r(A[0]);
    r.add(A[3]);
    r.add(B[0]);
    r.add(B[3]);
    ok &= r.ok();
    if (FLUX == FLUX_AUSM) ok &= ausm_plus_exact(B, A, nx, ny, side, P.gm1, P.rgm1, P.g2, f);
    else if (FLUX == FLUX_ROE) ok &= roe_exact(B, A, nx, ny, side, P.gamma, P.gm1, P.rgm1, f);
    else face_flux_fn<FLUX, double>(B, A, nx, ny, side, P.gamma, P.g2, f);
    return ok;
}

// Primitives and wave speed of a new conservative state: evaluate2d.jl:87-93
// as cell_update has it.  charlen / vmax is the cell's CFL length over speed.
struct CellPrims {
    double ux, uy, p, vmax, rmin;
};
__device__ __forceinline__ bool prims_exact(const double *U, double gam, double charlen, CellPrims &q) {
    const double rho = U[0], y = rcp_rn(rho);
    q.ux = div_by(U[1], rho, y);
    q.uy = div_by(U[2], rho, y);
    q.p = (gam - 1.0) * (U[3] - 0.5 * div_by(U[1] * U[1] + U[2] * U[2], rho, y));
    const double a2 = div_by(gam * q.p, rho, y);
    // a speed under 2^-200 is lost beside the sound speed
    const double w2 = q.ux * q.ux + q.uy * q.uy, floor2 = __hiloint2double(hi_pow2(-400), 0);
    q.vmax = sqrt_rn(w2 > floor2 ? w2 : floor2) + sqrt_rn(a2);
    q.rmin = div_rn(charlen, q.vmax);
    Divisors<-100, 200> r(rho);
    r.add(q.vmax);
    InRange<-100, 300> s(q.p);
    s.add(a2);
    Numerators t(U[1]);
    t.add(U[2]);
    return r.ok() && s.ok() && t.ok();
}

}  // namespace gd2d
