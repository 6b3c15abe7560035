// euler_fp64.cuh -- Euler physics in FP64 for the plain path.
//
// Every function evaluates the reference's Fortran expressions in the same order (the Fortran
// files are cited per function); this header is compiled with -fmad=false so that each + - * /
// is one IEEE operation.  All functions work in the frame rotated into the face normal
// direction: u = (rho, m_n, m_t1, m_t2, E), which is how the reference's y/z wrappers call the
// x-direction kernels (source/equations/euler/equations_mod.f90:81-127).
#pragma once

#include "common.cuh"
#include "ieee64.cuh"
#include "pmath64.cuh"

namespace nemo {

// pressure_elemental, source/equations/euler/equations_mod.f90:131-140
__device__ __forceinline__ double pressure64(const double* u, const OpConsts& k) {
    return k.km1 * (u[4] - 0.5 / u[0] * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]));
}

// xlambdaMax, source/equations/euler/equations_mod.f90:384-393 (soundspeed :288-297)
__device__ __forceinline__ double xlambda64(const double* u, const OpConsts& k) {
    double c = sqrt(k.kappa * pressure64(u, k) / u[0]);
    return fabs(u[1] / u[0]) + c;
}

// pressure, and xflux (source/equations/euler/equations_mod.f90:64-79), with the reciprocal of the
// density at hand (flux kernels)
template <class A>
__device__ __forceinline__ double pressure64(const double* u, const Rcp64& r, const OpConsts& k) {
    return k.km1 * (u[4] - A::quot(0.5, r) * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]));
}

__device__ __forceinline__ void xflux64(const double* u, double velx, double pres, double* f) {
    f[0] = u[1];
    f[1] = velx * u[1] + pres;
    f[2] = velx * u[2];
    f[3] = velx * u[3];
    f[4] = velx * (u[4] + pres);
}

// HLLC/HLLE hybrid, source/equations/euler/riemann/hllc/riemann_mod.f90:7-104.  Nine of its quotients
// share a density, two the sum of the roots and five the width of the fan.
template <class A>
__device__ __forceinline__ void hllc64(const double* UL, const double* UR, double* F, const OpConsts& k) {
    const double kappa = k.kappa;
    const double beta = k.hllc_beta;
    const Rcp64 rL = A::rcp(UL[0]), rR = A::rcp(UR[0]);
    double VL = A::quot(UL[1], rL);
    double VR = A::quot(UR[1], rR);
    double pL = pressure64<A>(UL, rL, k);
    double pR = pressure64<A>(UR, rR, k);
    double cL = A::root(A::quot(kappa * pL, rL));
    double cR = A::root(A::quot(kappa * pR, rR));
    double HL = A::quot(UL[4] + pL, rL);
    double HR = A::quot(UR[4] + pR, rR);
    double sL = A::root(UL[0]), sR = A::root(UR[0]);
    const Rcp64 rs = A::rcp(sL + sR);
    double Ht = A::quot(sL * HL + sR * HR, rs);
    double vt = A::quot(sL * VL + sR * VR, rs);
    double at = A::root(k.km1 * (Ht - 0.5 * (vt * vt)));
    double SL = fmin(fmin(vt - at, VL - beta * cL), 0.0);
    double SR = fmax(fmax(vt + at, VR + beta * cR), 0.0);
    // the supersonic cases (SL >= 0: the left flux, SR <= 0: the right flux) are selected at the
    // end instead of returned early: the same values, and no branch between the Riemann fluxes
    // of a line, which the compiler can then interleave (discarded values may be inf or NaN)
    double FL[5], FR[5];
    xflux64(UL, VL, pL, FL);
    xflux64(UR, VR, pR, FR);
    const bool supL = SL >= 0.0, supR = SR <= 0.0;
    double smooth = A::root(A::div(fabs(pL - pR), pL + pR));
    double SS = A::div(pR - pL + UL[1] * (SL - VL) - UR[1] * (SR - VR), UL[0] * (SL - VL) - UR[0] * (SR - VR));
    const bool left = (SL <= 0.0 && 0.0 <= SS);
    double U[5], FU[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
        U[v] = left ? UL[v] : UR[v];
        FU[v] = left ? FL[v] : FR[v];
    }
    const Rcp64 rU = {U[0], left ? rL.y : rR.y};
    const double S = left ? SL : SR;
    const double V = left ? VL : VR;
    const double p = left ? pL : pR;
    double Q = A::div(U[0] * (S - V), S - SS);
    double Us[5];
    Us[0] = Q;
    Us[1] = Q * SS;
    Us[2] = A::quot(Q * U[2], rU);
    Us[3] = A::quot(Q * U[3], rU);
    Us[4] = Q * (A::quot(U[4], rU) + (SS - V) * (SS + A::div(A::quot(p, rU), S - V)));
    const double oms = 1.0 - smooth;
    const double SLSR = SL * SR;
    const Rcp64 rd = A::rcp(SR - SL);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
        double FH = A::quot(SR * FL[v] - SL * FR[v] + SLSR * (UR[v] - UL[v]), rd);
        const double Fm = smooth * FH + oms * (FU[v] + S * (Us[v] - U[v]));
        F[v] = supL ? FL[v] : (supR ? FR[v] : Fm);
    }
}

// Rusanov, source/equations/euler/riemann/rusanov/riemann_mod.f90:7-24
template <class A>
__device__ __forceinline__ void rusanov64(const double* uL, const double* uR, double* F, const OpConsts& k) {
    double FL[5], FR[5];
    const Rcp64 rL = A::rcp(uL[0]), rR = A::rcp(uR[0]);
    const double VL = A::quot(uL[1], rL), VR = A::quot(uR[1], rR);
    double pL = pressure64<A>(uL, rL, k), pR = pressure64<A>(uR, rR, k);
    xflux64(uL, VL, pL, FL);
    xflux64(uR, VR, pR, FR);
    double lL = fabs(VL) + A::root(A::quot(k.kappa * pL, rL));
    double lR = fabs(VR) + A::root(A::quot(k.kappa * pR, rR));
    double lmax = fmax(lL, lR);
#pragma unroll
    for (int v = 0; v < 5; ++v) F[v] = 0.5 * (FL[v] + FR[v] + lmax * (uL[v] - uR[v]));
}

// FAST: HLLC fixed at compile time (a run-time switch is a branch around every flux)
template <class A, bool FAST>
__device__ __forceinline__ void riem64(int kind, const double* uL, const double* uR, double* F, const OpConsts& k) {
    if (!FAST && kind == 1) rusanov64<A>(uL, uR, F, k);
    else hllc64<A>(uL, uR, F, k);
}

// logmean with the absolute switch, source/equations/euler/two_point/chandrashekar/
// two_point_flux_mod.f90:13-32; x = a / b.  (Both means of a pair under one warp-wide branch each for the
// series and the logarithm interleaves their chains, but runs both for mixed warps: 397 against 383 us
// per stage at Sedov 32^3, 48.1 against 49.1 us on the smooth wave at 16^3.)
static __constant__ double LM_C[4] = {1e-4, 1.0 / 6.0, 2.0 / 45.0, 22.0 / 945.0};

template <class A>
__device__ __forceinline__ double logmean64(double a, double b, double x) {
    if (fabs(a - b) < LM_C[0]) {
        const double u = A::div(x * (x - 2.0) + 1.0, x * (x + 2.0) + 1.0);
        return (a + b) * (0.5 - u * (LM_C[1] - u * (LM_C[2] - LM_C[3] * u)));
    }
    return A::div(a - b, plog64(x));
}

// Per-node primitive data of the two-point flux: rho and its reciprocal, normal/tangential velocities,
// beta.
struct Node5 {
    double rho, y, vn, vt1, vt2, beta;
};

// Chandrashekar EC/KEP flux, two_point_flux_mod.f90:34-77 (the per-node quantities pressure,
// beta = 0.5*rho/p and velocities are computed once per node with the same expressions).
template <class A>
__device__ __forceinline__ void chandrashekar64(const Node5& u, const Node5& v, double* f, const OpConsts& k) {
    const double dens = logmean64<A>(u.rho, v.rho, A::quot(u.rho, Rcp64{v.rho, v.y}));
    double velx = 0.5 * (u.vn + v.vn);
    double vely = 0.5 * (u.vt1 + v.vt1);
    double velz = 0.5 * (u.vt2 + v.vt2);
    double pres = A::div(0.5 * (u.rho + v.rho), u.beta + v.beta);
    double ssum = (u.vn * u.vn + v.vn * v.vn) + (u.vt1 * u.vt1 + v.vt1 * v.vt1);
    ssum = ssum + (u.vt2 * u.vt2 + v.vt2 * v.vt2);
    double enth = A::div(k.c_enth, logmean64<A>(u.beta, v.beta, A::div(u.beta, v.beta))) + A::div(pres, dens) + velx * velx +
                  vely * vely + velz * velz - 0.25 * ssum;
    f[0] = dens * velx;
    f[1] = f[0] * velx + pres;
    f[2] = f[0] * vely;
    f[3] = f[0] * velz;
    f[4] = f[0] * enth;
}

// central flux 0.5*(f(u)+f(v)), source/equations/euler/two_point/standard/two_point_flux_mod.f90:13-49
template <class A>
__device__ __forceinline__ void central64(const double* u, const double* v, double* f, const OpConsts& k) {
    double fu[5], fv[5];
    const Rcp64 ru = A::rcp(u[0]), rv = A::rcp(v[0]);
    xflux64(u, A::quot(u[1], ru), pressure64<A>(u, ru, k), fu);
    xflux64(v, A::quot(v[1], rv), pressure64<A>(v, rv, k), fv);
#pragma unroll
    for (int c = 0; c < 5; ++c) f[c] = 0.5 * (fu[c] + fv[c]);
}

// Whether every flux of this state against another such state keeps Quick64's operands inside its domain:
// density and energy within 2^+-100, internal at least 2^-30 of total energy (velocities up to 2^20 sound
// speeds), no momentum between 0 and 2^-280.  With kappa - 1 within 2^-10..2^10 the pressure is then at least
// 2^-140, no speed of the fan nor what is left of a cancelling sum of them lies between 0 and 2^-179, the smallest
// numerator (the product of two momenta in the mean over the fan) is 2^-891 and the smallest quotient 2^-997.
// Ordinary flows meet the last condition: in a still ambient the exponents of the momenta double with every few
// elements from the disturbance (2^-229 on Sedov 32^3 after 40 steps).  A NaN fails the comparisons.
__device__ __forceinline__ bool within64(double x, int lo, int hi) {   // 2^lo <= x < 2^hi
    return (unsigned)__double2hiint(x) - ((unsigned)(1023 + lo) << 20) < (unsigned)(hi - lo) << 20;
}
__device__ __forceinline__ bool tiny64(double x, double limit) { return fabs(x) < limit && x != 0.0; }

__device__ __forceinline__ bool regular64(const double* u) {
    const double re = u[0] * u[4];
    const double ri = fma(-0.5, fma(u[1], u[1], fma(u[2], u[2], u[3] * u[3])), re);
    return within64(u[0], -100, 100) && within64(u[4], -100, 100) && ri >= 0x1p-30 * re && !tiny64(u[1], 0x1p-280) &&
           !tiny64(u[2], 0x1p-280) && !tiny64(u[3], 0x1p-280);
}

__device__ __forceinline__ bool isvalid64(const double* u, const OpConsts& k) {
    return (u[0] > 0.0) && (pressure64(u, k) > 0.0);
}

// Barotropic cooling after a stage (hook_post_rk_timestep_200,
// source/physics/cooling/barotropic_cooling_mod.f90:39-53): the energy of the barotropic equation of
// state, isothermal at or below dens_critical, adiabatic above (rho^kappa = exp(kappa log rho)).
__device__ __forceinline__ double cooled_energy64(const double* q, const OpConsts& k) {
    const double kin = 0.5 / q[0] * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    if (q[0] <= k.cool_rho) return kin + k.cool_ci * q[0];
    return kin + k.cool_ca * pexp64(k.kappa * plog64(q[0]));
}

}  // namespace nemo
