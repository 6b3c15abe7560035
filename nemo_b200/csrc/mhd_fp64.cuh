// mhd_fp64.cuh -- GLM-MHD fluxes of the plain FP64 stage kernel: the expressions of mhd_phys.cuh in the
// same order with the quotients of ieee64.cuh (shared reciprocals), the two-point flux on per-node
// primitives.  MU1: mu0 = 1 fixed at compile time (the HLLD requires it): multiplications and divisions
// by mu0 and 1/mu0 are exact and fall away.  Frame and variables as in mhd_phys.cuh.
#pragma once

#include "common.cuh"
#include "euler_fp64.cuh"
#include "ieee64.cuh"
#include "mhd_phys.cuh"
#include "pmath64.cuh"

namespace nemo {

template <bool MU1>
struct Mhd64 {
    double kappa, km1, skm1;   // kappa, kappa - 1, 1/(kappa - 1)
    double mu0_, ch;
    __device__ __forceinline__ double mu0() const { return MU1 ? 1.0 : mu0_; }
    // a / mu0 and (1 / mu0) a
    __device__ __forceinline__ double over_mu(double a) const { return MU1 ? a : a / mu0_; }
    __device__ __forceinline__ double smu(double a) const { return MU1 ? a : (1.0 / mu0_) * a; }
};

template <bool MU1>
__device__ __forceinline__ Mhd64<MU1> mhd64(const OpConsts& k, double ch) {
    return {k.kappa, k.km1, k.skm1, k.mu0, ch};
}

// pressure_elemental, source/equations/mhd/equations_mod.f90:223-234, with the reciprocal of the density
template <class A, bool MU1>
__device__ __forceinline__ double m_pressure64(const double* u, const Rcp64& r, const Mhd64<MU1>& P) {
    const double h = MU1 ? 0.5 : 0.5 / P.mu0_;
    return P.km1 * (u[4] - A::quot(0.5, r) * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) -
                    h * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7] + u[8] * u[8]));
}

// xflux, equations_mod.f90:64-139
template <class A, bool MU1>
__device__ __forceinline__ void m_xflux64(const double* U, const Rcp64& r, double* f, const Mhd64<MU1>& P) {
    const double kappaM2 = P.kappa - 2.0, s2mu_0 = MU1 ? 0.5 : 0.5 / P.mu0_;
    const double hmu = MU1 ? 0.5 : 0.5 * (1.0 / P.mu0_);
    const double Etotal = U[4] - hmu * (U[8] * U[8]);
    const double srho = A::quot(1.0, r);
    const double v1 = U[1] * srho, v2 = U[2] * srho, v3 = U[3] * srho;
    const double v_2 = v1 * v1 + v2 * v2 + v3 * v3;
    const double bb2 = U[5] * U[5] + U[6] * U[6] + U[7] * U[7];
    const double vb = U[5] * v1 + U[6] * v2 + U[7] * v3;
    const double pt = P.km1 * (Etotal - 0.5 * U[0] * v_2) - kappaM2 * s2mu_0 * bb2;
    const double Ep = Etotal + pt;
    const double sb = P.smu(U[5]);
    f[0] = U[1];
    f[1] = U[1] * v1 + pt - sb * U[5];
    f[2] = U[1] * v2 - sb * U[6];
    f[3] = U[1] * v3 - sb * U[7];
    f[4] = Ep * v1 - sb * vb;
    f[5] = 0.0;
    f[6] = v1 * U[6] - U[5] * v2;
    f[7] = v1 * U[7] - U[5] * v3;
    f[4] = f[4] + P.smu(P.ch) * U[5] * U[8];
    f[5] = f[5] + P.ch * U[8];
    f[8] = P.ch * U[5];
}

// Fastest_Signal_Speed + xlambdaMax, equations_mod.f90:693-714, :522-531
template <class A, bool MU1>
__device__ __forceinline__ double m_xlambda64(const double* U, const Rcp64& r, const Mhd64<MU1>& P) {
    const double pres = m_pressure64<A>(U, r, P);
    const double cs2 = A::quot(P.kappa * pres, r);
    const double ca2 = P.over_mu(A::quot(U[5] * U[5], r));
    const double va2 = P.over_mu(A::quot(U[6] * U[6] + U[7] * U[7], r)) + ca2;
    const double astar = A::root((cs2 + va2) * (cs2 + va2) - 4.0 * cs2 * ca2);
    const double c = A::root(0.5 * (cs2 + va2 + astar));
    return fabs(A::quot(U[1], r)) + c;
}

// Rusanov, source/equations/mhd/riemann/rusanov/riemann_mod.f90:7-24
template <class A, bool MU1>
__device__ __forceinline__ void m_rusanov64(const double* uL, const double* uR, double* F, const Mhd64<MU1>& P) {
    double FL[9], FR[9];
    const Rcp64 rL = A::rcp(uL[0]), rR = A::rcp(uR[0]);
    m_xflux64<A>(uL, rL, FL, P);
    m_xflux64<A>(uR, rR, FR, P);
    const double lmax = fmax(m_xlambda64<A>(uL, rL, P), m_xlambda64<A>(uR, rR, P));
#pragma unroll
    for (int v = 0; v < 9; ++v) F[v] = 0.5 * (FL[v] + FR[v] + lmax * (uL[v] - uR[v]));
}

// HLLD with the GLM pair upwind, as m_hlld_x (mhd_phys.cuh) expression by expression
template <class A>
__device__ __forceinline__ void m_hlld64(const double* uL, const double* uR, double* F, const Mhd64<true>& P) {
    const double half = 0.5, kappa = P.kappa;
    const Rcp64 rkm1 = {P.km1, P.skm1};
    const double bn = half * (uL[5] + uR[5]) - half * (uR[8] - uL[8]);
    const double psn = half * (uL[8] + uR[8]) - half * (uR[5] - uL[5]);
    const double bn2 = bn * bn;
    double rho[2], un[2], vt1[2], vt2[2], bt1[2], bt2[2], et[2], pt[2], cf[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double* u = s ? uR : uL;
        const Rcp64 r = A::rcp(u[0]);
        rho[s] = u[0];
        un[s] = A::quot(u[1], r);
        vt1[s] = A::quot(u[2], r);
        vt2[s] = A::quot(u[3], r);
        bt1[s] = u[6];
        bt2[s] = u[7];
        const double pr = P.km1 * (u[4] - A::quot(half, r) * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) -
                                   half * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7] + u[8] * u[8]));
        const double bb = bn2 + bt1[s] * bt1[s] + bt2[s] * bt2[s];
        et[s] = A::quot(pr, rkm1) + half * rho[s] * (un[s] * un[s] + vt1[s] * vt1[s] + vt2[s] * vt2[s]) + half * bb;
        pt[s] = pr + half * bb;
        const double cs2 = A::quot(kappa * pr, r);
        const double ca2 = A::quot(bn2, r);
        const double va2 = A::quot(bb, r);
        cf[s] = A::root(half * (cs2 + va2 + A::root((cs2 + va2) * (cs2 + va2) - 4.0 * cs2 * ca2)));
    }
    const double cmax = fmax(cf[0], cf[1]);
    const double SL = fmin(un[0], un[1]) - cmax;
    const double SR = fmax(un[0], un[1]) + cmax;
    double Fk[2][8], Uk[2][8];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double vb = un[s] * bn + vt1[s] * bt1[s] + vt2[s] * bt2[s];
        const double m = rho[s] * un[s];
        Fk[s][0] = m;
        Fk[s][1] = m * un[s] + pt[s] - bn2;
        Fk[s][2] = m * vt1[s] - bn * bt1[s];
        Fk[s][3] = m * vt2[s] - bn * bt2[s];
        Fk[s][4] = (et[s] + pt[s]) * un[s] - bn * vb;
        Fk[s][5] = 0.0;
        Fk[s][6] = un[s] * bt1[s] - bn * vt1[s];
        Fk[s][7] = un[s] * bt2[s] - bn * vt2[s];
        Uk[s][0] = rho[s];
        Uk[s][1] = m;
        Uk[s][2] = rho[s] * vt1[s];
        Uk[s][3] = rho[s] * vt2[s];
        Uk[s][4] = et[s];
        Uk[s][5] = bn;
        Uk[s][6] = bt1[s];
        Uk[s][7] = bt2[s];
    }
    if (SL > 0.0) {
#pragma unroll
        for (int v = 0; v < 8; ++v) F[v] = Fk[0][v];
    } else if (SR < 0.0) {
#pragma unroll
        for (int v = 0; v < 8; ++v) F[v] = Fk[1][v];
    } else {
        const double dL = rho[0] * (SL - un[0]), dR = rho[1] * (SR - un[1]);
        const double SM = A::div(dR * un[1] - dL * un[0] - pt[1] + pt[0], dR - dL);
        const double ptS = pt[0] + dL * (SM - un[0]);
        double rs[2], ws1[2], ws2[2], cs1[2], cs2[2], es[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double S = s ? SR : SL;
            const double d = s ? dR : dL;
            const Rcp64 rS = A::rcp(S - SM);
            rs[s] = A::quot(d, rS);
            const double den = d * (S - SM) - bn2;
            const Rcp64 rden = A::rcp(den);
            const double fv = A::quot(bn * (SM - un[s]), rden);
            const double fb = A::quot(d * (S - un[s]) - bn2, rden);
            const bool flat = fabs(den) < 1.0e-8;
            ws1[s] = flat ? vt1[s] : vt1[s] - fv * bt1[s];
            ws2[s] = flat ? vt2[s] : vt2[s] - fv * bt2[s];
            cs1[s] = flat ? bt1[s] : fb * bt1[s];
            cs2[s] = flat ? bt2[s] : fb * bt2[s];
            const double vb = un[s] * bn + vt1[s] * bt1[s] + vt2[s] * bt2[s];
            const double vbs = SM * bn + ws1[s] * cs1[s] + ws2[s] * cs2[s];
            es[s] = A::quot((S - un[s]) * et[s] - pt[s] * un[s] + ptS * SM + bn * (vb - vbs), rS);
        }
        const double sqL = A::root(rs[0]), sqR = A::root(rs[1]);
        const double SLs = SM - A::div(fabs(bn), sqL), SRs = SM + A::div(fabs(bn), sqR);
        const bool sr = !(SM >= 0.0);
        const double S = sr ? SR : SL;
        const double rsS = sr ? rs[1] : rs[0], ws1S = sr ? ws1[1] : ws1[0], ws2S = sr ? ws2[1] : ws2[0];
        const double cs1S = sr ? cs1[1] : cs1[0], cs2S = sr ? cs2[1] : cs2[0], esS = sr ? es[1] : es[0];
        const double Us[8] = {rsS, rsS * SM, rsS * ws1S, rsS * ws2S, esS, bn, cs1S, cs2S};
        const bool outer = sr ? (SRs < 0.0) : (SLs >= 0.0);
        if (outer) {
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const double FkS = sr ? Fk[1][v] : Fk[0][v], UkS = sr ? Uk[1][v] : Uk[0][v];
                F[v] = FkS + S * (Us[v] - UkS);
            }
        } else {
            double Uss[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) Uss[v] = Us[v];
            if (fabs(bn) >= 1.0e-12) {
                const double sg = bn < 0.0 ? -1.0 : 1.0;
                const double sden = A::div(1.0, sqL + sqR);
                const double w1 = (sqL * ws1[0] + sqR * ws1[1] + sg * (cs1[1] - cs1[0])) * sden;
                const double w2 = (sqL * ws2[0] + sqR * ws2[1] + sg * (cs2[1] - cs2[0])) * sden;
                const double c1 = (sqL * cs1[1] + sqR * cs1[0] + sg * sqL * sqR * (ws1[1] - ws1[0])) * sden;
                const double c2 = (sqL * cs2[1] + sqR * cs2[0] + sg * sqL * sqR * (ws2[1] - ws2[0])) * sden;
                const double wcs = ws1S * cs1S + ws2S * cs2S;
                const double wcss = w1 * c1 + w2 * c2;
                const double sq = sr ? sqR : sqL;
                Uss[2] = rsS * w1;
                Uss[3] = rsS * w2;
                Uss[4] = sr ? esS + sg * sq * (wcs - wcss) : esS - sg * sq * (wcs - wcss);
                Uss[6] = c1;
                Uss[7] = c2;
            }
            const double Ss = sr ? SRs : SLs;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const double FkS = sr ? Fk[1][v] : Fk[0][v], UkS = sr ? Uk[1][v] : Uk[0][v];
                F[v] = FkS + Ss * Uss[v] - (Ss - S) * Us[v] - S * UkS;
            }
        }
    }
    F[4] = F[4] + P.ch * bn * psn;
    F[5] = P.ch * psn;
    F[8] = P.ch * bn;
}

// LN_MEAN, source/equations/mhd/two_point/ec/two_point_flux_mod.f90:203-219 (relative switch); Xi = aR/aL
static __constant__ double LNM_EPS = 1.0e-4;

template <class A>
__device__ __forceinline__ double ln_mean64(double aL, double aR, double Xi) {
    const double u = A::div(Xi * (Xi - 2.0) + 1.0, Xi * (Xi + 2.0) + 1.0);
    if (u < LNM_EPS) return A::div((aL + aR) * 52.5, 105.0 + u * (35.0 + u * (21.0 + u * 15.0)));
    return A::div(aR - aL, plog64(Xi));
}

// Per-node data of the two-point flux in the frame of a direction
struct MNode64 {
    double rho, y, v[3], B[3], psi, beta;   // y = 1/rho, beta = rho/(2 p) with p in that frame's order
};

// pressure of the EC flux, whose beta is rho/(2 p) (psi^2/2 is subtracted first), momentum and field in the
// frame's order
template <bool MU1>
__device__ __forceinline__ double m_p64(double rho, const double* v, const double* B, double E, double psi,
                                        const Mhd64<MU1>& P) {
    const double hmu = MU1 ? 0.5 : 0.5 * (1.0 / P.mu0_);
    const double E1 = E - hmu * (psi * psi);
    const double v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    const double B2 = B[0] * B[0] + B[1] * B[1] + B[2] * B[2];
    return P.km1 * (E1 - 0.5 * (rho * v2 + P.smu(B2)));
}

// EC (Derigs) flux, source/equations/mhd/two_point/ec/two_point_flux_mod.f90:13-86.  In the places of
// F[5] and F[8] it returns {psi} and {B_n}, from which the gathering node forms both (c_h {psi}, c_h {B_n})
// and its non-conservative term.
template <class A, bool MU1>
__device__ __forceinline__ void m_ec64(const MNode64& L, const MNode64& R, double* F, const Mhd64<MU1>& P) {
    const double v2_L = L.v[0] * L.v[0] + L.v[1] * L.v[1] + L.v[2] * L.v[2];
    const double v2_R = R.v[0] * R.v[0] + R.v[1] * R.v[1] + R.v[2] * R.v[2];
    const double B2_L = L.B[0] * L.B[0] + L.B[1] * L.B[1] + L.B[2] * L.B[2];
    const double B2_R = R.B[0] * R.B[0] + R.B[1] * R.B[1] + R.B[2] * R.B[2];
    const double rhoLN = ln_mean64<A>(L.rho, R.rho, A::quot(R.rho, Rcp64{L.rho, L.y}));
    const double betaLN = ln_mean64<A>(L.beta, R.beta, A::div(R.beta, L.beta));
    double vAvg[3], BAvg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vAvg[c] = 0.5 * (L.v[c] + R.v[c]);
        BAvg[c] = 0.5 * (L.B[c] + R.B[c]);
    }
    const double v1_B2Avg = 0.5 * (L.v[0] * B2_L + R.v[0] * B2_R);
    const double vB_Avg = 0.5 * ((L.v[0] * L.B[0] + L.v[1] * L.B[1] + L.v[2] * L.B[2]) +
                                 (R.v[0] * R.B[0] + R.v[1] * R.B[1] + R.v[2] * R.B[2]));
    const double hs = MU1 ? 0.5 : (1.0 / P.mu0_) * 0.5;
    const double pTilde = 0.5 * (A::div(L.rho + R.rho, L.beta + R.beta) + hs * (B2_L + B2_R));
    const double psiAvg = 0.5 * (L.psi + R.psi);
    const double sB = P.smu(BAvg[0]);
    F[0] = rhoLN * vAvg[0];
    F[1] = F[0] * vAvg[0] - sB * BAvg[0] + pTilde;
    F[2] = F[0] * vAvg[1] - sB * BAvg[1];
    F[3] = F[0] * vAvg[2] - sB * BAvg[2];
    F[6] = vAvg[0] * BAvg[1] - BAvg[0] * vAvg[1];
    F[7] = vAvg[0] * BAvg[2] - BAvg[0] * vAvg[2];
    const double F5 = P.ch * psiAvg, F8 = P.ch * BAvg[0];
    const double s1 = vAvg[0] * F[1] + vAvg[1] * F[2] + vAvg[2] * F[3];
    const double s2 = BAvg[0] * F5 + BAvg[1] * F[6] + BAvg[2] * F[7];
    F[4] = F[0] * 0.5 * (A::div(P.skm1, betaLN) - 0.5 * (v2_L + v2_R)) + s1 +
           P.smu(s2 - 0.5 * v1_B2Avg + BAvg[0] * vB_Avg + F8 * psiAvg - P.ch * 0.5 * (L.psi * L.B[0] + R.psi * R.B[0]));
    F[5] = psiAvg;
    F[8] = BAvg[0];
}

// Non_Conservative_two_point_xFlux (Powell + GLM), source/equations/mhd/non_conservative_flux_mod.f90:10-45,
// of a node with velocity v, field B, psi and vB = v . B, for the pair means Bavg, Gavg; added to F.
template <bool MU1>
__device__ __forceinline__ void m_add_nc64(double* F, const double* v, const double* B, double psi, double vB,
                                           double Bavg, double Gavg, const Mhd64<MU1>& P) {
    const double gv = Gavg * v[0];
    F[0] = F[0] + 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        F[1 + c] = F[1 + c] + P.over_mu(Bavg * B[c]);
        F[5 + c] = F[5 + c] + Bavg * v[c];
    }
    F[4] = F[4] + (P.over_mu(Bavg * vB) + gv * P.over_mu(psi));
    F[8] = F[8] + gv;
}

// As regular64 (euler_fp64.cuh): density within 2^-100..2^40 and energy within 2^+-60 (code units, SI, and CGS down to
// 1e-30 g/cm^3), internal at least 2^-30 of total energy, no component of momentum and field and no psi between 0 and
// 2^-170, mu0 within 2^+-40.  The smallest numerator is the HLLD's B_n (S_M - v_n): S_M, a quotient of sums that may
// cancel, is at least 2^-493, B_n 2^-224 and their product with another cancellation 2^-770; the smallest quotient,
// of it by a denominator up to 2^218, is 2^-988.
__device__ __forceinline__ bool m_regular64(const double* u, double h) {   // h = 1/(2 mu0)
    const double re = u[0] * u[4];
    const double b2 = fma(u[5], u[5], fma(u[6], u[6], fma(u[7], u[7], u[8] * u[8])));
    const double k2 = fma(u[1], u[1], fma(u[2], u[2], u[3] * u[3]));
    const double ri = fma(-0.5, k2, u[0] * fma(-h, b2, u[4]));
    bool ok = within64(u[0], -100, 40) && within64(u[4], -60, 60) && ri >= 0x1p-30 * re;
#pragma unroll
    for (int v = 1; v < 9; ++v)
        if (v != 4) ok = ok && !tiny64(u[v], 0x1p-170);
    return ok;
}

}  // namespace nemo
