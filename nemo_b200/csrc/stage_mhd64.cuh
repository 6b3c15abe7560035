// stage_mhd64.cuh -- fused LSRK stage for GLM-MHD in plain FP64 (9 variables, bit-identical to the
// oracle); included by stage_fp64.cu, whose task layout it shares: one CTA of 64 threads per element,
// every two-point, face and subcell flux computed by one thread into shared memory, every node gathering
// its own terms in the oracle's order.  The pair fluxes are the symmetric EC part; each node adds its own
// Powell/GLM non-conservative term while it gathers.  The face fluxes carry the element's own-side term.
#pragma once

#include "mhd_fp64.cuh"

namespace nemo {
namespace mhd64k {

// Line form (a thread owned the three lines through (a, b): 255 registers, 8 warps per SM, every node's
// primitives and divisions by mu0 recomputed per pair) -> this, B200, us per stage: Orszag-Tang 32^3
// 1218 -> 636, 8^3 82 -> 23, 16^3 with Rusanov faces (general kernel) 187 -> 106; with the neighbour ids read
// ahead of the launch wait 611, 22, 104.  Bound by FP64 issue at 15 warps per SM (ncu, 32^3: issue 45 %, FP64
// pipe 42 %; stalls per issue: dependent latency 1.9, loads 1.6, barriers 1.4).
constexpr int MV = 9;
constexpr int CTAS = 8;                          // resident elements per SM: 8 x 27 KB of shared memory,
                                                 // 128 registers
// Shared memory of one element, in doubles
constexpr int MO_SU = 0;                          // [9][64] state
constexpr int MO_SP = MO_SU + MV * NP;             // [7][64] vx, vy, vz, beta_x, beta_y, beta_z, 1/rho
constexpr int MO_TR = MO_SP + 7 * NP;              // [9][96] neighbour traces / mortar rows, then face fluxes
constexpr int MO_SF = MO_TR + MV * 6 * NF;         // [9][6][16] pair fluxes of one direction
constexpr int MO_SV = MO_SF + MV * NPAIR * NF;     // [9][3][16] subcell fluxes (blended kernels)
constexpr int MELEM_PLAIN = MO_SV;
constexpr int MELEM_BLEND = MO_SV + MV * (NN - 1) * NF;
static_assert(MO_SF - MO_SP >= 6 * NP && MELEM_PLAIN - MO_SF >= MV * NP, "epilogue and repair scratch fit");

// column of line ab in a row of fluxes: the rows that a half-warp of nodes gathers from start on different
// banks
__device__ __forceinline__ int col(int row, int ab) { return ab ^ (4 * (row & 3)); }

// The fluxes of the 16 lines of direction d, as fluxes64
template <class A, bool BLEND, bool FAST, bool MU1>
__device__ __forceinline__ void m_fluxes64(int volume_flux, int surface_flux, int d, int w, int lane, double al,
                                           const double* su, double* tr, double* sF, double* sV, const int32_t* s_nbr,
                                           const OpConsts& k, const Mhd64<MU1>& P) {
    const double* sp = su + (MO_SP - MO_SU);
    const int c1 = d == 2 ? 0 : d + 1, c2 = d == 0 ? 2 : d - 1;
    // momenta; the field is 4 NP further on, the velocity VEL, beta (from m0) BETA
    const double *m0 = su + (1 + d) * NP, *m1 = su + (1 + c1) * NP, *m2 = su + (1 + c2) * NP;
    constexpr int FLD = 4 * NP, VEL = MO_SP - NP, BETA = MO_SP + 2 * NP;
    // ---- two-point fluxes, two pairs of the 16 lines at a time: warp 0 pairs 0, 1, 4, 5, warp 1 2, 3
#pragma unroll 1
    for (int g = w; g < 3; g += 2) {
        const int pq = 2 * g + (lane >> 4), ab = lane & 15;
        const int i = line_phys(d, ab, (0x211000 >> (4 * pq)) & 3), m = line_phys(d, ab, (0x332321 >> (4 * pq)) & 3);
        double F[MV];
        if (!FAST && volume_flux == NEMO_VOLFLUX_CENTRAL) {
            double ui[MV], um[MV], fu[MV], fm[MV];
            load_rot64(su, m0, m1, m2, NP, i, ui);
            load_rot64(su, m0, m1, m2, NP, m, um);
            m_xflux64<A>(ui, Rcp64{ui[0], sp[6 * NP + i]}, fu, P);
            m_xflux64<A>(um, Rcp64{um[0], sp[6 * NP + m]}, fm, P);
#pragma unroll
            for (int v = 0; v < MV; ++v) F[v] = 0.5 * (fu[v] + fm[v]);
        } else {
            const MNode64 ni = {su[i], sp[6 * NP + i], {m0[VEL + i], m1[VEL + i], m2[VEL + i]},
                                {m0[FLD + i], m1[FLD + i], m2[FLD + i]}, su[8 * NP + i], m0[BETA + i]};
            const MNode64 nm = {su[m], sp[6 * NP + m], {m0[VEL + m], m1[VEL + m], m2[VEL + m]},
                                {m0[FLD + m], m1[FLD + m], m2[FLD + m]}, su[8 * NP + m], m0[BETA + m]};
            m_ec64<A>(ni, nm, F, P);
        }
#pragma unroll
        for (int v = 0; v < MV; ++v) sF[(v * NPAIR + pq) * NF + col(pq, ab)] = F[v];
    }
    // ---- Riemann fluxes: round 0 the faces of the 16 lines with the own-side non-conservative term
    //      (warp 1), rounds 1 and 2 the FV subcell interfaces 0, 1 (warp 0) and 2 (half of warp 1)
    const int rounds = BLEND && al > 0.0 ? 3 : 1;
#pragma unroll 1
    for (int rt = 1 - w; rt < rounds; rt += 2) {
        const int hi = lane >> 4, ab = lane & 15;
        if (rt == 2 && hi) break;
        double uL[MV], uR[MV], F[MV];
        double* own_tr = tr + (2 * d + hi) * NF + ab;
        int own = 0;
        int32_t ne = 0;
        if (rt == 0) {
            ne = s_nbr[2 * d + hi];
            own = line_phys(d, ab, hi ? NN - 1 : 0);
            double uo[MV], un[MV];
            load_rot64(su, m0, m1, m2, NP, own, uo);
            if (ne == -1) load_rot64(su, m0, m1, m2, NP, own, un);   // domain boundary: the own trace
            else load_rot64(own_tr, own_tr + (1 + d) * 6 * NF, own_tr + (1 + c1) * 6 * NF, own_tr + (1 + c2) * 6 * NF, 6 * NF, 0, un);
#pragma unroll
            for (int v = 0; v < MV; ++v) {
                uL[v] = hi ? uo[v] : un[v];
                uR[v] = hi ? un[v] : uo[v];
            }
        } else {
            const int qi = 2 * (rt - 1) + hi;
            load_rot64(su, m0, m1, m2, NP, line_phys(d, ab, qi), uL);
            load_rot64(su, m0, m1, m2, NP, line_phys(d, ab, qi + 1), uR);
        }
        if (FAST || surface_flux == NEMO_SURFFLUX_HLLD) m_hlld64<A>(uL, uR, F, mhd64<true>(k, P.ch));
        else m_rusanov64<A>(uL, uR, F, P);
        if (rt == 0) {
            if (ne > -2) {   // a mortar's flux row is there already
                const double Bavg = 0.5 * (uL[5] + uR[5]), Gavg = 0.5 * (uL[8] + uR[8]);
                const double v[3] = {m0[VEL + own], m1[VEL + own], m2[VEL + own]};
                const double B[3] = {m0[FLD + own], m1[FLD + own], m2[FLD + own]};
                m_add_nc64(F, v, B, su[8 * NP + own], B[0] * v[0] + B[1] * v[1] + B[2] * v[2], Bavg, Gavg, P);
#pragma unroll
                for (int c = 0; c < MV; ++c) own_tr[c * 6 * NF] = F[c];
            }
        } else {
            const int row = 2 * (rt - 1) + hi;
#pragma unroll
            for (int v = 0; v < MV; ++v) sV[(v * (NN - 1) + row) * NF + col(row, ab)] = F[v];
        }
    }
}

// rhs terms in one direction's component order to the next one's
__device__ __forceinline__ void rotate_terms(const double* r, double* R) {
    R[0] = r[0];
    R[1] = r[2];
    R[2] = r[3];
    R[3] = r[1];
    R[4] = r[4];
    R[5] = r[6];
    R[6] = r[7];
    R[7] = r[5];
    R[8] = r[8];
}

// Node n's terms of direction d, in that direction's component order (pn: its position)
template <bool BLEND, bool FAST, bool MU1>
__device__ __forceinline__ void m_terms64(int volume_flux, int d, int n, int pn, double al, const double* su, const double* tr,
                                          const double* sF, const double* sV, const double* s_S, const double* s_winv,
                                          const Mhd64<MU1>& P, double* t) {
    const int c1 = d == 2 ? 0 : d + 1, c2 = d == 0 ? 2 : d - 1;
    const double *m0 = su + (1 + d) * NP, *m1 = su + (1 + c1) * NP, *m2 = su + (1 + c2) * NP;
    constexpr int FLD = 4 * NP, VEL = MO_SP - NP;
    // ---- the node's terms: its three pairs in ascending order of the other node, lift, FV, blend
    const int pos = (n >> (2 * d)) & 3;
    const int ab = d == 0 ? n >> 2 : (d == 1 ? (n & 3) | ((n >> 4) << 2) : n & 15);
    const unsigned rows = (unsigned)(0x0542053104300210ull >> (16 * pos));   // pair rows of this position
    const double vn[3] = {m0[VEL + pn], m1[VEL + pn], m2[VEL + pn]};
    const double Bn[3] = {m0[FLD + pn], m1[FLD + pn], m2[FLD + pn]};
    const double psi = su[8 * NP + pn];
    const double vB = Bn[0] * vn[0] + Bn[1] * vn[1] + Bn[2] * vn[2];
#pragma unroll
    for (int v = 0; v < MV; ++v) t[v] = 0.0;
#pragma unroll
    for (int mm = 0; mm < NN - 1; ++mm) {
        const int other = mm + (mm >= pos ? 1 : 0), row = (rows >> (4 * mm)) & 15;
        const double s = s_S[pos * NN + other];
        const double* f = sF + row * NF + col(row, ab);
        double F[MV];
#pragma unroll
        for (int v = 0; v < MV; ++v) F[v] = f[v * NPAIR * NF];
        double Bavg, Gavg;
        if (!FAST && volume_flux == NEMO_VOLFLUX_CENTRAL) {
            const int po = line_phys(d, ab, other);
            Bavg = 0.5 * (Bn[0] + m0[FLD + po]);
            Gavg = 0.5 * (psi + su[8 * NP + po]);
        } else {
            Gavg = F[5];
            Bavg = F[8];
            F[5] = P.ch * Gavg;
            F[8] = P.ch * Bavg;
        }
        m_add_nc64(F, vn, Bn, psi, vB, Bavg, Gavg, P);
#pragma unroll
        for (int v = 0; v < MV; ++v) t[v] = t[v] + s * F[v];
    }
    const double wi = s_winv[pos];
    const double* sS = tr + 2 * d * NF + ab;   // face fluxes of the line: [v][2][NF]
    if (pos == 0) {
#pragma unroll
        for (int v = 0; v < MV; ++v) t[v] = t[v] + wi * (-sS[v * 6 * NF]);
    }
    if (pos == NN - 1) {
#pragma unroll
        for (int v = 0; v < MV; ++v) t[v] = t[v] + wi * sS[v * 6 * NF + NF];
    }
    if (BLEND && al > 0.0) {
        double FL[MV], FR[MV];
        if (pos == 0) {
#pragma unroll
            for (int v = 0; v < MV; ++v) FL[v] = sS[v * 6 * NF];
        } else {
            const int po = line_phys(d, ab, pos - 1);
#pragma unroll
            for (int v = 0; v < MV; ++v) FL[v] = sV[(v * (NN - 1) + pos - 1) * NF + col(pos - 1, ab)];
            m_add_nc64(FL, vn, Bn, psi, vB, 0.5 * (m0[FLD + po] + Bn[0]), 0.5 * (su[8 * NP + po] + psi), P);
        }
        if (pos == NN - 1) {
#pragma unroll
            for (int v = 0; v < MV; ++v) FR[v] = sS[v * 6 * NF + NF];
        } else {
            const int po = line_phys(d, ab, pos + 1);
#pragma unroll
            for (int v = 0; v < MV; ++v) FR[v] = sV[(v * (NN - 1) + pos) * NF + col(pos, ab)];
            m_add_nc64(FR, vn, Bn, psi, vB, 0.5 * (Bn[0] + m0[FLD + po]), 0.5 * (psi + su[8 * NP + po]), P);
        }
#pragma unroll
        for (int v = 0; v < MV; ++v) t[v] = (1.0 - al) * t[v] + al * (wi * (FR[v] - FL[v]));
    }
}

// Per-node primitives of state q at sp[variable * NP]: velocities and, per direction, the EC flux's beta (its
// kinetic and magnetic sums run in the order of the rotated components)
template <class A, bool MU1>
__device__ __forceinline__ void m_primitives64(const double* q, const Rcp64& r, double* sp, const Mhd64<MU1>& P) {
    double vel[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vel[c] = A::quot(q[1 + c], r);
        sp[c * NP] = vel[c];
    }
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) {
        const double vr[3] = {vel[dd], vel[(dd + 1) % 3], vel[(dd + 2) % 3]};
        const double br[3] = {q[5 + dd], q[5 + (dd + 1) % 3], q[5 + (dd + 2) % 3]};
        sp[(3 + dd) * NP] = A::div(0.5 * q[0], m_p64(q[0], vr, br, q[4], q[8], P));
    }
}

// As plain_terms64 (stage_fp64.cu)
struct MTerms64 {
    double v[MV];
};
__device__ __noinline__ MTerms64 m_plain_terms64(const StageArgs& a, double al) {
    extern __shared__ __align__(16) double smem[];
    const OpConsts& k = c_ops64;
    const Mhd64<false> P = mhd64<false>(k, a.ctrl->glm_ch);   // mu0 = 1 changes no value
    const int64_t e = a.E_begin + blockIdx.x;
    const int n = threadIdx.x, lane = n & 31, w = n >> 5, pn = phys(n);
    double *su = smem + MO_SU, *sp = smem + MO_SP, *tr = smem + MO_TR, *sF = smem + MO_SF, *sV = smem + MO_SV;
    __syncthreads();
    double q[MV];
    for (int v = 0; v < MV; ++v) q[v] = su[v * NP + pn];
    m_primitives64<Plain64>(q, Plain64::rcp(q[0]), sp + pn, P);
    for (int p = n; p < 6 * NF; p += TPE) {
        const int f = p >> 4, ab = p & 15, ne = a.nbr[e * 6 + f];
        if (ne < 0) continue;   // a mortar's flux row is as it was
        const int m = line_node(f >> 1, ab & 3, ab >> 2, (f & 1) ? 0 : NN - 1);
        for (int v = 0; v < MV; ++v) tr[v * 6 * NF + p] = a.u_in[((int64_t)v * a.E + ne) * NP + m];
    }
    __syncthreads();
    MTerms64 R;
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        m_fluxes64<Plain64, true, false>(a.volume_flux, a.surface_flux, d, w, lane, al, su, tr, sF, sV, a.nbr + e * 6, k, P);
        __syncthreads();
        double t[MV];
        m_terms64<true, false>(a.volume_flux, d, n, pn, al, su, tr, sF, sV, k.S, k.winv, P, t);
        __syncthreads();
        const double cd = a.cdel[e * 3 + d];
        double r[MV];
        for (int v = 0; v < MV; ++v) r[v] = d == 0 ? cd * t[v] : R.v[v] + cd * t[v];
        rotate_terms(r, R.v);
    }
    return R;
}

}  // namespace mhd64k

template <bool BLEND, bool RHS_ONLY, bool FAST>
__global__ void __launch_bounds__(TPE, mhd64k::CTAS) k_stage_mhd64(const __grid_constant__ StageArgs a) {
    using namespace mhd64k;
    extern __shared__ __align__(16) double smem[];
    __shared__ double s_S[NN * NN], s_winv[NN], s_vi[NN * NN];
    __shared__ double s_alpha;
    __shared__ unsigned long long s_lam[2][4];
    __shared__ int s_bad, s_plain;
    __shared__ int32_t s_nbr[6];

    const OpConsts& k = c_ops64;
    Control* ctrl = a.ctrl;
    const int n = threadIdx.x, lane = n & 31, w = n >> 5;
    const int64_t E = a.E;
    const int64_t e = a.E_begin + blockIdx.x;
    if (n < NN * NN) {
        s_S[n] = k.S[n];
        s_vi[n] = k.Vinv[n];
        if (n < NN) s_winv[n] = k.winv[n];
    }
    // faces p of the neighbour traces this thread fetches, p = n and (warp 0) n + 64
    const int32_t nes[2] = {__ldg(a.nbr + e * 6 + (n >> 4)), n < 6 * NF - TPE ? __ldg(a.nbr + e * 6 + 4 + (n >> 4)) : -1};
    dep_sync();
    if (!RHS_ONLY && !a.prep_only && ctrl->done) return;
    double* const su = smem + MO_SU;
    double* const sp = smem + MO_SP;
    double* const tr = smem + MO_TR;
    double* const sF = smem + MO_SF;
    double* const sV = smem + MO_SV;
    const Mhd64<FAST> P = mhd64<FAST>(k, ctrl->glm_ch);

    double q[MV];
#pragma unroll
    for (int v = 0; v < MV; ++v) q[v] = __ldcg(a.u_in + ((int64_t)v * E + e) * NP + n);
    auto epilogue = [&]() {
        epilogue64<1>(a, q[0], m_pressure<double>(q, k.kappa, FAST ? 1.0 : k.mu0), sp, s_vi, s_lam, e, n, k,
                   [&](int dd) {
                       const double rr[MV] = {q[0], q[1 + dd], q[1 + (dd + 1) % 3], q[1 + (dd + 2) % 3], q[4],
                                              q[5 + dd], q[5 + (dd + 1) % 3], q[5 + (dd + 2) % 3], q[8]};
                       return m_xlambda<double>(rr, k.kappa, FAST ? 1.0 : k.mu0);
                   });
        if (a.epi_dt) {
            const double vm = fmax(fmax(fabs(q[1] / q[0]), fabs(q[2] / q[0])), fabs(q[3] / q[0]));
            const unsigned long long m = wmax64(vm);
            if (lane == 0) atomicMax(&ctrl->vmax_bits, m);
        }
    };
    if (a.prep_only) {
        __syncthreads();
        epilogue();
        return;
    }

    // neighbour traces (or mortar flux rows) of the 96 face nodes, asynchronously
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = n + r * TPE, f = p >> 4, ab = p & 15;
        if (p >= 6 * NF) break;
        const int32_t ne = nes[r];
        if (ab == 0) s_nbr[f] = ne;
        if (ne >= 0) {
            const double* g = a.u_in + (int64_t)ne * NP + line_node(f >> 1, ab & 3, ab >> 2, (f & 1) ? 0 : NN - 1);
#pragma unroll
            for (int v = 0; v < MV; ++v) cp_async8(tr + v * 6 * NF + p, g + (int64_t)v * E * NP);
        } else if (ne <= -2) {
            const double* g = a.mflux + (int64_t)(-2 - ne) * MV * NF + ab;
#pragma unroll
            for (int v = 0; v < MV; ++v) cp_async8(tr + v * 6 * NF + p, g + v * NF);
        }
    }
    if (!RHS_ONLY && a.stage > 0 && n < 4 * MV)   // the register rows, needed at the end
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.reg + ((int64_t)(n >> 2) * E + e) * NP + 16 * (n & 3)));
    if (n == 0) s_bad = s_plain = 0;
    if (BLEND && w == 0) smooth_alpha64(a, e, lane, &s_alpha);

    const int pn = phys(n);
#pragma unroll
    for (int v = 0; v < MV; ++v) su[v * NP + pn] = q[v];
    const Rcp64 ir = rcp64r(q[0]);
    sp[6 * NP + pn] = ir.y;
    m_primitives64<Quick64>(q, ir, sp + pn, P);
    asm volatile("cp.async.wait_all;" ::: "memory");
    // as in k_stage_euler64; us per stage without -> with it: Orszag-Tang 32^3 609 -> 627, 8^3 19.1 -> 19.6
    const double h = FAST ? 0.5 : 0.5 / k.mu0;
    bool regular = k.quick && m_regular64(q, h);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (nes[r] < 0) continue;
        double uo[MV];
#pragma unroll
        for (int v = 0; v < MV; ++v) uo[v] = tr[v * 6 * NF + n + r * TPE];
        regular = regular && m_regular64(uo, h);
    }
    __syncthreads();
    if (!regular) s_plain = 1;
    const double al = BLEND ? s_alpha : 0.0;

    // the node's rhs terms in the component order of the current direction (rotated on after each)
    double R[MV];
#pragma unroll
    for (int v = 0; v < MV; ++v) R[v] = 0.0;
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        m_fluxes64<Quick64, BLEND, FAST>(a.volume_flux, a.surface_flux, d, w, lane, al, su, tr, sF, sV, s_nbr, k, P);
        __syncthreads();
        double t[MV];
        m_terms64<BLEND, FAST>(a.volume_flux, d, n, pn, al, su, tr, sF, sV, s_S, s_winv, P, t);
        const double cd = __ldg(a.cdel + e * 3 + d);
        double r[MV];
#pragma unroll
        for (int v = 0; v < MV; ++v) r[v] = d == 0 ? cd * t[v] : R[v] + cd * t[v];
        rotate_terms(r, R);
        __syncthreads();
        if (s_plain) break;
    }
    if (s_plain) {
        const MTerms64 p = m_plain_terms64(a, al);
#pragma unroll
        for (int v = 0; v < MV; ++v) R[v] = p.v[v];
    }

    // ---- GLM damping, LSRK register and state update
    const int64_t g0 = e * NP + n;
    const double galpha = ctrl->glm_alpha;
    const int st = a.stage;
    const double A = rk_a(st);
    const double cdt = rk_c(st) * ctrl->dt[0];
    double rg[MV];
#pragma unroll
    for (int v = 0; v < MV; ++v) rg[v] = RHS_ONLY || st == 0 ? 0.0 : a.reg[(int64_t)v * E * NP + g0];
#pragma unroll
    for (int v = 0; v < MV; ++v) {
        const double u0 = su[v * NP + pn];
        double rhs = -R[v];
        if (v == 8) rhs = rhs - galpha * u0;
        if (RHS_ONLY) {
            a.rhs_out[(int64_t)v * E * NP + g0] = rhs;
        } else {
            const double rr = st == 0 ? rhs : A * rg[v] + rhs;
            a.reg[(int64_t)v * E * NP + g0] = rr;
            q[v] = u0 + cdt * rr;
        }
    }
    if (RHS_ONLY) return;
    if (a.positivity) {
        if (!m_isvalid<double>(q, k.kappa, FAST ? 1.0 : k.mu0)) s_bad = 1;
        __syncthreads();
        if (s_bad) {   // lanes 0..15 of warp 0 together, on a copy in node order
#pragma unroll
            for (int v = 0; v < MV; ++v) sF[v * NP + n] = q[v];
            __syncthreads();
            if (n < 16) {
                const bool repaired = repair_elem16_mhd<1>(sF, 0, n, k);
                if (!repaired && n == 0) atomicAdd(&ctrl->nbad, 1ull);
            }
            __syncthreads();
#pragma unroll
            for (int v = 0; v < MV; ++v) q[v] = sF[v * NP + n];
        }
    }
#pragma unroll
    for (int v = 0; v < MV; ++v) a.u_out[(int64_t)v * E * NP + g0] = q[v];
    if (st == 4 && a.tick && blockIdx.x == 0 && n == 0) {
        for (int g = 0; g < ctrl->ngroups; ++g) ctrl->t[g] = ctrl->t[g] + ctrl->dt[g];
        ctrl->steps += 1;
    }
    dep_launch();
    epilogue();
}

static int smem_mhd64(bool blend) { return (blend ? mhd64k::MELEM_BLEND : mhd64k::MELEM_PLAIN) * (int)sizeof(double); }

cudaError_t setup_stage_mhd64() {
    cudaError_t err;
    if ((err = attrs64(k_stage_mhd64<true, true, false>, smem_mhd64(true)))) return err;
    if ((err = attrs64(k_stage_mhd64<false, true, false>, smem_mhd64(false)))) return err;
    if ((err = attrs64(k_stage_mhd64<true, false, false>, smem_mhd64(true)))) return err;
    if ((err = attrs64(k_stage_mhd64<false, false, false>, smem_mhd64(false)))) return err;
    if ((err = attrs64(k_stage_mhd64<true, false, true>, smem_mhd64(true)))) return err;
    return attrs64(k_stage_mhd64<false, false, true>, smem_mhd64(false));
}

cudaError_t launch_stage_mhd64(const StageArgs& a, bool blend, bool rhs_only, cudaStream_t s) {
    if (a.E_own <= a.E_begin) return cudaSuccess;
    const unsigned grid = (unsigned)(a.E_own - a.E_begin);
    const int smem = smem_mhd64(blend);
    // the specialised kernel for HLLD faces (mu0 = 1) and the EC pair flux, the general one for the rest
    const bool fast = a.surface_flux == NEMO_SURFFLUX_HLLD && a.volume_flux == NEMO_VOLFLUX_EC_MHD;
    if (rhs_only) {
        if (blend) return launch_dep(k_stage_mhd64<true, true, false>, grid, TPE, smem, s, a);
        return launch_dep(k_stage_mhd64<false, true, false>, grid, TPE, smem, s, a);
    }
    if (fast) {
        if (blend) return launch_dep(k_stage_mhd64<true, false, true>, grid, TPE, smem, s, a);
        return launch_dep(k_stage_mhd64<false, false, true>, grid, TPE, smem, s, a);
    }
    if (blend) return launch_dep(k_stage_mhd64<true, false, false>, grid, TPE, smem, s, a);
    return launch_dep(k_stage_mhd64<false, false, false>, grid, TPE, smem, s, a);
}

}  // namespace nemo
