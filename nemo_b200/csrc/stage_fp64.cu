// stage_fp64.cu -- plain FP64 path: one fused kernel per LSRK stage (compiled with -fmad=false).
//
// One CTA of 64 threads per element, one thread per node.  Per stage and element it does what the
// reference spreads over hook_pre_rk_timestep_300 and hook_mid_rk_timestep_500:
//   1. the element's state into shared memory, the 96 neighbour trace nodes (or 2:1 mortar flux rows)
//      beside it by cp.async, in flight while
//   2. the per-node primitives (velocities, beta_d = rho/(2 p_d) per direction) are computed, and the node and
//      the traces checked for operands that the quotients of ieee64.cuh are not made for;
//   3. per direction, the 96 two-point fluxes of the split form (16 lines x 6 node pairs), the 32 face
//      fluxes (kernel_fill_faceflux, source/kernel/mcfv/3d/kernel_flux_mod.f90:47-278) and, where
//      alpha > 0, the 48 FV subcell fluxes, each an independent task of one thread with its result in
//      shared memory; then each node sums its own pairs in a fixed order, the surface lift, the FV
//      term and the convex blend (an element whose check failed does 2 and 3 again with / and sqrt);
//   4. the LSRK 5-4 register/state update (timedisc_probe, source/timedisc/rungekutta/
//      low-storage/4-5/timedisc_probe_mod.f90:7-39; rkstep_cb :19-49);
//   5. the positivity repair (dgfv_repair_3d, source/kernel/mcfv/3d/kernel_validate_mod.f90:159-272);
//   6. epilogue on the new state: the modal (or learned) indicator for the next stage and, on the
//      last stage, the per-element CFL bound for the next time step (kernel_timestep_mod.f90:348-394).
// The arithmetic follows oracle/nemo_oracle.cpp expression by expression, so the two agree to
// the last bit except where log/exp enter.
#include "common.cuh"
#include "euler_fp64.cuh"
#include "kernels.h"
#include "repair64.cuh"

namespace nemo {

__constant__ OpConsts c_ops64;

namespace {

// One flux per thread instead of one line per thread: a thread that owned a whole line kept 4 x 5
// accumulators and both face fluxes live across six inlined pair fluxes and five inlined Riemann solvers
// (96 registers and 1 KB of spills, 18 warps per SM, instruction fetch the second largest stall).  As
// tasks the kernel holds one copy of each flux, and no element waits for another of its CTA.  With the
// quotients of ieee64.cuh, B200, us per stage, line form -> this: Sedov 32^3 664 -> 381 (0.16 of the FP64
// FMA peak by algorithmic flops; 392 with the check of their domain), Kelvin-Helmholtz forest of 24k elements
// 619 -> 340, 4^3 elements 38 -> 19 (with the compiler's quotients and 16 warps per SM the task form alone was 727 at 32^3).
// What bounds it now (ncu, Sedov 32^3): 242 M warp instructions at 56 % issue, of which 103 M FP64 (the
// FP64 pipe 49 % busy); stalls per issue: dependent latency 2.3, CTA barriers 1.5, instruction fetch 1.2.
// Resident elements per SM at 14 / 12 / 10 / 8 (72, 80, 96, 128 registers): 424 / 397 / 403 / 420 us
// (measured with both logarithmic means of a pair under warp-wide branches).
constexpr int TPE = 64;              // threads per element, one per node
constexpr int V = 5;
constexpr int NPAIR = 6;             // node pairs of a line
constexpr int FROW = NF + 4;         // row stride of the pair / subcell fluxes: the rows that a
                                     // half-warp of nodes gathers from start 4 double-banks apart
constexpr int CTAS64 = 12;           // resident CTAs (elements) per SM asked of the register allocator

// Shared memory of one element, in doubles
constexpr int O_SU = 0;                          // [V][64] state
constexpr int O_SP = O_SU + V * NP;              // [7][64] vx, vy, vz, beta_x, beta_y, beta_z, 1/rho
constexpr int O_TR = O_SP + 7 * NP;              // [V][96] neighbour traces / mortar flux rows, then the
                                                 // face fluxes in their places
constexpr int O_SF = O_TR + V * 6 * NF;          // [V][6][FROW] pair fluxes of one direction
constexpr int O_SV = O_SF + V * NPAIR * FROW;    // [V][3][FROW] subcell fluxes (blended kernels)
constexpr int ELEM_PLAIN = O_SV;
constexpr int ELEM_BLEND = O_SV + V * (NN - 1) * FROW;
static_assert(O_SV - O_SP >= 6 * NP, "the epilogue's six node arrays fit behind the state");

// Position of node n in the [64] arrays of state and primitives: the x and y digits are exclusive-ored
// with a function of z (a GF(4) code), so that the 16 lines of each of the three directions fall on 16
// different double-banks (in node order the x- and y-lines conflict four ways).
__device__ __forceinline__ int swz(int z) { return (0x7e90 >> (4 * z)) & 15; }
__device__ __forceinline__ int phys(int n) { return n ^ swz(n >> 4); }
__device__ __forceinline__ int line_phys(int d, int ab, int i) {
    if (d == 0) return ((4 * ab) ^ swz(ab >> 2)) ^ i;
    if (d == 1) return (((ab & 3) | ((ab >> 2) << 4)) ^ swz(ab >> 2)) ^ (4 * i);
    return (ab ^ swz(i)) | (i << 4);
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

__device__ __forceinline__ double silu64(double x) { return x / (1.0 + pexp64(-x)); }

// Barrier of one element's 64 threads: of the CTA, or (ND = 3, see k_stage_euler64) of group g of it
template <int ND>
__device__ __forceinline__ void group_sync(int g) {
    if (ND == 1) __syncthreads();
    else asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory");
}

// maximum over the warp by bit patterns (non-negative values; a NaN counts as the largest)
__device__ __forceinline__ unsigned long long wmax64(double x) {
    unsigned long long v = (unsigned long long)__double_as_longlong(x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The element's blending coefficient, smoothed over its conforming neighbours (warp 0).
__device__ __forceinline__ void smooth_alpha64(const StageArgs& a, int64_t e, int lane, double* s_alpha) {
    double al = 0.0;
    if (lane == 6) al = a.alpha_in[e];
    if (a.smooth && lane < 6) {
        const int32_t ne = __ldg(a.nbr + e * 6 + lane);
        if (ne >= 0) al = 0.5 * a.alpha_in[ne];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) al = fmax(al, __shfl_xor_sync(0xffffffffu, al, o));
    if (lane == 0) {
        *s_alpha = al;
        if (a.alpha_used) a.alpha_used[e] = al;
    }
}

// state of the node at index i rotated into a direction whose momenta start at m0, m1, m2 (the magnetic
// field four variables further on); st: stride of the variables
__device__ __forceinline__ void load_rot64(const double* u, const double* m0, const double* m1, const double* m2, int st,
                                           int i, double* r) {
    r[0] = u[i];
    r[1] = m0[i];
    r[2] = m1[i];
    r[3] = m2[i];
    r[4] = u[4 * st + i];
    r[5] = m0[4 * st + i];
    r[6] = m1[4 * st + i];
    r[7] = m2[4 * st + i];
    r[8] = u[8 * st + i];
}

// Modal coefficients of the nodal values q (one per thread) into cm[64]: x and y inside a warp, z
// across the element's two warps; t1, t2 are [64] scratch.
template <int ND>
__device__ __forceinline__ double modal64(double q, double* t1, double* t2, const double* vi, int n) {
    const int x = n & 3, y = (n >> 2) & 3, z = n >> 4;
    t1[n] = q;
    __syncwarp();
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < NN; ++i) s = s + vi[x * NN + i] * t1[nidx(i, y, z)];
    t2[n] = s;
    __syncwarp();
    s = 0.0;
#pragma unroll
    for (int j = 0; j < NN; ++j) s = s + vi[y * NN + j] * t2[nidx(x, j, z)];
    __syncwarp();
    t1[n] = s;
    group_sync<ND>(0);
    s = 0.0;
#pragma unroll
    for (int k = 0; k < NN; ++k) s = s + vi[z * NN + k] * t1[nidx(x, y, k)];
    return s;
}

// Epilogue on this thread's node of density rho and pressure pr (of the new state of a stage, or of the
// uploaded state of a prepare launch): the blending coefficient for the next stage (modal indicator, or
// learned indicator with the modal one as fallback and judge) and, if requested, the per-element CFL bound
// from the wave speeds lambda(d).  sp: scratch of the element, six [64] arrays.  Sums run in the oracle's
// serial order.
template <int ND, typename Lambda>
__device__ __forceinline__ void epilogue64(const StageArgs& a, double rho, double pr, double* sp, const double* vi,
                                           unsigned long long (*s_lam)[4], int64_t e, int n, const OpConsts& k,
                                           Lambda lambda) {
    Control* ctrl = a.ctrl;
    const int lane = n & 31, w = n >> 5;
    if (a.alpha_out) {
        double* e2 = sp + 2 * NP;   // [3][64]: squared modes, those of order < N, those of order < N-1
        const double m = modal64<ND>(rho * pr, sp, sp + NP, vi, n);
        const int top = max(max(n & 3, (n >> 2) & 3), n >> 4);
        e2[n] = m * m;
        e2[NP + n] = top < NN - 1 ? m * m : 0.0;
        e2[2 * NP + n] = top < NN - 2 ? m * m : 0.0;
        group_sync<ND>(0);
        double am = 0.0;
        if (w == 0) {
            // one sum per lane 0..2, in mode order (the zeros change nothing)
            const double* el = e2 + (lane < 3 ? lane : 0) * NP;
            double s = 0.0;
#pragma unroll 16
            for (int p = 0; p < NP; ++p) s = s + el[p];
            const double total = __shfl_sync(0xffffffffu, s, 0);
            const double clip1 = __shfl_sync(0xffffffffu, s, 1);
            const double clip2 = __shfl_sync(0xffffffffu, s, 2);
            const double energy = fmax((total - clip1) / total, (clip1 - clip2) / clip1);
            double al = 1.0 / (1.0 + pexp64(k.ind_k * (energy - k.ind_T)));
            if (al < k.alpha_min) al = 0.0;
            else if (al > k.one_m_alpha_min) al = 1.0;
            am = fmin(k.alpha_max, al);
        }
        if (a.mlp64 == nullptr) {
            if (n == 0) a.alpha_out[e] = am;
        } else {
            // learned indicator: squared modes of rho and p, nodal rho and p, then warp 0 alone
            double* er = sp + 3 * NP;
            double* ep = sp + 4 * NP;
            double* np = sp + 5 * NP;
            group_sync<ND>(0);   // the sums above are done with e2
            const double mr = modal64<ND>(rho, sp, sp + NP, vi, n);
            group_sync<ND>(0);
            const double mp = modal64<ND>(pr, sp, sp + NP, vi, n);
            er[n] = mr * mr;
            ep[n] = mp * mp;
            np[n] = pr;
            group_sync<ND>(0);
            sp[n] = rho;     // nodal rho (the transform scratch is dead)
            group_sync<ND>(0);
            if (w == 0) {
                double* feat = sp + NP;      // [12]
                double* h1 = sp + NP + 16;   // [32]
                double* h2 = e2;             // [32]
                int fb = 0;
                // positivity-risk check: min nodal rho or p below a tenth of the element mean (lanes 0, 1)
                if (lane < 2) {
                    const double* q = lane == 0 ? sp : np;
                    double s = 0.0, mn = 1e300;
                    for (int p = 0; p < NP; ++p) {
                        s = s + q[p];
                        mn = fmin(mn, q[p]);
                    }
                    if (mn < 0.1 * (s / 64.0)) fb = 1;
                }
                if (lane < 12) {   // one feature per lane: quantity, direction, order
                    const int wq = lane / 6, i = lane % 6, d = i >> 1, want = NN - 1 - (i & 1);
                    const double* mw = wq ? ep : er;
                    double tot = 0.0, eo = 0.0;
                    for (int p = 0; p < NP; ++p) {
                        const double ee = mw[p];
                        tot = tot + ee;
                        if (((p >> (2 * d)) & 3) == want) eo = eo + ee;
                    }
                    const double f = plog64(eo / tot + 1e-12);
                    feat[lane] = f;
                    const double x = f / 10.0 + 1.0;
                    if (x < a.mlp64[MLP_NW + lane] || x > a.mlp64[MLP_NW + 12 + lane]) fb = 1;
                }
                __syncwarp();   // feat[]: a vote orders no memory
                fb = __any_sync(0xffffffffu, fb);
                const double* W1 = a.mlp64;
                const double* b1 = W1 + 32 * 12;
                const double* W2 = b1 + 32;
                const double* b2 = W2 + 32 * 32;
                const double* W3 = b2 + 32;
                double s = b1[lane];
                for (int i = 0; i < 12; ++i) s = s + W1[lane * 12 + i] * (feat[i] / 10.0 + 1.0);
                h1[lane] = silu64(s);
                __syncwarp();
                s = b2[lane];
                for (int i = 0; i < 32; ++i) s = s + W2[lane * 32 + i] * h1[i];
                h2[lane] = silu64(s);
                __syncwarp();
                if (lane == 0) {
                    double z = W3[32];
                    for (int j = 0; j < 32; ++j) z = z + W3[j] * h2[j];
                    double al = k.alpha_max / (1.0 + pexp64(-z));
                    if (al < k.alpha_min) al = 0.0;
                    if (fb) {
                        atomicAdd(&ctrl->fallback, 1ull);
                        al = am;
                    } else {
                        atomicAdd(&ctrl->judge_sum, fabs(al - am));
                        atomicAdd(&ctrl->judge_n, 1ull);
                    }
                    a.alpha_out[e] = al;
                }
            }
        }
    }
    if (a.epi_dt) {
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) {
            const unsigned long long lam = wmax64(lambda(dd));
            if (lane == 0) s_lam[w][dd] = lam;
        }
        group_sync<ND>(0);
        if (n == 0) {
            const double lf = __longlong_as_double((long long)max(s_lam[0][0], s_lam[1][0]));
            const double lg = __longlong_as_double((long long)max(s_lam[0][1], s_lam[1][1]));
            const double lh = __longlong_as_double((long long)max(s_lam[0][2], s_lam[1][2]));
            const double dte = fmin(fmin(a.delta[e * 3 + 0] / lf, a.delta[e * 3 + 1] / lg), a.delta[e * 3 + 2] / lh);
            const int g = a.group ? a.group[e] : 0;
            atomicMin(&ctrl->dtmin_bits[g], (unsigned long long)__double_as_longlong(dte));
            atomicMax(&ctrl->lmax_bits[g], (unsigned long long)__double_as_longlong(fmax(fmax(lf, lg), lh)));
        }
    }
}

// Per-node primitives of state q at sp[variable * NP]: velocities and, per direction d, beta_d = rho/(2 p_d),
// where p_d is the pressure of the state rotated into direction d (the reference evaluates the two-point flux on
// the rotated state, so the kinetic-energy sum runs in the rotated component order)
template <class A>
__device__ __forceinline__ void velocities64(const double* q, const Rcp64& r, double* sp) {
#pragma unroll
    for (int c = 0; c < 3; ++c) sp[c * NP] = A::quot(q[1 + c], r);
}

template <class A>
__device__ __forceinline__ void beta64(const double* q, const Rcp64& r, int d, double* sp, const OpConsts& k) {
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) {   // q indexed at compile time
        if (dd != d) continue;
        const double u[V] = {q[0], q[1 + dd], q[1 + (dd + 1) % 3], q[1 + (dd + 2) % 3], q[4]};
        sp[(3 + dd) * NP] = A::div(0.5 * q[0], pressure64<A>(u, r, k));
    }
}

template <class A>
__device__ __forceinline__ void primitives64(const double* q, const Rcp64& r, double* sp, const OpConsts& k) {
    velocities64<A>(q, r, sp);
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) beta64<A>(q, r, dd, sp, k);
}

// The fluxes of the 16 lines of direction d into shared memory, by the direction's two warps: two-point fluxes to
// sF, subcell fluxes to sV, face fluxes in the places of their traces in tr.
template <class A, bool BLEND, bool FAST>
__device__ __forceinline__ void fluxes64(int volume_flux, int surface_flux, int d, int w, int lane, double al,
                                         const double* su, double* tr, double* sF, double* sV, const int32_t* s_nbr,
                                         const OpConsts& k) {
    const double* sp = su + (O_SP - O_SU);
    const int c0 = d, c1 = d == 2 ? 0 : d + 1, c2 = d == 0 ? 2 : d - 1;
    const double *m0 = su + (1 + c0) * NP, *m1 = su + (1 + c1) * NP, *m2 = su + (1 + c2) * NP;   // momenta
    constexpr int VEL = O_SP - NP, BETA = O_SP + 2 * NP;   // from a momentum to its velocity, to its beta
    // ---- two-point fluxes, two pairs of the 16 lines at a time: warp 0 pairs 0, 1, 4, 5, warp 1 pairs 2, 3
    //      and then the faces (all pairs on warp 0: 396 against 383 us per stage at Sedov 32^3)
#pragma unroll 1
    for (int g = w; g < 3; g += 2) {
        const int pq = 2 * g + (lane >> 4), ab = lane & 15;
        const int i = line_phys(d, ab, (0x211000 >> (4 * pq)) & 3), m = line_phys(d, ab, (0x332321 >> (4 * pq)) & 3);
        double F[V];
        if (!FAST && volume_flux == NEMO_VOLFLUX_CENTRAL) {
            const double ui[V] = {su[i], m0[i], m1[i], m2[i], su[4 * NP + i]};
            const double um[V] = {su[m], m0[m], m1[m], m2[m], su[4 * NP + m]};
            central64<A>(ui, um, F, k);
        } else {
            const Node5 ni = {su[i], sp[6 * NP + i], m0[VEL + i], m1[VEL + i], m2[VEL + i], m0[BETA + i]};
            const Node5 nm = {su[m], sp[6 * NP + m], m0[VEL + m], m1[VEL + m], m2[VEL + m], m0[BETA + m]};
            chandrashekar64<A>(ni, nm, F, k);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) sF[(v * NPAIR + pq) * FROW + ab] = F[v];
    }
    // ---- Riemann fluxes: round 0 the two faces of the 16 lines (warp 1), rounds 1 and 2 the FV subcell
    //      interfaces 0, 1 (warp 0) and 2 (half of warp 1)
    const int rounds = BLEND && al > 0.0 ? 3 : 1;
#pragma unroll 1
    for (int rt = 1 - w; rt < rounds; rt += 2) {
        const int hi = lane >> 4, ab = lane & 15;
        if (rt == 2 && hi) break;
        const double *pL, *pR;
        int stL = NP, stR = NP;
        int32_t ne = 0;
        double* own_tr = tr + (2 * d + hi) * NF + ab;
        if (rt == 0) {
            ne = s_nbr[2 * d + hi];
            const double* own = su + line_phys(d, ab, hi ? NN - 1 : 0);
            const double* oth = ne == -1 ? own : own_tr;   // domain boundary: the own trace
            const int sto = ne == -1 ? NP : 6 * NF;
            pL = hi ? own : oth;
            pR = hi ? oth : own;
            stL = hi ? NP : sto;
            stR = hi ? sto : NP;
        } else {
            const int qi = 2 * (rt - 1) + hi;
            pL = su + line_phys(d, ab, qi);
            pR = su + line_phys(d, ab, qi + 1);
        }
        const double uL[V] = {pL[0], pL[(1 + c0) * stL], pL[(1 + c1) * stL], pL[(1 + c2) * stL], pL[4 * stL]};
        const double uR[V] = {pR[0], pR[(1 + c0) * stR], pR[(1 + c1) * stR], pR[(1 + c2) * stR], pR[4 * stR]};
        double F[V];
        riem64<A, FAST>(surface_flux, uL, uR, F, k);
        if (rt == 0) {
            if (ne > -2) {   // a mortar's flux row is there already
#pragma unroll
                for (int v = 0; v < V; ++v) own_tr[v * 6 * NF] = F[v];
            }
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) sV[(v * (NN - 1) + 2 * (rt - 1) + hi) * FROW + ab] = F[v];
        }
    }
}

// Node n's terms of direction d, in that direction's component order
template <bool BLEND>
__device__ __forceinline__ void terms64(int d, int n, double al, const double* tr, const double* sF, const double* sV,
                                        const double* s_S, const double* s_winv, double* t) {
    // ---- the node's terms: its three pairs in ascending order of the other node, lift, FV, blend
    const int pos = (n >> (2 * d)) & 3;
    const int ab = d == 0 ? n >> 2 : (d == 1 ? (n & 3) | ((n >> 4) << 2) : n & 15);
    const unsigned rows = (unsigned)(0x0542053104300210ull >> (16 * pos));   // pair rows of this position
#pragma unroll
    for (int v = 0; v < V; ++v) t[v] = 0.0;
#pragma unroll
    for (int mm = 0; mm < NN - 1; ++mm) {
        const double s = s_S[pos * NN + mm + (mm >= pos ? 1 : 0)];
        const double* f = sF + ((rows >> (4 * mm)) & 15) * FROW + ab;
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] = t[v] + s * f[v * NPAIR * FROW];
    }
    const double wi = s_winv[pos];
    const double* sS = tr + 2 * d * NF + ab;   // face fluxes of the line: [v][2][NF]
    if (pos == 0) {
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] = t[v] + wi * (-sS[v * 6 * NF]);
    }
    if (pos == NN - 1) {
#pragma unroll
        for (int v = 0; v < V; ++v) t[v] = t[v] + wi * sS[v * 6 * NF + NF];
    }
    if (BLEND && al > 0.0) {
        const double* fl = pos == 0 ? sS : sV + (pos - 1) * FROW + ab;
        const double* fr = pos == NN - 1 ? sS + NF : sV + pos * FROW + ab;
        const int sl = pos == 0 ? 6 * NF : (NN - 1) * FROW, sr = pos == NN - 1 ? 6 * NF : (NN - 1) * FROW;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double fv = wi * (fr[v * sr] - fl[v * sl]);
            t[v] = (1.0 - al) * t[v] + al * fv;
        }
    }
}

__device__ __forceinline__ void pair_sync(int bar) { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); }

// The node's rhs terms with the language's own quotients, by 64 threads that meet at barrier bar.  Out of line:
// for elements that are not regular, or border one that is not.  The face fluxes of the first attempt stand in
// the places of the traces, so these are fetched again.
struct Terms64 {
    double v[V];
};
__device__ __noinline__ Terms64 plain_terms64(const StageArgs& a, double al, int bar) {
    extern __shared__ __align__(16) double smem[];
    const OpConsts& k = c_ops64;
    const int64_t e = a.E_begin + blockIdx.x;
    const int n = threadIdx.x, lane = n & 31, w = n >> 5, pn = phys(n);
    double *su = smem + O_SU, *sp = smem + O_SP, *tr = smem + O_TR, *sF = smem + O_SF, *sV = smem + O_SV;
    pair_sync(bar);
    double q[V];
    for (int v = 0; v < V; ++v) q[v] = su[v * NP + pn];
    primitives64<Plain64>(q, Plain64::rcp(q[0]), sp + pn, k);
    for (int p = n; p < 6 * NF; p += TPE) {
        const int f = p >> 4, ab = p & 15, ne = a.nbr[e * 6 + f];
        if (ne < 0) continue;   // a mortar's flux row is as it was
        const int m = line_node(f >> 1, ab & 3, ab >> 2, (f & 1) ? 0 : NN - 1);
        for (int v = 0; v < V; ++v) tr[v * 6 * NF + p] = a.u_in[((int64_t)v * a.E + ne) * NP + m];
    }
    pair_sync(bar);
    Terms64 R;
    for (int d = 0; d < 3; ++d) {
        fluxes64<Plain64, true, false>(a.volume_flux, a.surface_flux, d, w, lane, al, su, tr, sF, sV, a.nbr + e * 6, k);
        pair_sync(bar);
        double t[V];
        terms64<true>(d, n, al, tr, sF, sV, k.S, k.winv, t);
        pair_sync(bar);
        const double cd = a.cdel[e * 3 + d];
        const int o[V] = {0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4};
        for (int v = 0; v < V; ++v) R.v[o[v]] = d == 0 ? cd * t[v] : R.v[o[v]] + cd * t[v];
    }
    return R;
}

}  // namespace

// ND directions at a time, each by a group of 64 threads with its own flux arrays.  ND = 1 (64 threads) packs
// an SM with elements; ND = 3 (192 threads) runs an element's directions side by side, which shortens the
// element (26 k cycles alone, 18 k of them the directions) when there are too few to fill the SMs anyway.
template <int ND, bool BLEND, bool RHS_ONLY, bool FAST>
__global__ void __launch_bounds__(ND * TPE, CTAS64 / ND) k_stage_euler64(const __grid_constant__ StageArgs a) {
    extern __shared__ __align__(16) double smem[];
    __shared__ double s_S[NN * NN], s_winv[NN], s_vi[NN * NN];   // operator rows, indexed per thread
    __shared__ double s_alpha;
    __shared__ unsigned long long s_lam[2][4];
    __shared__ int s_bad, s_plain;
    __shared__ int32_t s_nbr[6];

    const OpConsts& k = c_ops64;
    Control* ctrl = a.ctrl;
    const int tid = threadIdx.x, dg = ND == 1 ? 0 : tid / TPE, n = ND == 1 ? tid : tid % TPE, lane = n & 31, w = n >> 5;
    const int64_t E = a.E;
    const int64_t e = a.E_begin + blockIdx.x;
    if (tid < NN * NN) {
        s_S[tid] = k.S[tid];
        s_vi[tid] = k.Vinv[tid];
        if (tid < NN) s_winv[tid] = k.winv[tid];
    }
    // trace nodes p of the six faces this thread fetches: p = tid and, with 64 threads, (warp 0) tid + 64
    constexpr int FETCH = ND == 1 ? 2 : 1;
    int32_t nes[FETCH];
#pragma unroll
    for (int r = 0; r < FETCH; ++r)
        nes[r] = (ND == 1 && r == 0) || tid + r * TPE < 6 * NF ? __ldg(a.nbr + e * 6 + 4 * r + (tid >> 4)) : -1;
    dep_sync();
    const int32_t done = RHS_ONLY ? 0 : ctrl->done;   // looked at when the loads below are under way
    double* const su = smem + O_SU;
    double* const sp = smem + O_SP;
    double* const tr = smem + O_TR;
    constexpr int PER = (BLEND ? ELEM_BLEND : ELEM_PLAIN) - O_SF;   // flux arrays of a direction
    double* const sF = smem + O_SF + dg * PER;
    double* const sV = sF + (O_SV - O_SF);
    double* const sR = smem + O_SF + ND * PER;                       // ND = 3: [2][V][64] rhs terms of y and z

    double q[V];
#pragma unroll
    for (int v = 0; v < V; ++v) q[v] = __ldcg(a.u_in + ((int64_t)v * E + e) * NP + n);
    if (done && !a.prep_only) return;
    auto epilogue = [&]() {
        epilogue64<ND>(a, q[0], pressure64(q, k), sp, s_vi, s_lam, e, n, k, [&](int dd) {
            const double rr[V] = {q[0], q[1 + dd], q[1 + (dd + 1) % 3], q[1 + (dd + 2) % 3], q[4]};
            return xlambda64(rr, k);
        });
    };
    if (a.prep_only) {
        __syncthreads();
        if (dg == 0) epilogue();
        return;
    }

    // neighbour traces (or mortar flux rows) of the 96 face nodes, asynchronously
#pragma unroll
    for (int r = 0; r < FETCH; ++r) {
        const int p = tid + r * TPE, f = p >> 4, ab = p & 15;
        if (!(ND == 1 && r == 0) && p >= 6 * NF) break;
        const int32_t ne = nes[r];
        if (ab == 0) s_nbr[f] = ne;
        if (ne >= 0) {
            const double* g = a.u_in + (int64_t)ne * NP + line_node(f >> 1, ab & 3, ab >> 2, (f & 1) ? 0 : NN - 1);
#pragma unroll
            for (int v = 0; v < V; ++v) cp_async8(tr + v * 6 * NF + p, g + (int64_t)v * E * NP);
        } else if (ne <= -2) {
            const double* g = a.mflux + (int64_t)(-2 - ne) * V * NF + ab;
#pragma unroll
            for (int v = 0; v < V; ++v) cp_async8(tr + v * 6 * NF + p, g + v * NF);
        }
    }
    if (!RHS_ONLY && a.stage > 0 && tid < 4 * V)   // the register rows (four lines each), needed at the end
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.reg + ((int64_t)(tid >> 2) * E + e) * NP + 16 * (tid & 3)));
    if (tid == 0) s_bad = s_plain = 0;
    if (BLEND && tid < 32) smooth_alpha64(a, e, lane, &s_alpha);

    const int pn = phys(n);
    const Rcp64 ir = rcp64r(q[0]);
    if (dg == 0) {
#pragma unroll
        for (int v = 0; v < V; ++v) su[v * NP + pn] = q[v];
        sp[6 * NP + pn] = ir.y;
    }
    if (ND == 1) {
        primitives64<Quick64>(q, ir, sp + pn, k);
    } else {
        if (dg == 0) velocities64<Quick64>(q, ir, sp + pn);
        beta64<Quick64>(q, ir, dg, sp + pn, k);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // Whether this node and the traces this thread fetched keep to the domain of Quick64.  Looked at after the first
    // direction (a vote here, or the second attempt inside the loop, costs more).  us per stage without -> with it:
    // Sedov 32^3 379 -> 392, the 24k-element forest 333 -> 350, smooth 16^3 44.8 -> 46.1, 4^3 9.4 -> 9.4.
    bool regular = k.quick && regular64(q);
#pragma unroll
    for (int r = 0; r < FETCH; ++r) {
        if (nes[r] < 0) continue;
        const double* o = tr + tid + r * TPE;
        const double uo[V] = {o[0], o[6 * NF], o[2 * 6 * NF], o[3 * 6 * NF], o[4 * 6 * NF]};
        regular = regular && regular64(uo);
    }
    __syncthreads();
    if (!regular) s_plain = 1;
    const double al = BLEND ? s_alpha : 0.0;

    // The node's rhs terms, in the component order of the current direction: after each direction the
    // momentum entries are rotated on, so that the loop stays rolled.
    double R[V];
#pragma unroll
    for (int v = 0; v < V; ++v) R[v] = 0.0;
#pragma unroll 1
    for (int d = dg; d < (ND == 1 ? 3 : dg + 1); ++d) {
        const int c0 = d, c1 = d == 2 ? 0 : d + 1, c2 = d == 0 ? 2 : d - 1;
        fluxes64<Quick64, BLEND, FAST>(a.volume_flux, a.surface_flux, d, w, lane, al, su, tr, sF, sV, s_nbr, k);
        group_sync<ND>(dg);
        double t[V];
        terms64<BLEND>(d, n, al, tr, sF, sV, s_S, s_winv, t);
        const double cd = __ldg(a.cdel + e * 3 + d);
        if (ND == 3) {
#pragma unroll
            for (int v = 0; v < V; ++v) R[v] = cd * t[v];
            if (d > 0) {   // x keeps its terms in registers
                double* o = sR + (d - 1) * V * NP + n;
                o[0] = R[0];
                o[(1 + c0) * NP] = R[1];
                o[(1 + c1) * NP] = R[2];
                o[(1 + c2) * NP] = R[3];
                o[4 * NP] = R[4];
            }
        } else {
            double r[V];
#pragma unroll
            for (int v = 0; v < V; ++v) r[v] = d == 0 ? cd * t[v] : R[v] + cd * t[v];
            R[0] = r[0];
            R[1] = r[2];
            R[2] = r[3];
            R[3] = r[1];
            R[4] = r[4];
            __syncthreads();
            if (s_plain) break;
        }
    }
    if (ND == 3) {
        __syncthreads();
        if (dg != 0) return;   // the rest is group 0's
#pragma unroll
        for (int v = 0; v < V; ++v) R[v] = (R[v] + sR[v * NP + n]) + sR[(V + v) * NP + n];
    }
    if (s_plain) {
        const Terms64 p = plain_terms64(a, al, ND == 1 ? 0 : 1);
#pragma unroll
        for (int v = 0; v < V; ++v) R[v] = p.v[v];
    }

    // ---- rhs, LSRK register and state update
    const int64_t g0 = e * NP + n;
    if (RHS_ONLY) {
#pragma unroll
        for (int v = 0; v < V; ++v) a.rhs_out[(int64_t)v * E * NP + g0] = -R[v];
        return;
    }
    const int st = a.stage;
    const double A = rk_a(st);
    const double cdt = rk_c(st) * ctrl->dt[a.group ? a.group[e] : 0];
    double rg[V];
#pragma unroll
    for (int v = 0; v < V; ++v) rg[v] = st == 0 ? 0.0 : a.reg[(int64_t)v * E * NP + g0];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const double rhs = -R[v];
        const double rr = st == 0 ? rhs : A * rg[v] + rhs;
        a.reg[(int64_t)v * E * NP + g0] = rr;
        q[v] = su[v * NP + pn] + cdt * rr;
    }
    if (a.positivity) {
        if (!isvalid64(q, k)) s_bad = 1;
        group_sync<ND>(0);
        if (s_bad) {
            // lanes 0..15 of warp 0 repair the element together on a copy in node order (same
            // arithmetic and order as the serial dgfv_repair_3d)
#pragma unroll
            for (int v = 0; v < V; ++v) sF[v * NP + n] = q[v];
            group_sync<ND>(0);
            if (n < 16) {
                const bool repaired = repair_elem16<1>(sF, 0, n, k);
                if (!repaired && n == 0) atomicAdd(&ctrl->nbad, 1ull);
            }
            group_sync<ND>(0);
#pragma unroll
            for (int v = 0; v < V; ++v) q[v] = sF[v * NP + n];
        }
    }
    // ---- source term after the stage, then store the new state
    if (k.cool) q[4] = cooled_energy64(q, k);
#pragma unroll
    for (int v = 0; v < V; ++v) a.u_out[(int64_t)v * E * NP + g0] = q[v];
    if (st == 4 && a.tick && blockIdx.x == 0 && n == 0) {
        for (int g = 0; g < ctrl->ngroups; ++g) ctrl->t[g] = ctrl->t[g] + ctrl->dt[g];
        ctrl->steps += 1;
    }
    dep_launch();
    epilogue();
}

// Conserved totals: per-element weighted sums in the oracle's order, then a serial sum per
// variable (deterministic, bit-reproducible).  Both are chains of dependent additions; the loads are what
// can be taken off them: elements and chunks pass through shared memory (one thread per element reading its own
// rows, and one thread per variable reading its partial sums, waited for each load).  B200, us per
// nemo_gpu_totals call: Euler 32^3 1046 -> 198, 16^3 161 -> 50, 4^3 49 -> 27; GLM-MHD 32^3 1674 -> 224.
constexpr int TE = 64;            // elements per CTA of the first kernel (one thread each)
constexpr int TROW = NP + 1;      // padded row: the threads walk their rows on different banks

__global__ void __launch_bounds__(TE) k_totals_elem64(const double* __restrict__ u, const double* __restrict__ delta,
                                                      int64_t E, int64_t n, double* __restrict__ part) {
    extern __shared__ double s_u[];   // [TE][TROW]
    const OpConsts& k = c_ops64;
    const int v = blockIdx.y, t = threadIdx.x;
    const int64_t e0 = (int64_t)blockIdx.x * TE;
    const int nel = (int)min((int64_t)TE, n - e0);
    const double* src = u + ((int64_t)v * E + e0) * NP;
#pragma unroll 8
    for (int r = 0; r < nel; ++r) s_u[r * TROW + t] = __ldg(src + r * NP + t);   // an element's row is one coalesced read
    __syncthreads();
    if (t >= nel) return;
    const int64_t e = e0 + t;
    const double vol = delta[e * 3 + 0] * delta[e * 3 + 1] * delta[e * 3 + 2];
    double s = 0.0;
    for (int kk = 0; kk < NN; ++kk)
        for (int j = 0; j < NN; ++j)
            for (int i = 0; i < NN; ++i) s = s + k.wt[i] * k.wt[j] * k.wt[kk] * s_u[t * TROW + nidx(i, j, kk)];
    part[(int64_t)v * n + e] = vol * s;
}

// One CTA per variable: the threads bring the next chunk into shared memory while thread 0 adds up this one.
constexpr int TC = 1024, TSUM = 256;

__global__ void __launch_bounds__(TSUM) k_totals_sum64(const double* __restrict__ part, int64_t n, double* __restrict__ out) {
    __shared__ double s_c[2][TC];
    const double* p = part + (int64_t)blockIdx.x * n;
    const int t = threadIdx.x;
    const int64_t nchunk = (n + TC - 1) / TC;
    auto fetch = [&](int64_t c) {
#pragma unroll
        for (int i = 0; i < TC / TSUM; ++i) {
            const int64_t x = c * TC + t + i * TSUM;
            if (x < n) cp_async8(&s_c[c & 1][t + i * TSUM], p + x);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    double tot = 0.0;
    for (int64_t c = 0; c < nchunk; ++c) {
        if (c + 1 < nchunk) {
            fetch(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (t == 0) {
            const int m = (int)min((int64_t)TC, n - c * TC);
            const double* q = s_c[c & 1];
            if (m == TC) {
#pragma unroll 32
                for (int i = 0; i < TC; ++i) tot = tot + q[i];
            } else {
                for (int i = 0; i < m; ++i) tot = tot + q[i];
            }
        }
        __syncthreads();   // the chunk is free
    }
    if (t == 0) out[blockIdx.x] = tot;
}

// ---------------------------------------------------------------------------------------------
// launchers

static int smem64(int nd, bool blend) {
    return (O_SF + nd * ((blend ? ELEM_BLEND : ELEM_PLAIN) - O_SF) + (nd == 3 ? 2 * V * NP : 0)) * (int)sizeof(double);
}

// Up to so many elements, what the SMs hold at once with ND = 1, three directions at a time (set by the setup).
// B200, us per stage, blended: 64 elements 14.3 -> 9.2, 216 15.0 -> 10.6, 512 17 -> 14, 910 22.6 -> 21.6, 1584
// 31.0 -> 30.5; beyond, the wider CTAs' idle warps cost more than they save: 2197 39.1 -> 39.2, 4096 59.6 -> 65.8,
// 32768 380 -> 491.  With the check of the quotients' domain, smooth flow (few blended elements): 64 14.9 -> 9.6, 216
// 15.9 -> 11.7, 512 18.9 -> 15.5, 910 25.3 -> 24.2, 1584 26.4 -> 27.8, 4096 52.2 -> 63.1.
static int64_t wide_elems64 = 0;

template <int ND>
static cudaError_t launch64(const StageArgs& a, bool blend, bool rhs_only, cudaStream_t s) {
    const unsigned grid = (unsigned)(a.E_own - a.E_begin), nt = ND * TPE;
    const int smem = smem64(ND, blend);
    // the specialised kernel for HLLC faces and Chandrashekar pairs, the general one for the rest
    const bool fast = a.surface_flux == NEMO_SURFFLUX_HLLC && a.volume_flux == NEMO_VOLFLUX_CHANDRASHEKAR;
    if (rhs_only) {
        if (blend) return launch_dep(k_stage_euler64<ND, true, true, false>, grid, nt, smem, s, a);
        return launch_dep(k_stage_euler64<ND, false, true, false>, grid, nt, smem, s, a);
    }
    if (fast) {
        if (blend) return launch_dep(k_stage_euler64<ND, true, false, true>, grid, nt, smem, s, a);
        return launch_dep(k_stage_euler64<ND, false, false, true>, grid, nt, smem, s, a);
    }
    if (blend) return launch_dep(k_stage_euler64<ND, true, false, false>, grid, nt, smem, s, a);
    return launch_dep(k_stage_euler64<ND, false, false, false>, grid, nt, smem, s, a);
}

cudaError_t launch_stage_euler64(const StageArgs& a, bool blend, bool rhs_only, cudaStream_t s) {
    const int64_t n = a.E_own - a.E_begin;
    if (n <= 0) return cudaSuccess;
    return n <= wide_elems64 ? launch64<3>(a, blend, rhs_only, s) : launch64<1>(a, blend, rhs_only, s);
}

// The largest carveout: twelve elements take 220 KB of an SM's shared memory, and the kernel reads
// nothing twice through L1.
template <typename K>
static cudaError_t attrs64(K kernel, int smem) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}

template <int ND>
static cudaError_t setup64() {
    cudaError_t err;
    const int sb = smem64(ND, true), sn = smem64(ND, false);
    if ((err = attrs64(k_stage_euler64<ND, true, true, false>, sb)) != cudaSuccess) return err;
    if ((err = attrs64(k_stage_euler64<ND, false, true, false>, sn)) != cudaSuccess) return err;
    if ((err = attrs64(k_stage_euler64<ND, true, false, false>, sb)) != cudaSuccess) return err;
    if ((err = attrs64(k_stage_euler64<ND, false, false, false>, sn)) != cudaSuccess) return err;
    if ((err = attrs64(k_stage_euler64<ND, true, false, true>, sb)) != cudaSuccess) return err;
    return attrs64(k_stage_euler64<ND, false, false, true>, sn);
}

cudaError_t setup_stage_euler64(const OpConsts& ops) {
    cudaError_t err;
    int dev = 0, nsm = 0;
    if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
    if ((err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return err;
    wide_elems64 = CTAS64 * (int64_t)nsm;
    if ((err = setup64<1>()) != cudaSuccess) return err;
    if ((err = setup64<3>()) != cudaSuccess) return err;
    return cudaMemcpyToSymbol(c_ops64, &ops, sizeof(OpConsts));
}

cudaError_t launch_totals64(const double* u, const double* delta, int64_t E, int64_t n, int nv, double* part,
                            double* out, cudaStream_t s) {
    k_totals_elem64<<<dim3((unsigned)((n + TE - 1) / TE), (unsigned)nv), TE, TE * TROW * sizeof(double), s>>>(u, delta, E, n,
                                                                                                             part);
    k_totals_sum64<<<(unsigned)nv, TSUM, 0, s>>>(part, n, out);
    return cudaGetLastError();
}


// Positivity repair of element states held outside the library (the per-quad kernel_repair of a
// host, source/kernel/mcfv/3d/kernel_validate_mod.f90:27-157): one warp per element [nv][64] (the
// Fortran state(n,n,n,nv) layout); if a node is inadmissible, lanes 0..15 run the cooperative
// dgfv_repair_3d of the stage kernels on it.  ok[e] = 1 if the element is admissible afterwards.
__global__ void __launch_bounds__(32) k_repair_states64(double* __restrict__ st, int64_t n, int nv, int is_mhd,
                                                        int32_t* __restrict__ ok) {
    __shared__ double su[VMAX * NP];
    const OpConsts& k = c_ops64;
    const int64_t e = blockIdx.x;
    const int lane = threadIdx.x;
    double* g = st + e * (int64_t)nv * NP;
    for (int p = lane; p < nv * NP; p += 32) su[p] = g[p];
    __syncwarp();
    bool valid = true;
    for (int p = lane; p < NP; p += 32) {
        double q[VMAX];
        for (int v = 0; v < nv; ++v) q[v] = su[v * NP + p];
        valid = valid && (is_mhd ? m_isvalid<double>(q, k.kappa, k.mu0) : isvalid64(q, k));
    }
    bool good = __all_sync(0xffffffffu, valid);
    if (!good) {
        bool rep = false;
        if (lane < 16) rep = is_mhd ? repair_elem16_mhd<1>(su, 0, lane, k) : repair_elem16<1>(su, 0, lane, k);
        good = __shfl_sync(0xffffffffu, rep, 0);
        __syncwarp();
        for (int p = lane; p < nv * NP; p += 32) g[p] = su[p];
    }
    if (lane == 0) ok[e] = good ? 1 : 0;
}

cudaError_t launch_repair_states64(double* st, int64_t n, int nv, int mhd, int32_t* ok, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (n > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_repair_states64<<<(unsigned)n, 32, 0, s>>>(st, n, nv, mhd, ok);
    return cudaGetLastError();
}

}  // namespace nemo

// ---- GLM-MHD stage
#include "stage_mhd64.cuh"
