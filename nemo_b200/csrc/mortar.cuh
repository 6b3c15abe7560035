// mortar.cuh -- one pair of 2:1 mortars processed by 128 threads (64 per mortar, one per sub-face
// node): coarse trace staged in shared memory and prolonged (tensor product of the 1D interpolation
// matrices), Riemann flux against the fine quad's trace in the face's rotated frame (plus, for MHD,
// each side's non-conservative term), the fine rows written directly and the coarse row projected
// (1D projection matrices), sums in the oracle's order (oracle mortar_fluxes).  A prolonged sub-face
// trace with an inadmissible node (a strong shock on the coarse side) is replaced by the coarse face's
// mean, which is admissible; the reference interpolates without this guard.  Used by the mortar
// kernel (mortar.cu) and by the persistent FP32 stage kernel, which runs the mortar pairs as its
// first tasks and publishes each mortar with a release flag (epoch) that its element tiles acquire.
// Reference: the mortar part of kernel_fill_faceflux, source/kernel/mcfv/3d/kernel_flux_mod.f90:
// 100-118 and 252-269, with kernel_operators_interpolationMatrix / _projectionMatrix,
// source/kernel/dgsem/weakform/2d/kernel_operators_mod.f90:1010-1100.
#pragma once

#include "euler_fp64.cuh"
#include "kernels.h"
#include "mhd_fp64.cuh"

namespace nemo {
namespace mortar {

constexpr int MPB = 2;          // mortars per 128-thread task
// per mortar: coarse trace [V][16], half-prolonged trace [V][32], later half-projected fluxes [V][64], and the
// sub-face fluxes [4][V][16]; once per task the two pairs of 1D matrices
constexpr int scratch_doubles(int V) { return MPB * (V * NF + V * 64 + 4 * V * NF) + 4 * NN * NN; }
constexpr int SCRATCH_DOUBLES = scratch_doubles(9);

// The surface fluxes in Plain64, out of line: few nodes take them.  States go by value, so that those of the
// other path stay in registers.
template <int N>
struct Vec64 {
    double v[N];
};

template <int N>
__device__ __forceinline__ Vec64<N> vec64(const double* u) {
    Vec64<N> r;
#pragma unroll
    for (int v = 0; v < N; ++v) r.v[v] = u[v];
    return r;
}

template <int N>
__device__ __forceinline__ void take(double* F, const Vec64<N>& r) {
#pragma unroll
    for (int v = 0; v < N; ++v) F[v] = r.v[v];
}

static __device__ __noinline__ Vec64<5> riem64_plain(int kind, Vec64<5> uL, Vec64<5> uR, const OpConsts& k) {
    Vec64<5> F;
    riem64<Plain64, false>(kind, uL.v, uR.v, F.v, k);
    return F;
}

static __device__ __noinline__ Vec64<9> m_riem64_plain(int kind, Vec64<9> uL, Vec64<9> uR, const OpConsts& k, double ch) {
    Vec64<9> F;
    if (kind == NEMO_SURFFLUX_HLLD) m_hlld64<Plain64>(uL.v, uR.v, F.v, mhd64<true>(k, ch));
    else m_rusanov64<Plain64>(uL.v, uR.v, F.v, mhd64<false>(k, ch));
    return F;
}

// LGL-weighted mean of a coarse face trace held as [V][NF] (out of line: taken only on a shock)
static __device__ __noinline__ void face_mean(const double* uc, int V, double* out, const OpConsts& k) {
    for (int v = 0; v < V; ++v) {
        double acc = 0.0;
        for (int bb = 0; bb < NN; ++bb)
            for (int aa = 0; aa < NN; ++aa) acc = acc + (k.wt[aa] * k.wt[bb]) * uc[v * NF + aa + NN * bb];
        out[v] = acc;
    }
}

template <bool MHD>
__device__ __forceinline__ void mortar_pair(const MortarArgs& a, int64_t pair, double* scratch, const OpConsts& k) {
    constexpr int V = MHD ? 9 : 5;
    auto s_uc = reinterpret_cast<double (*)[V][NF]>(scratch);                       // [MPB][V][NF]
    auto s_in = reinterpret_cast<double (*)[V][64]>(scratch + MPB * V * NF);         // [MPB][V][64]
    auto s_fs = reinterpret_cast<double (*)[4][V][NF]>(scratch + MPB * V * (NF + 64));   // [MPB][4][V][NF]
    double* s_pro = scratch + MPB * V * (NF + 64 + 4 * NF);                          // [2][16], then prj [2][16]
    double* s_prj = s_pro + 2 * NN * NN;
    const int ml = threadIdx.x >> 6, r = threadIdx.x & 63;
    const int64_t m = pair * MPB + ml;
    const bool act = m < a.nm;
    const int32_t* t = a.mortar + 6 * (act ? m : 0);
    const int64_t E = a.E;
    const int64_t qc = t[0];
    const int fc = t[1], ff = fc ^ 1, d = fc >> 1;
    const bool coarse_left = (fc & 1) != 0;
    const int kq = r >> 4, i = r & 3, j = (r >> 2) & 3;
    const int s = kq & 1, tt = kq >> 1;
    double up[V], uf[V];
    if (threadIdx.x < 4 * NN * NN)   // the matrices are indexed per thread: shared, not constant memory
        s_pro[threadIdx.x] = threadIdx.x < 2 * NN * NN ? k.pro[threadIdx.x >> 4][threadIdx.x & 15]
                                                       : k.prj[(threadIdx.x >> 4) & 1][threadIdx.x & 15];
    if (act && r < NF) {
        const int n = line_node(d, r & 3, r >> 2, (fc & 1) ? NN - 1 : 0);
#pragma unroll
        for (int v = 0; v < V; ++v) s_uc[ml][v][r] = a.u_in[((int64_t)v * E + qc) * NP + n];
    }
    if (act) {
        const int64_t qf = t[2 + kq];
        const int nf = line_node(d, i, j, (ff & 1) ? NN - 1 : 0);
#pragma unroll
        for (int v = 0; v < V; ++v) uf[v] = a.u_in[((int64_t)v * E + qf) * NP + nf];
    }
    __syncthreads();
    // prolongation, one axis at a time: the first axis of a row is shared by the four nodes and two sub-faces
    // along the second
    if (act)
        for (int p = r; p < 32 * V; p += 64) {
            const int v = p >> 5, row = p & 31, bb = row & 3;   // row = (half, node i, bb)
            double in = 0.0;
#pragma unroll
            for (int aa = 0; aa < NN; ++aa) in = in + s_pro[(row >> 2) * NN + aa] * s_uc[ml][v][aa + NN * bb];
            s_in[ml][v][row] = in;
        }
    __syncthreads();
    if (act) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            double acc = 0.0;
#pragma unroll
            for (int bb = 0; bb < NN; ++bb) acc = acc + s_pro[tt * NN * NN + j * NN + bb] * s_in[ml][v][s * NF + i * NN + bb];
            up[v] = acc;
        }
        // a sub-face (16 lanes of this warp; act is warp-uniform) whose prolonged trace has an
        // inadmissible node takes the coarse face's mean instead, as the oracle does
        bool okn;
        if constexpr (MHD) okn = m_isvalid<double>(up, k.kappa, k.mu0);
        else okn = isvalid64(up, k);
        const unsigned badl = __ballot_sync(0xffffffffu, !okn);
        if (badl & (0xffffu << (16 * (kq & 1)))) face_mean(&s_uc[ml][0][0], V, up, k);
        // rotate into the face frame: component c of momentum (and field) -> original (d + c) % 3
        double rp[V], rf[V];
        rp[0] = up[0];
        rf[0] = uf[0];
        rp[4] = up[4];
        rf[4] = uf[4];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            rp[1 + c] = up[1 + (d + c) % 3];
            rf[1 + c] = uf[1 + (d + c) % 3];
        }
        if (MHD) {
            rp[8] = up[8];
            rf[8] = uf[8];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                rp[5 + c] = up[5 + (d + c) % 3];
                rf[5 + c] = uf[5 + (d + c) % 3];
            }
        }
        double uL[V], uR[V];   // by selection, not by pointer (which would put the arrays in local memory)
#pragma unroll
        for (int v = 0; v < V; ++v) {
            uL[v] = coarse_left ? rp[v] : rf[v];
            uR[v] = coarse_left ? rf[v] : rp[v];
        }
        double F[V], Gf[V], Gc[V];
        double* out = a.mflux + ((5 * m + 1 + kq) * V) * NF + (i + NN * j);
        if constexpr (MHD) {
            const double ch = a.ctrl->glm_ch;
            const double h = 0.5 / k.mu0;
            if (!(k.quick && m_regular64(up, h) && m_regular64(uf, h))) take(F, m_riem64_plain(a.surface_flux, vec64<9>(uL), vec64<9>(uR), k, ch));
            else if (a.surface_flux == NEMO_SURFFLUX_HLLD) m_hlld64<Quick64>(uL, uR, F, mhd64<true>(k, ch));
            else m_rusanov64<Quick64>(uL, uR, F, mhd64<false>(k, ch));
            m_nc_x<double>(rf, uL, uR, Gf, k.mu0);
            m_nc_x<double>(rp, uL, uR, Gc, k.mu0);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                out[v * NF] = F[v] + Gf[v];
                s_fs[ml][kq][v][i + NN * j] = F[v] + Gc[v];
            }
        } else {
            if (!(k.quick && regular64(up) && regular64(uf))) take(F, riem64_plain(a.surface_flux, vec64<5>(uL), vec64<5>(uR), k));
            else riem64<Quick64, false>(a.surface_flux, uL, uR, F, k);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                out[v * NF] = F[v];
                s_fs[ml][kq][v][i + NN * j] = F[v];
            }
        }
    }
    __syncthreads();
    // projection, one axis at a time: thread (kq, jj, aa) the first, then the coarse nodes sum over the
    // sub-faces and jj in the oracle's order
    if (act) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            double in = 0.0;
#pragma unroll
            for (int ii = 0; ii < NN; ++ii) in = in + s_prj[s * NN * NN + i * NN + ii] * s_fs[ml][kq][v][ii + NN * j];
            s_in[ml][v][r] = in;
        }
    }
    __syncthreads();
    if (act) {
        double* out = a.mflux + (5 * m * V) * NF;
        for (int p = r; p < NF * V; p += 64) {
            const int v = p >> 4, aa = p & 3, bb = (p >> 2) & 3;
            double acc = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int jj = 0; jj < NN; ++jj)
                    acc = acc + s_prj[(q >> 1) * NN * NN + bb * NN + jj] * s_in[ml][v][q * NF + jj * NN + aa];
            out[p] = acc;
        }
    }
    if (a.mflag) {  // publish: the mortar's five flux rows are complete for this epoch
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0 || threadIdx.x == 64) {
            if (act) {
                __threadfence();
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.mflag + m), "r"(a.epoch) : "memory");
            }
        }
    }
}

}  // namespace mortar
}  // namespace nemo
