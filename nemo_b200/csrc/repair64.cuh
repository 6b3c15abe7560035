// repair64.cuh -- positivity repair of one element held in shared memory (FP64, rare path).
#pragma once

#include "common.cuh"
#include "euler_fp64.cuh"
#include "mhd_phys.cuh"

namespace nemo {

// dgfv_repair_3d (source/kernel/mcfv/3d/kernel_validate_mod.f90:159-272) with N_NODES = 4: if a
// node is inadmissible, squeeze 2x2x2 tiles of node means towards their mean in steps of
// repair_decr until the tile means are admissible, first on the 8 octants (2^3 nodes each), then
// node by node inside each octant.  su holds the tile's state [V][EPC][64].  The element's 16 threads
// (a half-warp that calls it as a whole) work together, for V variables and an admissibility test
// valid(q): no per-thread tile arrays, so it inlines without a call frame.  Level 1 squeezes the 8 octants
// (lanes 0..7, one octant each); level 2 squeezes the 8 nodes of each octant (lanes 0..7 and 8..15
// take one octant each, four rounds).  Each lane sums its tile in the serial routine's node order,
// the means run over the tiles in tile order, and all lanes of a block take the same squeeze steps.
template <int EPC, int V, typename Valid>
__device__ __forceinline__ bool repair_coop16(double* su, int el, int lane, double decr, Valid valid) {
    auto at = [&](int v, int p) -> double& { return su[(v * EPC + el) * NP + p]; };
    const unsigned half = threadIdx.x & 16;
#pragma unroll 1
    for (int level = 1; level <= 2; ++level) {
        const int rounds = level == 1 ? 1 : 4;
#pragma unroll 1
        for (int rd = 0; rd < rounds; ++rd) {
            const int grp = lane >> 3, t = lane & 7;
            const bool use = level == 2 || grp == 0;
            const unsigned gm = 0xffu << (half + 8 * grp);   // the 8 lanes of this block
            const int ii = t & 1, jj = (t >> 1) & 1, kk = t >> 2;
            // block origin (level 2: octant (q, pp, r) = blk bits) and the tile's node range
            const int blk = level == 1 ? 0 : 2 * rd + grp;
            const int q = blk & 1, pp = (blk >> 1) & 1, r = blk >> 2;
            const int nn = level == 1 ? 2 : 1;
            const int i0 = level == 1 ? 2 * ii : 2 * q + ii;
            const int j0 = level == 1 ? 2 * jj : 2 * pp + jj;
            const int k0 = level == 1 ? 2 * kk : 2 * r + kk;
            const double ws = level == 1 ? 0.125 : 1.0;
            double tile[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                double acc = 0.0;
                if (use)
                    for (int kx = k0; kx < k0 + nn; ++kx)
                        for (int jx = j0; jx < j0 + nn; ++jx)
                            for (int ix = i0; ix < i0 + nn; ++ix) acc = acc + ws * at(v, nidx(ix, jx, kx));
                tile[v] = acc;
            }
            if (!use) continue;
            const bool bad = !valid(tile);
            if (__ballot_sync(gm, bad) == 0u) continue;   // the block's tiles are admissible
            double mean[V], hile[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                double sum = 0.0;
#pragma unroll
                for (int tt = 0; tt < 8; ++tt) sum = sum + __shfl_sync(gm, tile[v], (int)(half + 8 * grp) + tt);
                mean[v] = 0.125 * sum;
                hile[v] = tile[v] - mean[v];
            }
            double squeeze = 1.0;
#pragma unroll 1
            while (squeeze > 0.0) {
                squeeze = fmax(0.0, squeeze - decr);
                double tv[V];
#pragma unroll
                for (int v = 0; v < V; ++v) tv[v] = mean[v] + squeeze * hile[v];
                if (__ballot_sync(gm, !valid(tv)) == 0u) break;
            }
            for (int kx = k0; kx < k0 + nn; ++kx)
                for (int jx = j0; jx < j0 + nn; ++jx)
                    for (int ix = i0; ix < i0 + nn; ++ix) {
                        const int p = nidx(ix, jx, kx);
#pragma unroll
                        for (int v = 0; v < V; ++v) at(v, p) = mean[v] + squeeze * (at(v, p) - mean[v]);
                    }
        }
        __syncwarp(0xffffu << half);
    }
    bool ok = true;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int p = lane + 16 * m;
        double qv[V];
#pragma unroll
        for (int v = 0; v < V; ++v) qv[v] = at(v, p);
        ok = ok && valid(qv);
    }
    return __ballot_sync(0xffffu << half, !ok) == 0u;
}

template <int EPC>
__device__ __forceinline__ bool repair_elem16(double* su, int el, int lane, const OpConsts& k) {
    return repair_coop16<EPC, 5>(su, el, lane, k.repair_decr, [&](const double* q) { return isvalid64(q, k); });
}

template <int EPC>
__device__ __forceinline__ bool repair_elem16_mhd(double* su, int el, int lane, const OpConsts& k) {
    return repair_coop16<EPC, 9>(su, el, lane, k.repair_decr,
                                 [&](const double* q) { return m_isvalid<double>(q, k.kappa, k.mu0); });
}

}  // namespace nemo
