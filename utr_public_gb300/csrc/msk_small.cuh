// msk_small.cuh -- the wave chain of a small grid's slice loop in one launch: one
// thread-block cluster per unit (orientation x configuration).
//
// For N x N grids with N <= 256 a unit's wave W = S(psi) stays in L2, and a
// slice-step is too small to fill the GPU from one launch per pass.  The
// transmissions do not depend on the wave: those of a group of slices are made
// beforehand by full launches (splat, band limit, row inverse; run_slices), t[(k -
// s0) * nunits + u] = iS(B_k), and a cluster of Q CTAs then runs the unit's slices,
// CTA r owning LPC rows and LPC columns:
//
//   row phase     W = S(iS(W) t_k)   on the CTA's rows (P3), t_k fetched before
//                                    the barrier that W waits for
//   column phase  W = iF(P F(W))/nx  on the CTA's columns (P4)
//
// with a cluster barrier (release / acquire, so every CTA's global writes of one
// phase are visible to the others in the next) after each, none after the columns
// of a slice whose successor has no atoms: they stay with their CTA.  Every row and
// column is computed with the line transforms and multipliers of the multi-launch
// passes (k_col_pass, k_row_transmit) on the 16-points-a-thread plan
// (FftPlan<N, 16>: twice the threads per line, half the serial chain).  Loads of
// data another CTA wrote go through L2 (ld.global.cg).  Bound: the chain of L2
// round trips, two transforms and a barrier of each phase.  One unit of 256^2, 32
// slices: 0.18 ms; 0.47 ms when the other half of each CTA splatted and
// band-limited the next slice between the same barriers -- the atom scan was the
// longest chain of a slice.  Every CTA arrives at every cluster barrier.
#pragma once

#include "msk_passes.cuh"

namespace msk {

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Every thread of the cluster: this CTA's earlier writes (global and shared)
// visible to every CTA of the cluster after it.
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int N>
struct SmallWaveCfg {
    static constexpr int EV = 16;
    using P = FftPlan<N, EV>;
    static constexpr int T = P::T, E = P::E;
    static constexpr int LPC = N >= 256 ? 16 : 8;  // rows and columns of a CTA
    static constexpr int Q = N / LPC;
    // CTAs an SM up to which a call's clusters beat the launch loop (small_grid_ok)
    static constexpr int PER = N >= 256 ? 1 : N >= 128 ? 2 : 8;
    static constexpr int NT = LPC * T;
    static constexpr size_t SMEM = (size_t)LPC * P::PADN * 8;
    static_assert(NT % 32 == 0 && T <= 32, "whole warps of whole lines");
};

template <int N>
__global__ void __launch_bounds__(SmallWaveCfg<N>::NT, 1)
k_small_wave(const Geom g, int nunits, int s0, int s1, int nsl1, const int *__restrict__ slice_off,
             const float2 *__restrict__ t, float2 *W, int arbitrary)
{
    using C = SmallWaveCfg<N>;
    constexpr int T = C::T, E = C::E, LPC = C::LPC, EV = C::EV, PADN = C::P::PADN;
    extern __shared__ __align__(128) unsigned char smem[];
    float2 *sm = reinterpret_cast<float2 *>(smem);
    const int rank = (int)cluster_rank();
    const int u = blockIdx.x / C::Q;
    const size_t plane = (size_t)N * N;
    float2 *Wu = W + (size_t)u * plane;
    const int *so = slice_off + (size_t)u * nsl1;
    const int rl = threadIdx.x / T, rt = threadIdx.x % T, row = rank * LPC + rl;
    const int cc = threadIdx.x % LPC, ct = threadIdx.x / LPC, col = rank * LPC + cc;
    const bool in_band = rank * LPC <= g.band_p || rank * LPC + LPC - 1 >= g.band_q;
    float2 *wrow = Wu + (size_t)row * N;
    float2 q[E];
    auto fetch = [&](int k) {  // t_k on this row
        const float2 *src = t + ((size_t)(k - s0) * nunits + u) * plane + (size_t)row * N;
#pragma unroll
        for (int m = 0; m < E; m++) q[m] = __ldg(&src[rt + m * T]);
    };
    bool has_k = so[s0 + 1] > so[s0];
    if (has_k) fetch(s0);
    for (int k = s0; k < s1; k++) {
        const bool has_n = k + 1 < s1 && so[k + 2] > so[k + 1];
        // the wave is arbitrary (not yet zero out of band) before its first
        // propagator pass
        const bool full = arbitrary && k == s0;
        if (has_k) {
            float2 *xb = sm + rl * PADN;
            float2 v[E];
#pragma unroll
            for (int m = 0; m < E; m++)
                v[m] = band_zero<E>(m) && !full ? make_float2(0.0f, 0.0f) : __ldcg(&wrow[rt + m * T]);
            fft_line<N, true, 1, 0, EV>(v, xb, 0, rt, g.tw_row16);
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = cmul(v[m], q[m]);
            fft_line<N, false, 1, 0, EV>(v, xb, 0, rt, g.tw_row16);
#pragma unroll
            for (int m = 0; m < E; m++)
                if (!band_zero<E>(m) && !out_of_band(g, rt + m * T)) wrow[rt + m * T] = v[m];
        }
        if (has_n) fetch(k + 1);
        if (has_k) cluster_sync();
        if (in_band || full) {
            float2 v[E];
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = __ldcg(&Wu[(size_t)(ct + m * T) * N + col]);
            fft_line<N, false, LPC, 1, EV>(v, sm, cc, ct, g.tw_col16);
            const int2 ab = __ldg(&g.kband[col]);
            const float2 py = __ldg(&g.propy[col]);
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int ix = ct + m * T;
                v[m] = !band_zero<E>(m) && (ix <= ab.x || ix >= ab.y)
                           ? cmul(cmul(v[m], py), __ldg(&g.propx[ix]))
                           : make_float2(0.0f, 0.0f);
            }
            fft_line<N, true, LPC, 1, EV>(v, sm, cc, ct, g.tw_col16);
#pragma unroll
            for (int m = 0; m < E; m++) Wu[(size_t)(ct + m * T) * N + col] = v[m];
        }
        if (has_n) cluster_sync();
        else __syncthreads();  // the columns' exchange is read
        has_k = has_n;
    }
}

}  // namespace msk
