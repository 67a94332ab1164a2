// msk_wide.cuh -- the wave chain of one unit on a 512^2 or 1024^2 grid in one
// cooperative launch over many SMs (a single calculate() call, a tilt series of
// one orientation), as k_small_wave (msk_small.cuh) is for smaller grids.
//
// A slice is a transmit and a propagator; as launches each took 10-12 us for one
// unit, most of it launch latency and one CTA's dependent chain.  Here Q CTAs
// stay resident (cooperative launch), CTA r owning LPC rows and LPC columns, and
// the two phases of a slice are separated by barriers among the CTAs through a
// counter in global memory; every wait has a limit, after which the error flag
// is set and every CTA returns.  The transmissions come as iS(B_k), made
// beforehand for a group of slices, and are fetched before the barrier that W
// waits for.  Rows and columns run the 32-point plan's transforms with the same
// roundings as the launch loop's passes: the same bits.
//
// Bound: the chain of each phase (L2 round trip, two transforms, barrier), 9.6 us
// a slice at 512^2 and 13.6 at 1024^2.  A calculate() call of 96 slices of 512^2
// takes 1.71 ms with it and 2.14 without, 160 slices of 1024^2 5.40 and 5.72.
// 128 CTAs: the largest power of two that fits 152 SMs, 4 or 8 lines a CTA.
#pragma once

#include "msk_small.cuh"

namespace msk {

template <int N>
struct WideCfg {
    static constexpr bool OK = N == 512 || N == 1024;
    using P = FftPlan<N>;
    static constexpr int T = P::T, E = P::E;
    static constexpr int Q = 128;          // CTAs
    static constexpr int LPC = N >= Q ? N / Q : 1;  // rows and columns of a CTA
    static constexpr int NT = LPC * T;
    static constexpr size_t SMEM = (size_t)LPC * P::PADN * 8;
};

// Barrier among the CTAs of the launch: `count` counts arrivals, `target` is what
// it reaches when all have come.  Every thread's earlier global writes are
// visible to every CTA after it.  False (in every thread) when the wait ran out.
__device__ __forceinline__ bool launch_sync(unsigned *count, unsigned target, int *err)
{
    __syncthreads();
    int late = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        const long long t0 = clock64();
        for (;;) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
            if (c >= target) break;
            if (clock64() - t0 > kWaitCycles) {
                atomicOr(err, kErrWaitTimeout);
                late = 1;
                break;
            }
        }
        __threadfence();
    }
    return !__syncthreads_or(late);
}

// Slices s0 .. s1-1 of the one unit; t: grid k - s0 is iS(B_k); `count` zeroed.
template <int N>
__global__ void __launch_bounds__(WideCfg<N>::NT, 1)
k_wide_wave(const Geom g, int s0, int s1, const int *__restrict__ so, const float2 *__restrict__ t,
            float2 *W, int arbitrary, unsigned *count)
{
    using C = WideCfg<N>;
    constexpr int T = C::T, E = C::E, LPC = C::LPC, PADN = C::P::PADN;
    extern __shared__ __align__(128) unsigned char smem[];
    float2 *sm = reinterpret_cast<float2 *>(smem);
    const int rank = blockIdx.x;
    const size_t plane = (size_t)N * N;
    const int rl = threadIdx.x / T, rt = threadIdx.x % T, row = rank * LPC + rl;
    const int cc = threadIdx.x % LPC, ct = threadIdx.x / LPC, col = rank * LPC + cc;
    const bool in_band = rank * LPC <= g.band_p || rank * LPC + LPC - 1 >= g.band_q;
    float2 *wrow = W + (size_t)row * N;
    unsigned target = 0;
    float2 q[E];
    auto fetch = [&](int k) {  // t_k on this row
        const float2 *src = t + (size_t)(k - s0) * plane + (size_t)row * N;
#pragma unroll
        for (int m = 0; m < E; m++) q[m] = __ldg(&src[rt + m * T]);
    };
    bool has_k = so[s0 + 1] > so[s0];
    if (has_k) fetch(s0);
    for (int k = s0; k < s1; k++) {
        const bool has_n = k + 1 < s1 && so[k + 2] > so[k + 1];
        const bool full = arbitrary && k == s0;  // W not yet zero out of band
        if (has_k) {
            float2 *xb = sm + rl * PADN;
            float2 v[E];
#pragma unroll
            for (int m = 0; m < E; m++)
                v[m] = band_zero<E>(m) && !full ? make_float2(0.0f, 0.0f) : __ldcg(&wrow[rt + m * T]);
            fft_line<N, true, 1, 0>(v, xb, 0, rt, g.tw_row);
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = cmul(v[m], q[m]);
            fft_line<N, false, 1, 0>(v, xb, 0, rt, g.tw_row);
#pragma unroll
            for (int m = 0; m < E; m++)
                if (!band_zero<E>(m) && !out_of_band(g, rt + m * T)) wrow[rt + m * T] = v[m];
        }
        if (has_n) fetch(k + 1);
        if (has_k && !launch_sync(count, target += C::Q, g.err)) return;
        if (in_band || full) {
            float2 v[E];
#pragma unroll
            for (int m = 0; m < E; m++) v[m] = __ldcg(&W[(size_t)(ct + m * T) * N + col]);
            fft_line<N, false, LPC, 1>(v, sm, cc, ct, g.tw_col);
            const int2 ab = __ldg(&g.kband[col]);
            const float2 py = __ldg(&g.propy[col]);
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int ix = ct + m * T;
                v[m] = !band_zero<E>(m) && (ix <= ab.x || ix >= ab.y)
                           ? cmul(cmul(v[m], py), __ldg(&g.propx[ix]))
                           : make_float2(0.0f, 0.0f);
            }
            fft_line<N, true, LPC, 1>(v, sm, cc, ct, g.tw_col);
#pragma unroll
            for (int m = 0; m < E; m++) W[(size_t)(ct + m * T) * N + col] = v[m];
        }
        if (has_n) {
            if (!launch_sync(count, target += C::Q, g.err)) return;
        } else {
            __syncthreads();  // the columns' exchange is read
        }
        has_k = has_n;
    }
}

}  // namespace msk
