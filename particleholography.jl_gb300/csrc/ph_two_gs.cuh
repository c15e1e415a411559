// ph_two_gs.cuh -- the Gerchberg-Saxton passes and the passes of a propagation on
// the two-stage row transform.
//
// A pass reads whole rows, transforms them, applies a product or an amplitude to the
// values that a thread holds, transforms back with the mirrored plan and stores
// transposed: one exchange per transform.  4 rows per CTA, one or two warps (or half
// a warp) per row.  What bounds it is latency: at 1024^2 a pass is 256 CTAs that run
// once, so its time is one row's (loads, four butterflies stages, two exchanges)
// plus the launch, which overlaps the previous pass's end (programmatic dependent
// launch).  Per pass, against the one-shot passes of the row engine: 2.7 us (12.6)
// at 256^2, 6.1 us (19.2) at 768^2.  A whole propagation at 2048^2, its transfer
// formed as the rows that the column pass reads: 90 us (the row engine's 99, with
// the transfers gathered).
#pragma once

#include "ph_launch.cuh"
#include "ph_two.cuh"

namespace ph {
namespace two {

enum GsMode {
    GS_COL = 0,        // rows kx: forward, times ht[kx][ky], inverse, transposed store
    GS_ROW = 1,        // rows y: inverse, amplitude replacement, forward, transposed store
    GS_ROW_FINAL = 2,  // inverse, amplitude replacement, natural store
    GS_ROW_INV = 3,    // inverse, natural store
};

template <int N>
struct PassG {
    using PL = Plan<N>;
    static constexpr int RB = 4;
    static constexpr int THREADS = RB * PL::L;
    static constexpr int PITCH = N + 4;                      // elements between staged rows
    static constexpr size_t STAGE = (size_t)RB * PITCH * 8;
    static constexpr size_t XB = (size_t)Mirror<N>::XWORDS * 4;
    static constexpr size_t SMEM = STAGE + RB * XB;
    static constexpr int CTAS = 256 / THREADS;
};

template <int N, int MODE, bool RESID>
__global__ void __launch_bounds__(PassG<N>::THREADS, PassG<N>::CTAS) k_two_gs(const GsParams p) {
    using C = PassG<N>;
    using PL = Plan<N>;
    constexpr int E = PL::E, L = PL::L, M = PL::M;
    constexpr bool INV1 = MODE != GS_COL;                    // direction of the first transform
    constexpr bool BACK = MODE == GS_COL || MODE == GS_ROW;  // there is a second one
    constexpr bool AMP = MODE == GS_ROW || MODE == GS_ROW_FINAL;
    constexpr bool EARLY = M == 1 && E <= 32;                // the operands fit beside the transform's values
    extern __shared__ __align__(128) unsigned char ph_smem[];
    const int r = threadIdx.x / L, l = threadIdx.x % L;
    float *ex = reinterpret_cast<float *>(ph_smem + C::STAGE + r * C::XB);
    const auto sync = [&] {
        if constexpr (L <= 32) __syncwarp();
        else named_bar_sync(1 + r, L);
    };
    const int row0 = blockIdx.x * C::RB, row = row0 + r;
    const bool valid = row < p.nrows;
    const size_t at = (size_t)min(row, p.nrows - 1) * N;     // (rows beyond the last: its values again, not stored)
    grid_dependents_launch();
    grid_dependency_wait();                                  // the previous pass wrote src and may still read dst

    // the operand of value k = l + L m + E o: the transfer or the amplitude
    const auto operand = [&](int m, int o) -> float2 {
        const int k = (M * L == E ? l + L * m : min(l + L * m, E - 1)) + E * o;
        if constexpr (MODE == GS_COL) return __ldg(p.ht + at + k);
        else if constexpr (AMP) return make_float2(__ldg(p.amp + at + k), 0.0f);
        else return make_float2(0.0f, 0.0f);
    };
    float2 op[L];   // EARLY: fetched before the exchange; else one transform at a time
    float2 u[M * L];
    {
        float2 v[E], w[E], z[M * L];
        level1<E, INV1>(w, [&](int i) { return p.src[at + l + L * i]; });
        level2<E, INV1>(w, [&](int o, float2 x) { v[o] = stage_twiddle<INV1>(p.tw, twiddle_offset(N), o, L, l, x); });
        if constexpr (EARLY) {
#pragma unroll
            for (int o = 0; o < L; ++o) op[o] = operand(0, o);
        }
        exchange<N>(v, z, ex, l, sync);
        double acc0 = 0.0, acc1 = 0.0;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if constexpr (!EARLY) {
#pragma unroll
                for (int o = 0; o < L; ++o) op[o] = operand(m, o);
            }
            float2 q[L];
            level1<L, INV1>(q, [&](int i) { return z[m * L + i]; });
            const bool live = M * L == E || l + L * m < E;
            level2<L, INV1>(q, [&](int o, float2 x) {
                if constexpr (RESID) {
                    if (valid && live) {
                        const double d = sqrt((double)x.x * x.x + (double)x.y * x.y) - (double)op[o].x;
                        acc0 += d * d;
                        acc1 += (double)op[o].x * op[o].x;
                    }
                }
                const float2 g = MODE == GS_COL ? cmul2(x, op[o]) : AMP ? amplitude_replace(x, op[o].x) : x;
                if constexpr (BACK) {
                    u[m * L + o] = g;
                } else {
                    if (valid && live) p.dst[at + l + L * m + E * o] = g;
                }
            });
        }
        if constexpr (RESID) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                acc0 += __shfl_xor_sync(0xffffffffu, acc0, o);
                acc1 += __shfl_xor_sync(0xffffffffu, acc1, o);
            }
            if ((threadIdx.x & 31) == 0) {
                atomicAdd(p.resid, acc0);
                atomicAdd(p.resid + 1, acc1);
            }
        }
    }
    if constexpr (BACK) {
        float2 y[E];
        {
            float2 v[M * L];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int t = M * L == E ? l + L * m : min(l + L * m, E - 1);
                float2 q[L];
                level1<L, !INV1>(q, [&](int i) { return u[m * L + i]; });
                level2<L, !INV1>(q, [&](int o, float2 x) { v[m * L + o] = stage_twiddle<!INV1>(p.tw, mirror_offset(N), o, E, t, x); });
            }
            mirror_exchange<N>(v, y, ex, l, sync);
        }
        float2 *stage = reinterpret_cast<float2 *>(ph_smem);
        {
            float2 w[E];
            level1<E, !INV1>(w, [&](int i) { return y[i]; });
            level2<E, !INV1>(w, [&](int o, float2 x) { stage[r * C::PITCH + l + L * o] = x; });
        }
        __syncthreads();
        const int rows = min(C::RB, p.nrows - row0);
        for (int i = threadIdx.x; i < N * C::RB; i += C::THREADS) {
            const int q = i % C::RB, k = i / C::RB;
            if (q < rows) p.dst[(size_t)k * p.nrows + row0 + q] = stage[q * C::PITCH + k];
        }
    }
}

template <int N, int MODE, bool RESID = false>
cudaError_t launch_gs(const GsParams &p, cudaStream_t s) {
    using C = PassG<N>;
    static_assert((C::SMEM + 1024) * C::CTAS <= 228 * 1024, "the CTAs of an SM share its shared memory");
    auto kern = k_two_gs<N, MODE, RESID>;
    if constexpr (C::SMEM > 48 * 1024) {   // per-device opt-in to more than 48 KB of dynamic shared memory
        static unsigned long long done_mask = 0;
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(__atomic_load_n(&done_mask, __ATOMIC_ACQUIRE) & bit)) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
            if (e != cudaSuccess) return e;
            __atomic_fetch_or(&done_mask, bit, __ATOMIC_ACQ_REL);
        }
    }
    const int gx = (p.nrows + C::RB - 1) / C::RB;
    if (gx == 0) return cudaSuccess;
    return launch_dependent(kern, dim3(gx), C::THREADS, C::SMEM, s, p);
}

}  // namespace two
}  // namespace ph
