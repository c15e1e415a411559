// ph_two_f.cuh -- the forward passes of a reconstruction (rows, then spectrum
// columns) on the two-stage row transform.
//
// Both are bound by latency at small frames and by memory at large ones.  The
// forward rows take 4 rows per CTA: at 256^2 that is 64 CTAs, where the 512-thread
// CTAs of the row engine were 8 (7.5 us, now 2.1).  Their outputs pass through
// shared-memory rows (pitch N + 4 elements: writes along a row and reads across
// the 4 rows are both free of bank conflicts), so that the transposed store
// writes 32-byte sectors.
//
// The spectrum is the column transform, in place, and an elementwise kernel that
// forms the state.  In one kernel the phase rates (two arctangents and a logarithm
// per value, ~200 instructions) ran on the few warps that a transform's registers
// leave: 19 us of a 53 us call at 256^2, 45 us at 768^2, 68 us at 2048^2 with the
// transfers staged by tensor maps; now 6.7, 11.5 and 49 us.
#pragma once

#include "ph_launch.cuh"
#include "ph_two.cuh"

namespace ph {
namespace two {

template <int N>
struct PassF {
    using PL = Plan<N>;
    static constexpr int RB = 4;
    static constexpr int THREADS = RB * PL::L;
    static constexpr int PITCH = N + 4;                      // elements between staged rows
    static constexpr size_t STAGE = (size_t)RB * PITCH * 8;
    static constexpr size_t XB = (size_t)PL::XWORDS * 4;
    static constexpr size_t SMEM = STAGE + RB * XB;
    static constexpr int CTAS = PL::E >= 48 ? 256 / THREADS : 512 / THREADS;
};

// The transform of a thread's row: load(i) gives x[l + L i], store(k, v) takes output
// k.  ex: the row's exchange region; r: its number within the CTA.
template <int N, bool INV, class Load, class Store>
__device__ __forceinline__ void transform(const float2 *__restrict__ tw, float *ex, int r, int l, Load &&load,
                                          Store &&store) {
    using PL = Plan<N>;
    constexpr int E = PL::E, L = PL::L;
    const auto sync = [&] {
        if constexpr (L <= 32) __syncwarp();
        else named_bar_sync(1 + r, L);
    };
    float2 z[PL::M * L];
    {
        float2 v[E], w[E];
        level1<E, INV>(w, load);
        level2<E, INV>(w, [&](int o, float2 x) { v[o] = stage_twiddle<INV>(tw, twiddle_offset(N), o, L, l, x); });
        exchange<N>(v, z, ex, l, sync);
    }
#pragma unroll
    for (int m = 0; m < PL::M; ++m) {
        float2 w[L];
        level1<L, INV>(w, [&](int i) { return z[m * L + i]; });
        const bool live = PL::M * L == E || l + L * m < E;
        level2<L, INV>(w, [&](int o, float2 x) {
            if (live) store(l + L * m + E * o, x);
        });
    }
}

template <int N, int MODE>
__global__ void __launch_bounds__(PassF<N>::THREADS, PassF<N>::CTAS) k_two_fwd(const FwdRowsT<MODE> p) {
    static_assert(MODE == FWD_COMPLEX || MODE == FWD_SQRT_REAL, "padded frames run the row engine");
    using C = PassF<N>;
    using PL = Plan<N>;
    extern __shared__ __align__(128) unsigned char ph_smem[];
    grid_dependents_launch();
    const int z = blockIdx.z;
    const float2 *src = p.nitems > 1 ? p.src_items[z] : p.src;
    const float *src_real = p.nitems > 1 ? p.src_real_items[z] : p.src_real;
    float2 *dst = p.dst + (size_t)z * p.dst_stride;
    const int y0 = blockIdx.x * C::RB, r = threadIdx.x / PL::L, l = threadIdx.x % PL::L;
    const int y = min(y0 + r, p.nrows - 1);   // (rows beyond the last: its values again, not stored)
    float2 *stage = reinterpret_cast<float2 *>(ph_smem);
    float *ex = reinterpret_cast<float *>(ph_smem + C::STAGE + r * C::XB);
    // (the square root's rare path is a branch: with each load beside its root, 32
    // loads ran one after the other)
    float real[MODE == FWD_SQRT_REAL ? PL::E : 1];
    if constexpr (MODE == FWD_SQRT_REAL) {
#pragma unroll
        for (int i = 0; i < PL::E; ++i) real[i] = __ldg(src_real + (size_t)y * N + l + PL::L * i);
    }
    const auto load = [&](int i) -> float2 {
        if constexpr (MODE == FWD_COMPLEX) return src[(size_t)y * N + l + PL::L * i];
        else return make_float2(sqrtf(real[i]), 0.f);
    };
    transform<N, false>(p.tw, ex, r, l, load, [&](int k, float2 v) { stage[r * C::PITCH + k] = v; });
    __syncthreads();
    const int rows = min(C::RB, p.nrows - y0);
    for (int i = threadIdx.x; i < N * C::RB; i += C::THREADS) {
        const int q = i % C::RB, kx = i / C::RB;
        if (q < rows) dst[(size_t)kx * p.nrows + y0 + q] = stage[q * C::PITCH + kx];
    }
}

// Rows kx of a1 [nx][ny = N], forward FFT along ky, in place (a row's threads have
// read it all before the first of them writes).
template <int N>
__global__ void __launch_bounds__(PassF<N>::THREADS, PassF<N>::CTAS) k_two_cols(const SpectrumCols p) {
    using PL = Plan<N>;
    extern __shared__ __align__(128) unsigned char ph_smem[];
    grid_dependents_launch();
    grid_dependency_wait();
    const int r = threadIdx.x / PL::L, l = threadIdx.x % PL::L;
    const int kx = blockIdx.x * PassF<N>::RB + r;
    const bool valid = kx < p.nx;
    float2 *row = const_cast<float2 *>(p.a1) + (size_t)blockIdx.z * p.a1_stride + (size_t)min(kx, p.nx - 1) * N;
    float *ex = reinterpret_cast<float *>(ph_smem + r * PassF<N>::XB);
    transform<N, false>(
        p.tw, ex, r, l, [&](int i) { return row[l + PL::L * i]; },
        [&](int k, float2 v) {
            if (valid) row[k] = v;
        });
}

// DEPENDENT: as a programmatic dependent (k_two_cols waits for the forward rows).
template <int N, bool DEPENDENT, class Kernel, class Params>
cudaError_t launch_f(Kernel kern, size_t smem, const Params &p, int nrows, int items, cudaStream_t s) {
    using C = PassF<N>;
    static_assert((C::SMEM + 1024) * C::CTAS <= 228 * 1024, "the CTAs of an SM share its shared memory");
    if (smem > 48 * 1024) {   // per-device opt-in to more than 48 KB of dynamic shared memory
        static unsigned long long done_mask = 0;
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(__atomic_load_n(&done_mask, __ATOMIC_ACQUIRE) & bit)) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            __atomic_fetch_or(&done_mask, bit, __ATOMIC_ACQ_REL);
        }
    }
    const int gx = (nrows + C::RB - 1) / C::RB;
    if (gx == 0) return cudaSuccess;
    if constexpr (DEPENDENT) return launch_dependent(kern, dim3(gx, 1, items), C::THREADS, smem, s, p);
    kern<<<dim3(gx, 1, items), C::THREADS, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace two
}  // namespace ph
