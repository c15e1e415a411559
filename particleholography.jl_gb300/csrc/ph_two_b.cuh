// ph_two_b.cuh -- reconstruction pass B on the two-stage row transform.
#pragma once

#include "ph_launch.cuh"
#include "ph_two.cuh"

namespace ph {
namespace two {

// Rows y of T, inverse FFT along kx and the epilogue of ReconB.  A CTA is four
// warps; a row belongs to one warp (two rows per warp at 128 .. 512, two
// warps per row from 1536), so no barrier spans more than its threads.
// The row of slice b + 1 arrives by bulk copy as soon as slice b's has been
// read into registers.  The running minima and their slices live in tensor
// memory, 2 E columns of the thread's own lane: in registers they would not fit
// beside the transform's 2 E values, and shared memory bounds the pass.
//
// 2048 = 2 x 1024 (and 1536 = 2 x 768): one warp transforms x[n] + x[n + 1024] (the even outputs),
// the other (x[n] - x[n + 1024]) W^n (the odd ones).  Each row is read twice (8
// bytes per voxel more), but 32 values per thread leave room for 16 warps per
// SM: 3.19 ms per 2048^2 x 512 launch, against 3.64 ms with 64 values per
// thread and 8 warps (latency: 54 % of issue slots), and 3.86 ms in the
// three-stage row engine.  1024^2 x 256: 0.365 ms (0.483 in the engine; the
// copy peak would take 0.316).  4096^2 x 128, 64 values: 3.82 ms (4.37).
// 3 * 2^a: 768^2 x 256 0.247 ms (0.357), 1536^2 x 256 1.01 ms (1.35).
// Measured slower: the stage factors read from the W^i table (gathers of up to
// 32 lines: 3.77 ms at 2048) or held in registers across slices (spills).
// SLICE: the slice of every minimum is kept and merged with it (64-bit words);
// without it the minima alone go to proj32 as float bits: half the tensor memory,
// and neither an unpacking kernel nor a 64-bit word per pixel.
template <int N, int EPI, bool GROUPED, bool SLICE = true>
struct PassB {
    static constexpr int H = halves(N);                      // transforms a row is split into
    using PL = Plan<N / H>;
    static constexpr int THREADS = 128;
    static constexpr int TPR = H * PL::L;                    // threads per row
    static constexpr int ROWS = THREADS / TPR;
    static constexpr int CTAS = PL::E >= 48 ? 2 : 4;         // per SM: 255 registers at 48 and 64 values, 128 below
    static constexpr int CC = PL::M * PL::L;                 // outputs per thread (with the idle ones)
    static constexpr bool MIN = EPI == EPI_PROJ || EPI == EPI_VOL;
    static constexpr uint32_t COLS = SLICE || CC < 32 ? 2 * CC : CC;   // minima, then slices
    static constexpr size_t IN = (size_t)N * 8;
    static constexpr size_t XB = (size_t)PL::XWORDS * 4;
    using F = Factors<N / H, true, H>;
    static constexpr size_t SMEM = ROWS * (IN + H * XB) + F::BYTES + ROWS * 8 + 16;
};

template <int N, int EPI, bool GROUPED, bool SLICE>
__global__ void __launch_bounds__(128, PassB<N, EPI, GROUPED, SLICE>::CTAS) k_two_b(const ReconB<EPI, GROUPED> p) {
    using C = PassB<N, EPI, GROUPED, SLICE>;
    using PL = typename C::PL;
    constexpr int E = PL::E, L = PL::L, H = C::H, ROWS = C::ROWS;
    extern __shared__ __align__(128) unsigned char ph_smem[];
    float2 *tab = reinterpret_cast<float2 *>(ph_smem + ROWS * (C::IN + H * C::XB));
    uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(tab) + C::F::BYTES);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bars + ROWS);

    int group = p.group, b1max = p.nbatch;
    const float2 *t = p.t;
    unsigned long long *proj64 = p.proj64;
    if constexpr (GROUPED) {
        const int z = (int)blockIdx.z;
        group = p.item_group(z);
        b1max = p.item_nb(z);
        t += (size_t)z * p.item_t_stride;
        proj64 += (size_t)z * p.p64_stride;
    }
    const int b0 = blockIdx.y * group, b1 = min(b0 + group, b1max);
    if (b0 >= b1) return;

    const int warp = threadIdx.x >> 5;
    const int r = threadIdx.x / C::TPR, h = threadIdx.x / L % H, l = threadIdx.x % L;
    const int y = blockIdx.x * ROWS + r;
    const bool valid = y < p.rows;
    const bool track = EPI == EPI_PROJ || (EPI == EPI_VOL && p.proj32 != nullptr);   // (volumes without SLICE only)
    if constexpr (C::MIN) {
        if (warp == 0) tc::tmem_alloc(slot, C::COLS);
    }
    C::F::fill(tab, p.tw);
    if (threadIdx.x < ROWS) mbar_init(bars + threadIdx.x, 1);
    if (threadIdx.x == 0) mbar_fence_init();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    grid_dependency_wait();   // T is written
    const uint32_t tm = C::MIN ? *slot + ((uint32_t)(warp & 3) << 21) : 0;

    // a warp whose rows all lie beyond the last row has nothing to do (rows are
    // whole warps, or two per warp: the guard is uniform over a row's threads)
    const int first = blockIdx.x * ROWS + (C::TPR >= 32 ? r : 2 * warp);
    if (first < p.rows) {
        float2 *in = reinterpret_cast<float2 *>(ph_smem + r * C::IN);
        float *ex = reinterpret_cast<float *>(ph_smem + ROWS * C::IN + (r * H + h) * C::XB);
        const auto sync = [&] {
            if constexpr (L <= 32) __syncwarp();
            else named_bar_sync(1 + r, L);
        };
        const auto sync_row = [&] {
            if constexpr (C::TPR <= 32) __syncwarp();
            else named_bar_sync(1 + r, C::TPR);
        };
        const uint64_t policy = l2_evict_first();   // T is read once
        const auto issue = [&](int b) {   // one thread per row: the row of slice b
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(bars + r, N * 8);
            bulk_g2s(in, t + ((size_t)b * p.rows + y) * N, N * 8, bars + r, policy);
        };
        if (l == 0 && h == 0 && valid) issue(b0);
        if constexpr (C::MIN) {
            float inf[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) inf[i] = __int_as_float(0x7f800000);
            float zero[16] = {};
#pragma unroll
            for (int c = 0; c < C::CC; c += 16) {
                tmem_st16(tm + c, inf);
                if constexpr (SLICE) tmem_st16(tm + C::CC + c, zero);
            }
            tmem_wait_st();
        }
        uint32_t parity = 0;
        for (int b = b0; b < b1; ++b) {
            const int k = p.k0 + b;
            if (valid) mbar_wait(bars + r, parity, p.err);
            if constexpr (L < 32) __syncwarp();
            parity ^= 1u;
            float2 z[C::CC];
            {
                float2 v[E], w[E];
                if constexpr (H == 1) {
                    level1<E, true>(w, [&](int i) { return in[l + L * i]; });
                } else {
                    // x[n] + x[n + N/2] (even outputs) or (x[n] - x[n + N/2]) W_N^n (odd outputs), n = l + L i:
                    // here the constant part of the twiddle, W_(N/L)^i; the lane's is in f.a
                    const float sign = h == 0 ? 1.0f : -1.0f;
                    level1<E, true>(
                        w, [&](int i) { return fma2s(sign, in[l + L * i + N / 2], in[l + L * i]); },
                        [&](auto N2, auto &t) {
                            if (h != 0) {
                                static_for<PL::P>([&](auto N1) {
                                    constexpr int i = PL::Q * decltype(N1)::value + decltype(N2)::value;
                                    t[decltype(N1)::value] = ctw<i, N / L, true>(t[decltype(N1)::value]);
                                });
                            }
                        });
                }
                typename C::F f;   // re-read every slice: in registers throughout they would spill
                f.load(opaque(tab), l, h);
                sync_row();   // the row is in registers (and the exchange region free): refill it
                if (l == 0 && h == 0 && valid && b + 1 < b1) issue(b + 1);
                level2<E, true>(w, [&](int o, float2 x) { v[o] = f.apply(o, x); });
                exchange<N / H>(v, z, ex, l, sync);
            }
#pragma unroll
            for (int m = 0; m < PL::M; ++m) {
                float2 w[L], u[L];
                level1<L, true>(w, [&](int i) { return z[m * L + i]; });
                level2<L, true>(w, [&](int o, float2 x) { u[o] = x; });
                const bool live = PL::M * L == E || l + L * m < E;   // not an idle thread's
                // output o is column x = H (l + L m + E o) + h
                if constexpr (C::MIN) {
#pragma unroll
                    for (int c = 0; c < L; c += 16) {
                        float i2[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 q = u[c + i];
                            i2[i] = fmaf(q.x, q.x, q.y * q.y);
                        }
                        if constexpr (EPI == EPI_VOL) {
                            // the type is chosen once per 16 values
                            const size_t row = (size_t)k * p.vol_slice_stride + (size_t)y * N + H * (l + L * m + E * c) + h;
                            const auto store16 = [&](auto *vol, auto &&convert) {
                                auto *out = vol + row;
#pragma unroll
                                for (int i = 0; i < 16; ++i) {
                                    i2[i] = clamp01(i2[i]);
                                    const auto q = convert(i2[i]);
                                    if (valid && live) out[H * E * i] = q;
                                }
                            };
                            if (p.vol_dtype == 3) {
                                store16(reinterpret_cast<double *>(p.vol), [](float v) { return (double)v; });
                            } else if (p.vol_dtype == 5) {   // binary volume: the clamped Float32 intensity <= threshold
                                const float thr = p.threshold;
                                store16(reinterpret_cast<uint8_t *>(p.vol), [thr](float v) { return (uint8_t)(v <= thr ? 1 : 0); });
                            } else {
                                store16(reinterpret_cast<float *>(p.vol), [](float v) { return v; });
                            }
                        }
                        if (track) {
                            float mv[16], mk[16];
                            tmem_ld16(tm + m * L + c, mv);
                            if constexpr (SLICE) tmem_ld16(tm + C::CC + m * L + c, mk);
                            tmem_wait(mv);
                            if constexpr (SLICE) tmem_wait(mk);
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                if (i2[i] < mv[i]) {
                                    mv[i] = i2[i];
                                    if constexpr (SLICE) mk[i] = __int_as_float(k);
                                }
                            }
                            tmem_st16(tm + m * L + c, mv);
                            if constexpr (SLICE) tmem_st16(tm + C::CC + m * L + c, mk);
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < L; ++i) {
                        const int x = H * (l + L * m + E * i) + h;
                        if (valid && live)
                            reinterpret_cast<float2 *>(p.vol)[(size_t)k * p.vol_slice_stride + (size_t)y * N + x] = u[i];
                    }
                }
            }
            if constexpr (C::MIN) tmem_wait_st();
        }
        if constexpr (C::MIN) {
            if (track) {
#pragma unroll
                for (int c = 0; c < C::CC; c += 16) {
                    float mv[16], mk[16];
                    tmem_ld16(tm + c, mv);
                    if constexpr (SLICE) tmem_ld16(tm + C::CC + c, mk);
                    tmem_wait(mv);
                    if constexpr (SLICE) tmem_wait(mk);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int m = (c + i) / L, o = (c + i) % L;
                        const int xo = H * (l + L * m + E * o) + h;
                        if (valid && (PL::M * L == E || l + L * m < E)) {
                            const size_t at = (size_t)y * N + xo;
                            if constexpr (SLICE) atomicMin(proj64 + at, pack_min(mv[i], __float_as_int(mk[i])));
                            else atomicMin(p.proj32 + at, __float_as_uint(mv[i]));   // (non-negative: ordered as bits)
                        }
                    }
                }
            }
        }
    }
    if constexpr (C::MIN) {
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (warp == 0) tc::tmem_dealloc(*slot, C::COLS);
    }
}

template <int N, int EPI, bool GROUPED, bool SLICE>
cudaError_t launch_b_form(const ReconB<EPI, GROUPED> &p, int groups, int items, cudaStream_t s) {
    using C = PassB<N, EPI, GROUPED, SLICE>;
    static_assert((C::SMEM + 1024) * C::CTAS <= 228 * 1024, "the CTAs of an SM share its shared memory");
    auto kern = k_two_b<N, EPI, GROUPED, SLICE>;
    static unsigned long long done_mask = 0;   // per-device opt-in to more than 48 KB of dynamic shared memory
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&done_mask, __ATOMIC_ACQUIRE) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        __atomic_fetch_or(&done_mask, bit, __ATOMIC_ACQ_REL);
    }
    const int gx = (p.rows + C::ROWS - 1) / C::ROWS;
    if (gx == 0 || groups == 0) return cudaSuccess;
    return launch_dependent(kern, dim3(gx, groups, items), C::THREADS, C::SMEM, s, p);
}

template <int N, int EPI, bool GROUPED>
cudaError_t launch_b(const ReconB<EPI, GROUPED> &p, int groups, int items, cudaStream_t s) {
    if constexpr (EPI == EPI_PROJ && !GROUPED)
        if (p.proj32 == nullptr) return launch_b_form<N, EPI, GROUPED, true>(p, groups, items, s);
    if constexpr (GROUPED) return launch_b_form<N, EPI, GROUPED, true>(p, groups, items, s);
    else return launch_b_form<N, EPI, GROUPED, false>(p, groups, items, s);
}

}  // namespace two
}  // namespace ph
