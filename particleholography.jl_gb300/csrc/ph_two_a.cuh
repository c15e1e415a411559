// ph_two_a.cuh -- reconstruction pass A on the two-stage row transform.
#pragma once


#include "ph_launch.cuh"
#include "ph_two.cuh"

namespace ph {
namespace two {

// X_k = X_0 Hdz^k, inverse FFT along ky, transposed tensor-map store of T.  A CTA
// holds the RB rows kx of one box; a row belongs to one warp (two rows per warp
// at 128 .. 512, two warps per row at 3072 and 4096), so that the exchange needs no CTA
// barrier.  X_k and Hdz of a thread's values live in tensor memory (4 E columns
// of its own lane): every slice reads both and writes back X_{k+1} = X_k Hdz.  X
// is formed anew from the spectrum state at every multiple of `chain` slices.
//
// Precision: a projection is as near to the 64-bit one as with every slice formed
// directly by the row engine (relative errors at 12 random distances, there and here:
// 256^2 3.5e-7 and 3.2e-7, 1024^2 3.9e-7 and 3.7e-7, 2048 x 1536 3.7e-7 and 3.7e-7; the
// engine's chains at 2048^2 8.4e-7, here 4.0e-7).  For that Hdz has to be right to well
// below a rounding, since its error adds up along the chain, and that of the zero
// frequency shows in every pixel (with Hdz from sincospif and exp2f: 4.3e-7 at 1024^2,
// 4.5e-7 at 2048 x 1536); and X from the polynomials of `rotated` rather than __sincosf,
// which is good to 1e-7 only.  A chain is as long as that leaves room for: at 256^2 x 32
// 27 us with 4 and 29 with 8 (small groups walk to their start), at 4096 x 256 x 48 296
// and 285, at 512^2 x 64 87 and 83; at 1024^2 x 256 863 with 8 and 842 with 16; at
// 2048 x 1536 x 157 16 gives 4.0e-7.
//
// In the row engine this pass moved 87 bytes per voxel through the shared-memory
// data path (chain 24, two exchanges 32, staging 16, twiddles 15); here 32 to 40.
// Per launch, before and now: 1024^2 x 256 0.68 and 0.47 ms, 2048^2 x 512 5.43
// and 4.55 ms, 4096^2 x 128 9.3 and 5.15 ms (no more clusters).  What is left:
// arithmetic and its latency (50 % of the FP32 pipe, 45 to 54 % of issue slots),
// then the stores: without them 0.46 ms at 1024.
//
// Boxes of 8 kx (64 bytes): of 4 kx at 1024, 0.77 ms (32-byte pieces of lines
// that other CTAs complete); of 16 kx, 0.60 ms (one CTA per SM).  4096 keeps 4:
// a box's rows have to fit the CTA.  The stores evict T first, since the next
// pass reads it long after: 0.56 -> 0.49 ms at 1024, 2.29 -> 2.21 ms at 2048^2 x
// 256.  Measured slower at 2048: 2 x 1024 with 32 values per thread (2.57 ms);
// two groups of tensor-memory columns per wait.
//
// 3 * 2^a lengths (12, 24 or 48 values per thread; a quarter of the threads idle
// in stage 2), per launch in the row engine and here: 384^2 x 512 0.83 and 0.16 ms,
// 768^2 x 256 1.13 and 0.33 ms, 1536^2 x 256 3.25 and 1.48 ms, 3072^2 x 64 3.49 and
// 1.74 ms (the engine has no tensor-map store there and reads the phase rates from
// L2 for every slice).

// y per box: the largest of 256, 128, 64 that divides the length.
__host__ __device__ constexpr int box_y(int n) { return n % 256 == 0 ? 256 : n % 128 == 0 ? 128 : 64; }

template <int N>
struct PassA {
    using PL = Plan<N>;
    using F = Factors<N, true>;
    static constexpr int RB = N <= 2048 ? 8 : 4;             // rows kx per CTA: one box
    static constexpr int THREADS = RB * PL::L;
    static constexpr int CTAS = (PL::E >= 48 ? 256 : 512) / THREADS;
    static constexpr uint32_t WCOLS = 4 * PL::E;             // tensor-memory columns of a warp
    // (an allocation is a power of two)
    static constexpr uint32_t COLS = 1u << ilog2c(2 * (int)(WCOLS * (THREADS / 128)) - 1);
    static constexpr size_t STAGE = (size_t)RB * N * 8;
    static constexpr size_t XB = (size_t)PL::XWORDS * 4;
    static constexpr size_t SMEM = STAGE + RB * XB + F::BYTES + 24;
    static constexpr int BOX_Y = box_y(N);
    // slices between two formations of X
    __host__ __device__ static constexpr uint32_t chain(int nx) {
        return N <= 256 ? (nx < 4096 ? 4 : 8) : N == 1024 || PL::E == 64 ? 16 : 8;
    }
};

// Byte offset of (y, row r) in the staging [y][RB], with the tensor map's
// swizzle (16-byte chunks exchanged by the address bits above 128 bytes): lanes
// of consecutive y are RB x 8 bytes apart, and would meet in few banks.  The
// exchange has a period of 512 (256) bytes, so a multiple of that may be added after.
template <int RB>
__device__ __forceinline__ uint32_t stage_offset(int y, int r) {
    const uint32_t a = (uint32_t)(y * RB + r) * 8;
    return a ^ ((a >> 3) & (RB == 8 ? 0x30u : 0x10u));
}

// exp(2 pi i turns / 2^32) 2^w, off by at most 1e-8 before its one rounding where the
// modulus is near one, so that a stored Float32 factor comes out as it was.  `angle`: lane
// i's entry of the 32 angles 2 pi i / 32, (cos hi, cos lo, sin hi, sin lo); the whole warp calls.
__device__ __forceinline__ float2 unit_power(uint32_t turns, float w, const float4 angle) {
    const uint32_t i = (turns + (1u << 26)) >> 27;                 // the nearest of them
    const float x = (float)(int32_t)(turns - (i << 27)) * 1.46291807926715968e-9f, x2 = x * x;   // 2 pi / 2^32
    const float ch = __shfl_sync(0xffffffffu, angle.x, i & 31), cl = __shfl_sync(0xffffffffu, angle.y, i & 31);
    const float sh = __shfl_sync(0xffffffffu, angle.z, i & 31), sl = __shfl_sync(0xffffffffu, angle.w, i & 31);
    const float sn = fmaf(x * x2, fmaf(x2, 1.0f / 120.0f, -1.0f / 6.0f), x);
    const float cs1 = x2 * fmaf(x2, fmaf(x2, -1.0f / 720.0f, 1.0f / 24.0f), -0.5f);   // cos - 1
    float c1 = cl + fmaf(ch, cs1, -sh * sn), s1 = sl + fmaf(sh, cs1, ch * sn);
    if (fabsf(w) < 0x1p-14f) {   // the modulus minus one, whose rounding is not that of a value near one
        const float m1 = w * 0.69314718055994530942f;   // (its square is below 2e-9)
        c1 = fmaf(ch + c1, m1, c1);
        s1 = fmaf(sh + s1, m1, s1);
        return make_float2(ch + c1, sh + s1);
    }
    const float mag = exp2f(w);
    return make_float2((ch + c1) * mag, (sh + s1) * mag);
}

// x0 exp(2 pi i turns / 2^32) 2^w: the nearest quarter turn, and Taylor polynomials of the
// rest (at most pi / 4; truncated below 4e-9).
__device__ __forceinline__ float2 rotated(float2 x0, uint32_t turns, float w) {
    const uint32_t q = (turns + (1u << 29)) >> 30;
    const float x = (float)(int32_t)(turns - (q << 30)) * 1.46291807926715968e-9f, x2 = x * x;   // 2 pi / 2^32
    const float sn = fmaf(x * x2, fmaf(x2, fmaf(x2, fmaf(x2, 1.0f / 362880.0f, -1.0f / 5040.0f), 1.0f / 120.0f), -1.0f / 6.0f), x);
    const float cs = fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 1.0f / 40320.0f, -1.0f / 720.0f), 1.0f / 24.0f), -0.5f), 1.0f);
    const float a = q & 1 ? sn : cs, b = q & 1 ? cs : sn, mag = exp2f(w);
    const float c = (q + 1) & 2 ? -a : a, s = q & 2 ? -b : b;
    return cmul(x0, make_float2(c * mag, s * mag));
}

template <int N, bool GROUPED>
__global__ void __launch_bounds__(PassA<N>::THREADS, PassA<N>::CTAS)
    k_two_a(const ReconAT<GROUPED> p, const __grid_constant__ CUtensorMap tmap) {
    using C = PassA<N>;
    using PL = typename C::PL;
    constexpr int E = PL::E, L = PL::L, RB = C::RB, P = PL::P, Q = PL::Q;
    extern __shared__ __align__(1024) unsigned char ph_smem[];
    unsigned char *stage = ph_smem;
    float2 *tab = reinterpret_cast<float2 *>(ph_smem + C::STAGE + RB * C::XB);
    uint64_t *bar = reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(tab) + C::F::BYTES);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bar + 1);

    // Launch order: two slice groups at a time, the groups of one row block
    // consecutive, so that they share its state rows in L2 and neighbouring row
    // blocks write the neighbouring pieces of T's rows together (2048^2 x 512: 4.55
    // ms; all 8 groups at a time 4.77, one 4.73).
    constexpr int AT_ONCE = 2;
    const int lin = blockIdx.y * gridDim.x + blockIdx.x;
    const int chunk = lin / (AT_ONCE * (int)gridDim.x), at = lin % (AT_ONCE * (int)gridDim.x);
    const int wide = min(AT_ONCE, (int)gridDim.y - chunk * AT_ONCE);
    const int g = chunk * AT_ONCE + at % wide, kx0 = at / wide * RB;
    int group = p.group, b1max = p.nbatch;
    const float4 *state = p.state;
    if constexpr (GROUPED) {
        const int z = (int)blockIdx.z;
        group = p.item_group(z);
        b1max = p.item_nb(z);
        state += (size_t)z * p.item_state_stride;
    }
    const int b0 = g * group, b1 = min(b0 + group, b1max);
    if (b0 >= b1) return;

    const int warp = threadIdx.x >> 5;
    const int r = threadIdx.x / L, l = threadIdx.x % L;
    if (warp == 0) tc::tmem_alloc(slot, C::COLS);
    C::F::fill(tab, p.tw);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    grid_dependency_wait();   // the state is written, and T no longer read
    // columns of this warp; group n2 of the first butterflies: X of its P inputs, then Hdz of them
    const uint32_t tm = *slot + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * C::WCOLS;
    // (rows beyond nx transform row nx - 1 again; the tensor map drops their columns)
    const float4 *srow = state + (size_t)min(kx0 + r, p.nx - 1) * N;
    float *ex = reinterpret_cast<float *>(ph_smem + C::STAGE + r * C::XB);
    const auto sync = [&] {
        if constexpr (L <= 32) __syncwarp();
        else named_bar_sync(2 + r, L);
    };

    // a group's values (inputs i = Q n1 + n2) -> tensor-memory columns at `at`
    const auto put = [&](uint32_t at, const float2 (&t)[P]) {
        if constexpr (P == 4) {
            tmem_st8(at, t);
        } else {
            float q[16];
#pragma unroll
            for (int i = 0; i < 8; ++i) { q[2 * i] = t[i].x; q[2 * i + 1] = t[i].y; }
            tmem_st16(at, q);
        }
    };
    const uint64_t policy = l2_evict_first();   // T is read by the next pass, long after
    for (int b = b0; b < b1; ++b) {
        tmem_wait_st();
        const uint32_t k = (uint32_t)(p.k0 + b), ahead = k % C::chain(p.nx);
        const bool first = b == b0;
        if (first || ahead == 0) {
            // X at the last multiple of the chain, then the chain's own products: X_k does
            // not depend on where a group or a range of slices starts.  The first time
            // also Hdz.
            const float4 angle = __ldg(p.ptab + (threadIdx.x & 31) * (kPhaseTable / 32));
            float4 st[P];
            const auto read = [&](int n2) {
#pragma unroll
                for (int n1 = 0; n1 < P; ++n1) st[n1] = srow[l + L * (Q * n1 + n2)];
            };
            read(0);
#pragma unroll 1
            for (int n2 = 0; n2 < Q; ++n2) {
                float4 cur[P];
#pragma unroll
                for (int n1 = 0; n1 < P; ++n1) cur[n1] = st[n1];
                if (n2 + 1 < Q) read(n2 + 1);   // the next group's state is on its way
                float2 t[P];
                if (k == ahead) {   // (the first chain starts from X_0 as it is)
#pragma unroll
                    for (int n1 = 0; n1 < P; ++n1) t[n1] = make_float2(cur[n1].x, cur[n1].y);
                } else {
#pragma unroll
                    for (int n1 = 0; n1 < P; ++n1)
                        t[n1] = rotated(make_float2(cur[n1].x, cur[n1].y), (k - ahead) * __float_as_uint(cur[n1].z),
                                        (float)(k - ahead) * cur[n1].w);
                }
                if (first) {
                    float2 hd[P];
#pragma unroll
                    for (int n1 = 0; n1 < P; ++n1) hd[n1] = unit_power(__float_as_uint(cur[n1].z), cur[n1].w, angle);
                    put(tm + n2 * 4 * P + 2 * P, hd);
#pragma unroll 1
                    for (uint32_t i = 0; i < ahead; ++i)
#pragma unroll
                        for (int n1 = 0; n1 < P; ++n1) t[n1] = cmul2(t[n1], hd[n1]);
                }
                put(tm + n2 * 4 * P, t);
            }
            tmem_wait_st();
        }
        float2 z[PL::M * L];
        {
            float2 v[E], w[E];
            constexpr int V = P / 4;    // loads of 16 columns per group
            float x[2][V][16];          // X and Hdz of two groups: the next is on its way while one is used
            const auto fetch = [&](int n2) {
#pragma unroll
                for (int i = 0; i < V; ++i) tmem_ld16(tm + n2 * 4 * P + 16 * i, x[n2 & 1][i]);
            };
            fetch(0);
            static_for<Q>([&](auto N2) {
                constexpr int n2 = decltype(N2)::value, H0 = P == 4 ? 8 : 0;   // P = 8: Hdz in the second 16
                auto &xx = x[n2 & 1];
#pragma unroll
                for (int i = 0; i < V; ++i) tmem_wait(xx[i]);
                if constexpr (n2 + 1 < Q) fetch(n2 + 1);
                float2 t[P], next[P];
#pragma unroll
                for (int n1 = 0; n1 < P; ++n1) {
                    t[n1] = make_float2(xx[0][2 * n1], xx[0][2 * n1 + 1]);
                    next[n1] = cmul2(t[n1], make_float2(xx[V - 1][H0 + 2 * n1], xx[V - 1][H0 + 2 * n1 + 1]));
                }
                put(tm + n2 * 4 * P, next);
                bfly<P, true>(t);
                static_for<P>([&](auto K1) {
                    constexpr int k1 = decltype(K1)::value;
                    w[P * n2 + k1] = ctw<n2 * k1, E, true>(t[k1]);
                });
            });
            typename C::F f;
            f.load(opaque(tab), l);
            level2<E, true>(w, [&](int o, float2 y) { v[o] = f.apply(o, y); });
            sync();   // every thread has read the previous exchange
            exchange<N>(v, z, ex, l, sync);
        }
        float2 u[PL::M * L];   // u[m L + o] = value of y = l + L m + E o
#pragma unroll
        for (int m = 0; m < PL::M; ++m) {
            float2 w[L];
            level1<L, true>(w, [&](int i) { return z[m * L + i]; });
            level2<L, true>(w, [&](int o, float2 y) { u[m * L + o] = y; });
        }
        // the previous slice's boxes have left the staging
        if (threadIdx.x == 0) {
            bulk_wait_read_all();
            mbar_arrive(bar);
        }
        mbar_wait(bar, (uint32_t)(b - b0) & 1u, p.err);
        // where steps of L and E in y are whole periods of the swizzle, one offset serves all
        constexpr int PERIOD = RB == 8 ? 512 : 256;
        constexpr bool WHOLE = L * RB * 8 % PERIOD == 0 && E * RB * 8 % PERIOD == 0;
        unsigned char *out = stage + stage_offset<RB>(l, r);
#pragma unroll
        for (int m = 0; m < PL::M; ++m)
            if (PL::M * L == E || l + L * m < E) {
#pragma unroll
                for (int o = 0; o < L; ++o) {
                    const int dy = L * m + E * o;
                    *reinterpret_cast<float2 *>(WHOLE ? out + dy * RB * 8 : stage + stage_offset<RB>(l + dy, r)) =
                        u[m * L + o];
                }
            }
        fence_proxy_async_smem();
        if (warp == 0) {
            named_bar_sync(1, C::THREADS);
            if (threadIdx.x == 0) {
#pragma unroll 1
                for (int q = 0; q < N / C::BOX_Y; ++q) {
                    const unsigned char *box = stage + (size_t)q * C::BOX_Y * RB * 8;
                    if constexpr (GROUPED) tma_store_4d(&tmap, box, kx0, q * C::BOX_Y, b, (int)blockIdx.z, policy);
                    else tma_store_3d(&tmap, box, kx0, q * C::BOX_Y, b, policy);
                }
                bulk_commit();
            }
        } else {
            named_bar_arrive(1, C::THREADS);
        }
    }
    if (threadIdx.x == 0) bulk_wait_all();   // the shared memory outlives the last boxes' reads
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(*slot, C::COLS);
}

template <int N, bool GROUPED>
cudaError_t launch_a(const ReconAT<GROUPED> &p, const CUtensorMap &tm, int groups, int items, cudaStream_t s) {
    using C = PassA<N>;
    static_assert(C::SMEM + 1024 <= 228 * 1024 / C::CTAS, "the CTAs of an SM share its shared memory");
    static_assert(C::COLS * C::CTAS <= 512, "and its tensor memory");
    auto kern = k_two_a<N, GROUPED>;
    static unsigned long long done_mask = 0;   // per-device opt-in to more than 48 KB of dynamic shared memory
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&done_mask, __ATOMIC_ACQUIRE) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        __atomic_fetch_or(&done_mask, bit, __ATOMIC_ACQ_REL);
    }
    const int gx = (p.nx + C::RB - 1) / C::RB;
    if (gx == 0 || groups == 0) return cudaSuccess;
    return launch_dependent(kern, dim3(gx, groups, items), C::THREADS, C::SMEM, s, p, tm);
}

}  // namespace two
}  // namespace ph
