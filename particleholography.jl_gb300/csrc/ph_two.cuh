// ph_two.cuh -- the two-stage row transform: N = E x L with E values per thread
// and L threads per row, so that a row crosses shared memory once.
//
// What bounds the reconstruction passes is the shared-memory / L1 data path
// (128 bytes per clock and SM).  The three-stage engine of ph_fft.cuh moves
// 63 bytes per voxel through it in the row pass at 2048 (bulk copy 8, first
// read 8, two exchanges 32, table twiddles 15): 3.4 ms of the 3.9 ms that a
// 2048^2 x 512 launch took.  With 64 values per thread one exchange is left
// (16 bytes), and the stage twiddles are products of 14 factors that a thread
// holds in registers: 32 bytes per voxel.  The butterflies use packed FP32
// (two lanes per issue slot; the FP32 pipe itself is as fast with scalar
// code, so this buys issue slots only).
//
// Stage 1: thread l (0 .. L-1) transforms the E values x[l + L e] and
// multiplies output k1 by W_N^(l k1).  Exchange.  Stage 2: thread t holds, for
// m < E / L, the L values of k1 = t + L m and transforms them: output k2 is
// X[k1 + E k2].  The exchange moves the real parts, then the imaginary parts,
// through E rows of L words (pitch L + 4): single-word writes with lanes
// consecutive and 16-byte reads with lanes 4 words apart, both free of bank
// conflicts, and half the shared memory of a complex exchange.
#pragma once

#include "ph_passes.cuh"
#include "ph_tc.cuh"

namespace ph {
namespace two {

// ---------------------------------------------------------------- packed butterflies

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// a + s t, s real
__device__ __forceinline__ float2 fma2s(float s, float2 t, float2 a) { return __ffma2_rn(t, make_float2(s, s), a); }
// a + i b and a - i b (scalar: a packed add would need the halves of b exchanged first)
__device__ __forceinline__ float2 addi(float2 a, float2 b) { return make_float2(a.x - b.y, a.y + b.x); }
__device__ __forceinline__ float2 subi(float2 a, float2 b) { return make_float2(a.x + b.y, a.y - b.x); }
__device__ __forceinline__ float2 cmul2(float2 a, float2 b) {
    const float2 t = __fmul2_rn(a, make_float2(b.x, b.x));
    return make_float2(fmaf(-a.y, b.y, t.x), fmaf(a.x, b.y, t.y));
}
// v * W_R^K (W = exp(-2 pi i / R), conjugate when INV)
template <int K, int R, bool INV>
__device__ __forceinline__ float2 ctw(float2 v) {
    constexpr int k = ((K % R) + R) % R;
    if constexpr (k == 0 || (2 * k) % R == 0 || (4 * k) % R == 0) {
        return twiddle_const<K, R, INV>(v);
    } else {
        constexpr float c = Tw<K, R, INV>::c, s = Tw<K, R, INV>::s;
        const float2 t = __fmul2_rn(v, make_float2(c, c));
        return make_float2(fmaf(-s, v.y, t.x), fmaf(s, v.x, t.y));
    }
}

template <bool INV>
__device__ __forceinline__ void d4(float2 &a0, float2 &a1, float2 &a2, float2 &a3) {
    const float2 s02 = add2(a0, a2), d02 = sub2(a0, a2), s13 = add2(a1, a3), d13 = sub2(a1, a3);
    a0 = add2(s02, s13);
    a2 = sub2(s02, s13);
    a1 = INV ? addi(d02, d13) : subi(d02, d13);
    a3 = INV ? subi(d02, d13) : addi(d02, d13);
}

// Natural order in and out; the 45-degree rotations are folded into the last adds.
template <bool INV>
__device__ __forceinline__ void d8(float2 (&v)[8]) {
    constexpr float h = 0.70710678118654752440f;
    float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    d4<INV>(e0, e1, e2, e3);
    d4<INV>(o0, o1, o2, o3);
    v[0] = add2(e0, o0);
    v[4] = sub2(e0, o0);
    v[2] = INV ? addi(e2, o2) : subi(e2, o2);
    v[6] = INV ? subi(e2, o2) : addi(e2, o2);
    const float2 t1 = INV ? addi(o1, o1) : subi(o1, o1);   // sqrt(2) W_8 o1
    v[1] = fma2s(h, t1, e1);
    v[5] = fma2s(-h, t1, e1);
    const float2 t3 = INV ? subi(o3, o3) : addi(o3, o3);   // -sqrt(2) W_8^3 o3
    v[3] = fma2s(-h, t3, e3);
    v[7] = fma2s(h, t3, e3);
}

template <bool INV>
__device__ __forceinline__ void d3(float2 &a, float2 &b, float2 &c) {
    constexpr float h = 0.86602540378443864676f;   // sqrt(3) / 2
    const float2 s = add2(b, c), d = sub2(b, c), m = fma2s(-0.5f, s, a);
    a = add2(a, s);
    const float2 p = make_float2(fmaf(-h, d.y, m.x), fmaf(h, d.x, m.y));   // m + i h d
    const float2 q = make_float2(fmaf(h, d.y, m.x), fmaf(-h, d.x, m.y));   // m - i h d
    b = INV ? p : q;
    c = INV ? q : p;
}
template <bool INV>
__device__ __forceinline__ void d6(float2 (&v)[6]) {   // n = 3 n1 + n2, k = k1 + 2 k2
    float2 e0 = add2(v[0], v[3]), e1 = add2(v[1], v[4]), e2 = add2(v[2], v[5]);
    float2 o0 = sub2(v[0], v[3]), o1 = ctw<1, 6, INV>(sub2(v[1], v[4])), o2 = ctw<2, 6, INV>(sub2(v[2], v[5]));
    d3<INV>(e0, e1, e2);
    d3<INV>(o0, o1, o2);
    v[0] = e0; v[2] = e1; v[4] = e2;
    v[1] = o0; v[3] = o1; v[5] = o2;
}

template <int R, bool INV>
__device__ __forceinline__ void bfly(float2 (&v)[R]) {
    static_assert(R == 2 || R == 3 || R == 4 || R == 6 || R == 8, "a butterfly of this size");
    if constexpr (R == 2) {
        const float2 t = v[0];
        v[0] = add2(t, v[1]);
        v[1] = sub2(t, v[1]);
    } else if constexpr (R == 3) d3<INV>(v[0], v[1], v[2]);
    else if constexpr (R == 4) d4<INV>(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 6) d6<INV>(v);
    else d8<INV>(v);
}

// R = P Q: n = Q n1 + n2, k = k1 + P k2.
__host__ __device__ constexpr int split_p_of(int r) { return r == 64 || r % 24 == 0 ? 8 : 4; }
template <int R>
constexpr int split_p() { return split_p_of(R); }
template <int R>
constexpr int split_q() { return R / split_p<R>(); }

// The first level of a length-R transform: v[Q n1 + n2] -> y[P n2 + k1], internal twiddles applied.
// load(i) gives input i; prologue(n2, t) may change the inputs t[n1] = x[Q n1 + n2] of one butterfly.
template <int R, bool INV, class Load, class Prologue>
__device__ __forceinline__ void level1(float2 (&y)[R], Load &&load, Prologue &&prologue) {
    constexpr int P = split_p<R>(), Q = split_q<R>();
    static_for<Q>([&](auto N2) {
        constexpr int n2 = decltype(N2)::value;
        float2 t[P];
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) t[n1] = load(Q * n1 + n2);
        prologue(N2, t);
        bfly<P, INV>(t);
        static_for<P>([&](auto K1) {
            constexpr int k1 = decltype(K1)::value;
            y[P * n2 + k1] = ctw<n2 * k1, R, INV>(t[k1]);
        });
    });
}
template <int R, bool INV, class Load>
__device__ __forceinline__ void level1(float2 (&y)[R], Load &&load) {
    level1<R, INV>(y, load, [](auto, auto &) {});
}
// The second level: y -> natural-order outputs, handed to out(k, v) for k = k1 + P k2.
template <int R, bool INV, class Out>
__device__ __forceinline__ void level2(const float2 (&y)[R], Out &&out) {
    constexpr int P = split_p<R>(), Q = split_q<R>();
    static_for<P>([&](auto K1) {
        constexpr int k1 = decltype(K1)::value;
        float2 t[Q];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) t[n2] = y[P * n2 + k1];
        bfly<Q, INV>(t);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) out(k1 + P * k2, t[k2]);
    });
}

// ---------------------------------------------------------------- shape

// The lengths that have a two-stage transform.
#define PH_FOR_EACH_N_TWO(X) X(128) X(192) X(256) X(384) X(512) X(768) X(1024) X(1536) X(2048) X(3072) X(4096)

// Values per thread, threads per row, and transforms of length L per thread in
// stage 2.  At 128 and the 3 * 2^a lengths the last of these (all, where M = 1)
// has only the threads t < E - (M - 1) L: the others compute on the last one's
// values and drop them.
__host__ __device__ constexpr int values(int n) {
    return n % 3 == 0 ? (n <= 192 ? 12 : n <= 768 ? 24 : 48) : n <= 128 ? 8 : n <= 256 ? 16 : n <= 1024 ? 32 : 64;
}
__host__ __device__ constexpr bool supported(int n) {
    return n == 128 || n == 192 || n == 256 || n == 384 || n == 512 || n == 768 || n == 1024 || n == 1536 ||
           n == 2048 || n == 3072 || n == 4096;
}

// The lengths whose rows pass B transforms as two of half the length (ph_two_b.cuh).
__host__ __device__ constexpr int halves(int n) { return n == 2048 || n == 1536 ? 2 : 1; }

// A length's table in global memory holds, behind the row engine's (ph_fft.cuh),
//  - the stage factors of the transform, [factor][l]: W^(l p), p = 1 .. P - 1, then
//    W^(l P q), q = 1 .. Q - 1;
//  - the stage twiddles themselves, W^(l k1) as [k1][l], and those of its mirror
//    (below), W^(t' q1) as [q1][t'];
//  - where halves(n) = 2, the factors of the two transforms of length n / 2,
//    [factor][h][l]: W^(l (2 p + h)), p = 0 .. P - 1, then W^(2 l P q).
// All of them but the W^(l P q) carry a gain: the constants of the butterflies round to
// moduli below one on average (1 / sqrt(2) by 1.7e-8, sqrt(3) / 2 by 1.8e-8), so that a
// transform shrinks its values by up to 4e-8, all of them alike.  Over the four transforms
// of a propagation that is 1.5e-7, more than half of its error (noise at 1024^2 2.60e-7,
// with the gain 2.13e-7, in the row engine 2.37e-7).
__host__ __device__ constexpr int factors_of(int r, int lanes, int h) {
    return (split_p_of(r) + r / split_p_of(r) - (h > 1 ? 1 : 2)) * h * lanes;
}
__host__ __device__ constexpr int factors_offset(int n) { return plan_tw_size(n, engine_e(n, PassBase::EPT)); }
__host__ __device__ constexpr int twiddle_offset(int n) {
    return factors_offset(n) + factors_of(values(n), n / values(n), 1);
}
__host__ __device__ constexpr int mirror_offset(int n) { return twiddle_offset(n) + n; }
__host__ __device__ constexpr int half_offset(int n) { return mirror_offset(n) + n; }
__host__ __device__ constexpr int table_size(int n) {
    return half_offset(n) + (halves(n) > 1 ? factors_of(values(n / 2), n / 2 / values(n / 2), 2) : 0);
}

template <int N>
struct Plan {
    static constexpr int E = values(N), L = N / E, M = (E + L - 1) / L;
    static_assert(L == 16 || L == 32 || L == 64, "a row is half a warp, a warp or two");
    static constexpr int PITCH = L + 4;                      // words between the exchange rows of k1, k1 + 1
    // words of a row's exchange region; two rows of one warp (L = 16) sit 16 banks apart
    static constexpr int XWORDS = E * PITCH + (L == 16 && (E * PITCH) % 32 == 0 ? 16 : 0);
    static constexpr int P = split_p<E>(), Q = split_q<E>();
};

// The factors of a thread's stage twiddles: W_N^(l (k1 + P k2)) = a[k1] b[k2].
// H = 2: the transform is half h (the even or odd outputs) of one of length 2 N;
// the inputs of h = 1 still lack the lane's factor W_2N^l, which goes into a.
template <int N, bool INV, int H = 1>
struct Factors {
    using PL = Plan<N>;
    static constexpr int P0 = H > 1 ? 0 : 1;          // the first factor that is not 1
    static constexpr int COUNT = PL::P - P0 + PL::Q - 1;
    static constexpr size_t BYTES = (size_t)COUNT * H * PL::L * 8;
    float2 a[PL::P], b[PL::Q];
    // The CTA's copy of the table, [factor][h][l], so that a warp's loads are contiguous
    // (from the W^i table they would be gathers of up to 32 lines).  tw: the table of H N.
    __device__ __forceinline__ static void fill(float2 *tab, const float2 *__restrict__ tw) {
        static_assert(COUNT * H * PL::L == factors_of(PL::E, PL::L, H), "as the table holds them");
        constexpr int at = H == 1 ? factors_offset(N) : half_offset(H * N);
        for (int i = threadIdx.x; i < COUNT * H * PL::L; i += blockDim.x) tab[i] = load_tw<INV>(tw, at + i);
    }
    __device__ __forceinline__ void load(const float2 *tab, int l, int h = 0) {
        tab += h * PL::L + l;
#pragma unroll
        for (int p = P0; p < PL::P; ++p) a[p] = tab[(p - P0) * H * PL::L];
#pragma unroll
        for (int q = 1; q < PL::Q; ++q) b[q] = tab[(PL::P - P0 + q - 1) * H * PL::L];
    }
    // v times the twiddle of output k
    __device__ __forceinline__ float2 apply(int k, float2 v) const {
        const int p = k % PL::P, q = k / PL::P;
        if (P0 == 1 && p == 0 && q == 0) return v;
        if (q == 0) return cmul2(v, a[p]);
        if (P0 == 1 && p == 0) return cmul2(v, b[q]);
        return cmul2(v, cmul2(a[p], b[q]));
    }
};

// v times the stage twiddle of output k of thread l (of lanes), from the length's table at
// `offset`: rounded once, where the passes of one transform per launch have it at hand.
// (As products of two rounded factors the noise of a propagated field was 2 to 17 %
// higher, 13 % at 1024^2.)
template <bool INV>
__device__ __forceinline__ float2 stage_twiddle(const float2 *__restrict__ tw, int offset, int k, int lanes, int l,
                                                float2 v) {
    return k == 0 ? v : cmul2(v, load_tw<INV>(tw, offset + k * lanes + l));
}

// One exchange through the row's region `ex`: v[k1] of thread t -> u[m L + i] =
// the value of (l = i, k1 = t + L m).  sync covers the threads of the region.
template <int N, class Sync>
__device__ __forceinline__ void exchange(const float2 (&v)[Plan<N>::E], float2 (&u)[Plan<N>::M * Plan<N>::L], float *ex,
                                         int t, const Sync &sync) {
    using PL = Plan<N>;
    float *wr = ex + t;
    // (an idle thread reads the last row)
    const auto row = [&](int m) {
        return ex + (PL::M * PL::L == PL::E ? t + PL::L * m : min(t + PL::L * m, PL::E - 1)) * PL::PITCH;
    };
#pragma unroll
    for (int k = 0; k < PL::E; ++k) wr[k * PL::PITCH] = v[k].x;
    sync();
#pragma unroll
    for (int m = 0; m < PL::M; ++m) {
        const float *rd = row(m);
#pragma unroll
        for (int i = 0; i < PL::L; i += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(rd + i);
            u[m * PL::L + i].x = q.x;
            u[m * PL::L + i + 1].x = q.y;
            u[m * PL::L + i + 2].x = q.z;
            u[m * PL::L + i + 3].x = q.w;
        }
    }
    sync();
#pragma unroll
    for (int k = 0; k < PL::E; ++k) wr[k * PL::PITCH] = v[k].y;
    sync();
#pragma unroll
    for (int m = 0; m < PL::M; ++m) {
        const float *rd = row(m);
#pragma unroll
        for (int i = 0; i < PL::L; i += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(rd + i);
            u[m * PL::L + i].y = q.x;
            u[m * PL::L + i + 1].y = q.y;
            u[m * PL::L + i + 2].y = q.z;
            u[m * PL::L + i + 3].y = q.w;
        }
    }
}

// ---------------------------------------------------------------- the mirrored transform

// The outputs of a transform sit as its mirror's inputs: thread t holds x[t' + E i],
// t' = t + L m (m < M), i < L.  Stage 1: transforms of length L over i, times
// W_N^(t' q1).  Exchange through rows q1 of E words (pitch E + 4).  Stage 2: thread
// t = q1 holds the E values t' and transforms them: output q2 is X[q1 + L q2].  So
// two transforms with a product between them need one exchange each.
template <int N>
struct Mirror {
    using PL = Plan<N>;
    static constexpr int PITCH = PL::E + 4;
    // words of a row's region for both exchanges; two rows of one warp 16 banks apart
    static constexpr int WORDS = cmax(PL::E * PL::PITCH, PL::L * PITCH);
    static constexpr int XWORDS = PL::L == 16 ? (WORDS + 31) / 32 * 32 + 16 : WORDS;
};
// v[m L + q1] of thread t (t' = t + L m) -> y[t'] of thread q1.
template <int N, class Sync>
__device__ __forceinline__ void mirror_exchange(const float2 (&v)[Plan<N>::M * Plan<N>::L], float2 (&y)[Plan<N>::E],
                                                float *ex, int t, const Sync &sync) {
    using PL = Plan<N>;
    constexpr int PITCH = Mirror<N>::PITCH;
    const float *rd = ex + t * PITCH;
    const auto half = [&](auto part) {
        constexpr int c = decltype(part)::value;
        sync();   // the region's last reads
#pragma unroll
        for (int m = 0; m < PL::M; ++m)
            if (PL::M * PL::L == PL::E || t + PL::L * m < PL::E) {
#pragma unroll
                for (int q = 0; q < PL::L; ++q) ex[q * PITCH + t + PL::L * m] = c == 0 ? v[m * PL::L + q].x : v[m * PL::L + q].y;
            }
        sync();
#pragma unroll
        for (int i = 0; i < PL::E; i += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(rd + i);
            (c == 0 ? y[i].x : y[i].y) = q.x;
            (c == 0 ? y[i + 1].x : y[i + 1].y) = q.y;
            (c == 0 ? y[i + 2].x : y[i + 2].y) = q.z;
            (c == 0 ? y[i + 3].x : y[i + 3].y) = q.w;
        }
    };
    half(std::integral_constant<int, 0>{});
    half(std::integral_constant<int, 1>{});
}

// ---------------------------------------------------------------- tensor memory as thread-private storage

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15};" ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]),
        "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
}
// Waits for the loads issued so far; the values pass through it, so that no use moves above it.
__device__ __forceinline__ void tmem_wait(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]),
                   "+f"(v[15])::"memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float2 (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(v[0].x),
                 "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

}  // namespace two
}  // namespace ph
