// ph_ccl.cu -- connected-component labeling of equal-valued 8-connected
// regions (the semantics of ParticleHolography.jl src/ccl.jl:186-211) by
// lock-free union-find, plus the root compaction behind count_labels /
// cu_find_valid_labels (ccl.jl:213-238) and device-side bounding rectangles.
//
// Union-find after the published ECL-CC scheme (Jaiganesh & Burtscher, HPDC
// 2018).  Parents are kept in label form throughout: pixel i of an image holds
// 1 + the index (within its image) of its parent, background holds 0.  Every
// parent is at most the pixel itself, and a root holds its own index + 1;
// hooking links the larger of two roots to the smaller with compare-and-swap;
// finds shorten the path they walk (pointer jumping).  The root of a tree is
// therefore the minimum linear index of its component, and what a pixel holds
// once it points at its root is the reference's label.  Every loop is bounded by
// an iteration limit that raises the context's error flag instead of running on.
#include <cstdint>
#include <cuda_runtime.h>

namespace ph {

template <class T>
__device__ __forceinline__ bool ccl_fg(T v);
template <>
__device__ __forceinline__ bool ccl_fg<float>(float v) { return v > 0.0f; }
template <>
__device__ __forceinline__ bool ccl_fg<uint8_t>(uint8_t v) { return v != 0; }

// Equality of pixel values: Float32 compares the values, Bool its truth.
__device__ __forceinline__ bool ccl_eq(float a, float b) { return a == b; }
__device__ __forceinline__ bool ccl_eq(uint8_t a, uint8_t b) { return (a != 0) == (b != 0); }

// Root of x, shortening the walked path on the way (benign races: every
// value written is an ancestor of the slot it is written to).
__device__ __forceinline__ uint32_t ccl_find(uint32_t *lab, uint32_t x, int64_t limit, int *err) {
    uint32_t cur = __ldcg(lab + x);
    if (cur == x) return x;
    uint32_t prev = x;
    int64_t it = 0;
    uint32_t next;
    while (cur > (next = __ldcg(lab + cur))) {
        lab[prev] = next;
        prev = cur;
        cur = next;
        if (++it > limit) { atomicExch(err, 1); break; }
    }
    return cur;
}

// Root of x without writing anything: the flatten pass may not shorten other
// pixels' paths, or a shortcut written after that pixel's own final root would
// leave a non-root label behind.
__device__ __forceinline__ uint32_t ccl_root(const uint32_t *lab, uint32_t x, int64_t limit, int *err) {
    uint32_t cur = __ldcg(lab + x), next;
    int64_t it = 0;
    while (cur > (next = __ldcg(lab + cur))) {
        cur = next;
        if (++it > limit) { atomicExch(err, 1); break; }
    }
    return cur;
}

// Links the trees of a and b (the larger root under the smaller).
__device__ __forceinline__ void ccl_hook(uint32_t *lab, uint32_t a, uint32_t b, int64_t limit, int *err) {
    uint32_t ra = ccl_find(lab, a, limit, err);
    uint32_t rb = ccl_find(lab, b, limit, err);
    int64_t it = 0;
    while (ra != rb) {
        if (ra < rb) { uint32_t t = ra; ra = rb; rb = t; }
        // ra > rb: make ra point to rb if ra is still a root
        const uint32_t ret = atomicCAS(lab + ra, ra, rb);
        if (ret == ra) return;
        ra = ret;   // ra gained a parent meanwhile: continue from it
        if (++it > limit) { atomicExch(err, 1); return; }
    }
}

// ---- tile-local phase: one CTA labels a 32 x 32 tile in shared memory

constexpr int kTile = 32;

// Local root of tile pixel x (parents in shared memory), shortening the path.
__device__ __forceinline__ int ccl_lfind(volatile int *p, int x, int64_t limit, int *err) {
    int cur = p[x];
    if (cur == x) return x;
    int prev = x, next;
    int64_t it = 0;
    while (cur > (next = p[cur])) {
        p[prev] = next;
        prev = cur;
        cur = next;
        if (++it > limit) { atomicExch(err, 1); break; }
    }
    return cur;
}

__device__ __forceinline__ int ccl_lroot(volatile int *p, int x, int64_t limit, int *err) {
    int cur = p[x], next;
    int64_t it = 0;
    while (cur > (next = p[cur])) {
        cur = next;
        if (++it > limit) { atomicExch(err, 1); break; }
    }
    return cur;
}

__device__ __forceinline__ void ccl_lhook(int *p, int a, int b, int64_t limit, int *err) {
    int ra = ccl_lfind(p, a, limit, err), rb = ccl_lfind(p, b, limit, err);
    int64_t it = 0;
    while (ra != rb) {
        if (ra < rb) { const int t = ra; ra = rb; rb = t; }
        const int ret = atomicCAS(p + ra, ra, rb);
        if (ret == ra) return;
        ra = ret;
        if (++it > limit) { atomicExch(err, 1); return; }
    }
}

// Each 32 x 32 tile on its own, one warp per tile.  What bounds it is memory
// (read the image, write the labels), as long as a tile costs few instructions:
//  - an empty tile writes zeros (most tiles of a thresholded volume);
//  - a tile with one foreground value is a bit mask, one 32-bit word per row, lane
//    = row.  Its nodes are the runs of each row: a run starts at the first run of
//    the row above that it touches (its range widened by one, 8-connectivity) and
//    hooks the others; then pointer doubling over the runs;
//  - a tile of several values is hooked pixel by pixel.
// Inside a tile, row-major order is linear order, so a local root is the minimum
// index of its local component.  A row that starts a slice has no row above.
// (100 x 1024^2 Bool, about 1 % foreground: 0.32 ms with one 256-thread CTA per
// tile and pixel-wise hooks, 0.137 ms in this form, where the copy rate allows
// 0.077; what follows it, border, compression and background, 0.66 ms before and
// 0.10 ms now.)
template <class T>
struct CclLocal {
    static constexpr int WARPS = sizeof(T) == 1 ? 8 : 4;
};

template <class T>
__global__ void __launch_bounds__(CclLocal<T>::WARPS * 32)
    k_ccl_local(const T *__restrict__ img, uint32_t *__restrict__ lab, uint32_t rows, uint32_t cols, uint32_t tiles_x,
                uint64_t tiles, uint32_t slice_rows, int64_t limit, int *err) {
    constexpr int WARPS = CclLocal<T>::WARPS;
    __shared__ int s_parent[WARPS][kTile * kTile];
    __shared__ T s_value[sizeof(T) == 1 ? 1 : WARPS][sizeof(T) == 1 ? 1 : kTile * kTile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t tile = (uint64_t)blockIdx.x * WARPS + warp;
    if (tile >= tiles) return;
    int *sp = s_parent[warp];
    const uint32_t y0 = (uint32_t)(tile / tiles_x) * kTile, x0 = (uint32_t)(tile % tiles_x) * kTile;
    const uint32_t nrows = min((uint32_t)kTile, rows - y0);
    const bool xin = x0 + lane < cols;
    const size_t at = (size_t)y0 * cols + x0 + lane;   // pixel (0, lane) of the tile
    // lane = column while the rows are read; the ballots leave row r's mask in lane r
    T v[sizeof(T) == 1 ? 1 : kTile];
    uint32_t m = 0;
    T first = T(0);
#pragma unroll
    for (int r = 0; r < kTile; ++r) {
        const T q = (xin && r < nrows) ? img[at + (size_t)r * cols] : T(0);
        const uint32_t b = __ballot_sync(0xffffffffu, ccl_fg<T>(q));
        if (lane == r) m = b;
        if constexpr (sizeof(T) != 1) {
            v[r] = q;
            if (!ccl_fg<T>(first)) first = ccl_fg<T>(q) ? q : first;
        }
    }
    if (!__any_sync(0xffffffffu, m != 0)) {
        if (xin)
            for (uint32_t r = 0; r < nrows; ++r) lab[at + (size_t)r * cols] = 0;
        return;
    }
    // lane = row from here: its index within its slice
    const uint32_t yl = (y0 + lane) % slice_rows;
    bool one_value = true;
    if constexpr (sizeof(T) != 1) {
        const T v0 = __shfl_sync(0xffffffffu, first, __ffs(__ballot_sync(0xffffffffu, ccl_fg<T>(first))) - 1);
#pragma unroll
        for (int r = 0; r < kTile; ++r) one_value = one_value && (!ccl_fg<T>(v[r]) || ccl_eq(v[r], v0));
        one_value = __all_sync(0xffffffffu, one_value);
    }
    if (one_value) {
        uint32_t up = __shfl_up_sync(0xffffffffu, m, 1);
        if (lane == 0 || yl == 0) up = 0;
        const uint32_t starts = m & ~(m << 1), up_starts = up & ~(up << 1);
        // the bits of up that the run starting at s touches; the run of up that holds bit b
        const auto touching = [&](int s) {
            const uint32_t run = m & ~(m + (1u << s)) & (~0u << s);   // s and the ones above it
            return up & (run | (run << 1) | (run >> 1));
        };
        const auto up_run = [&](int b) { return 31 - __clz(up_starts & ((2u << b) - 1u)); };
        for (uint32_t t = starts; t; t &= t - 1) {
            const int s = __ffs(t) - 1;
            const uint32_t ov = touching(s);
            sp[lane * kTile + s] = ov ? (lane - 1) * kTile + up_run(__ffs(ov) - 1) : lane * kTile + s;
        }
        __syncwarp();
        for (uint32_t t = starts; t; t &= t - 1) {
            const int s = __ffs(t) - 1;
            uint32_t ov = touching(s);
            for (bool linked = true; ov; linked = false) {   // the first run is the parent already
                const int u = up_run(__ffs(ov) - 1);
                if (!linked) ccl_lhook(sp, lane * kTile + s, (lane - 1) * kTile + u, limit, err);
                ov &= up + (1u << u);                         // past that run
            }
        }
        __syncwarp();
        for (int i = 0; i < 5; ++i) {   // pointer doubling: the usual depth, a row each
            for (uint32_t t = starts; t; t &= t - 1) {
                const int n = lane * kTile + __ffs(t) - 1;
                sp[n] = sp[sp[n]];
            }
            __syncwarp();
        }
        for (uint32_t t = starts; t; t &= t - 1) {   // (each writes its own root only)
            const int n = lane * kTile + __ffs(t) - 1;
            sp[n] = ccl_lroot(sp, n, limit, err);
        }
        __syncwarp();
        for (int r = 0; r < (int)nrows; ++r) {
            const uint32_t mr = __shfl_sync(0xffffffffu, m, r), yr = __shfl_sync(0xffffffffu, yl, r);
            uint32_t l = 0;
            if ((mr >> lane) & 1u) {
                const int q = sp[r * kTile + 31 - __clz((mr & ~(mr << 1)) & ((2u << lane) - 1u))];
                l = (yr - (uint32_t)(r - q / kTile)) * cols + x0 + (uint32_t)(q % kTile) + 1u;
            }
            if (xin) lab[at + (size_t)r * cols] = l;
        }
        return;
    }
    if constexpr (sizeof(T) != 1) {   // several values: pixel by pixel, lane = column
        T *sv = s_value[warp];
#pragma unroll
        for (int r = 0; r < kTile; ++r) sv[r * kTile + lane] = v[r];
        __syncwarp();
        for (int r = 0; r < kTile; ++r) {
            const int l = r * kTile + lane;
            const T q = sv[l];
            const bool top = r == 0 || __shfl_sync(0xffffffffu, yl, r) == 0;
            int p = l;
            if (ccl_fg<T>(q)) {
                if (lane > 0 && ccl_eq(sv[l - 1], q)) p = l - 1;
                if (!top) {
                    if (lane + 1 < kTile && ccl_eq(sv[l - kTile + 1], q)) p = l - kTile + 1;
                    if (ccl_eq(sv[l - kTile], q)) p = l - kTile;
                    if (lane > 0 && ccl_eq(sv[l - kTile - 1], q)) p = l - kTile - 1;
                }
            }
            sp[l] = p;
        }
        __syncwarp();
        for (int r = 0; r < kTile; ++r) {
            const int l = r * kTile + lane;
            const T q = sv[l];
            const bool top = r == 0 || __shfl_sync(0xffffffffu, yl, r) == 0;
            if (!ccl_fg<T>(q)) continue;
            if (lane > 0 && ccl_eq(sv[l - 1], q)) ccl_lhook(sp, l, l - 1, limit, err);
            if (!top) {
                if (lane > 0 && ccl_eq(sv[l - kTile - 1], q)) ccl_lhook(sp, l, l - kTile - 1, limit, err);
                if (ccl_eq(sv[l - kTile], q)) ccl_lhook(sp, l, l - kTile, limit, err);
                if (lane + 1 < kTile && ccl_eq(sv[l - kTile + 1], q)) ccl_lhook(sp, l, l - kTile + 1, limit, err);
            }
        }
        __syncwarp();
        for (int r = 0; r < (int)nrows; ++r) {
            const int l = r * kTile + lane;
            const uint32_t yr = __shfl_sync(0xffffffffu, yl, r);
            uint32_t out = 0;
            if (ccl_fg<T>(sv[l])) {
                const int q = ccl_lroot(sp, l, limit, err);
                out = (yr - (uint32_t)(r - q / kTile)) * cols + x0 + (uint32_t)(q % kTile) + 1u;
            }
            if (xin) lab[at + (size_t)r * cols] = out;
        }
    }
}

// ---- merge across tile borders: the pairs whose earlier neighbour lies in
// another tile (W, NW of the left column; NW, N, NE of the top row; NE of the
// right column) are hooked in the global parents.  One warp per tile, its 94
// border pixels in three rounds.  Within a warp, pairs whose current parents are
// the same two nodes link the same two trees, so one lane of each such set hooks
// (between tiles of one value, as in a near-total foreground, one hook per
// neighbour tile instead of one per border pixel).
// `base`: the labels of the pixels' slice start there; a, b: pixels of it.
__device__ __forceinline__ void ccl_hook_dedup(uint32_t *lab, bool cond, size_t base, size_t a, size_t b, int64_t limit,
                                               int *err) {
    const unsigned act = __ballot_sync(0xffffffffu, cond);
    if (cond) {
        const uint32_t la = __ldcg(lab + a), lb = __ldcg(lab + b);
        const unsigned long long key = ((unsigned long long)(uint32_t)(base + la) << 32) | (uint32_t)(base + lb);
        const unsigned peers = __match_any_sync(act, key);
        // labels of a slice are 1-based: node n of the slice is lab[base - 1 + n]
        if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) ccl_hook(lab + base - 1, la, lb, limit, err);
    }
}

template <class T>
__global__ void __launch_bounds__(256)
    k_ccl_border(const T *__restrict__ img, uint32_t *lab, uint32_t rows, uint32_t cols, uint32_t tiles_x, uint64_t tiles,
                 uint32_t slice_rows, int64_t limit, int *err) {
    const uint64_t tile = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= tiles) return;
    const int lane = threadIdx.x & 31;
    const uint32_t y0 = (uint32_t)(tile / tiles_x) * kTile, x0 = (uint32_t)(tile % tiles_x) * kTile;
    // lane = column of the top row, then row of the left and of the right column
#pragma unroll
    for (int round = 0; round < 3; ++round) {
        const uint32_t y = y0 + (round == 0 ? 0 : lane), x = x0 + (round == 0 ? lane : round == 1 ? 0 : kTile - 1);
        const bool on = y < rows && x < cols && (round == 0 || lane > 0);
        const size_t i = (size_t)y * cols + x;
        const T v = on ? img[i] : T(0);
        const bool fg = on && ccl_fg<T>(v);
        if (!__any_sync(0xffffffffu, fg)) continue;
        const uint32_t yl = y % slice_rows;
        const size_t base = (size_t)(y - yl) * cols, u = i - cols;
        const bool up = fg && yl != 0;
        if (round == 0) {
            ccl_hook_dedup(lab, fg && lane == 0 && x > 0 && ccl_eq(img[i - 1], v), base, i, i - 1, limit, err);
            ccl_hook_dedup(lab, up && x > 0 && ccl_eq(img[u - 1], v), base, i, u - 1, limit, err);
            ccl_hook_dedup(lab, up && ccl_eq(img[u], v), base, i, u, limit, err);
            ccl_hook_dedup(lab, up && x + 1 < cols && ccl_eq(img[u + 1], v), base, i, u + 1, limit, err);
        } else if (round == 1) {
            ccl_hook_dedup(lab, fg && x > 0 && ccl_eq(img[i - 1], v), base, i, i - 1, limit, err);
            ccl_hook_dedup(lab, up && x > 0 && ccl_eq(img[u - 1], v), base, i, u - 1, limit, err);
        } else {
            ccl_hook_dedup(lab, up && x + 1 < cols && ccl_eq(img[u + 1], v), base, i, u + 1, limit, err);
        }
    }
}

// Every foreground pixel takes its root's label.  The foreground is found in the
// smaller array: the image where a pixel is one byte (16 per load, VEC), else the
// labels (4 per load), both 16-byte aligned.
template <class T, bool VEC>
__global__ void __launch_bounds__(256)
    k_ccl_flatten(const T *__restrict__ img, uint32_t *lab, int64_t n, int64_t slice_n, int64_t limit, int *err) {
    constexpr int K = !VEC ? 1 : sizeof(T) == 1 ? 16 : 4;
    const int64_t i0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) * K;
    if (i0 >= n) return;
    uint32_t last = 0, last_root = 0;
    int64_t base = (i0 / slice_n) * slice_n;
    const auto flatten = [&](int64_t i) {
        if (i - base >= slice_n) { base = (i / slice_n) * slice_n; last = 0; }
        uint32_t *p = lab + base - 1;   // node of the slice -> its parent
        const uint32_t l = lab[i];
        if (l != last) { last = l; last_root = ccl_root(p, l, limit, err); }   // a run's pixels hold one label
        if (last_root != l) lab[i] = last_root;
    };
    if constexpr (!VEC) {
        if (ccl_fg<T>(img[i0])) flatten(i0);
    } else if constexpr (sizeof(T) == 1) {
        if (i0 + K <= n) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(img + i0));
            if ((q.x | q.y | q.z | q.w) == 0) return;
        }
        for (int64_t w = i0; w < min(i0 + K, n); w += 4) {
            if (w + 4 <= n && *reinterpret_cast<const uint32_t *>(img + w) == 0) continue;
            for (int64_t i = w; i < min(w + 4, n); ++i)
                if (ccl_fg<T>(img[i])) flatten(i);
        }
    } else {
        if (i0 + K <= n) {
            const uint4 q = *reinterpret_cast<const uint4 *>(lab + i0);
            if ((q.x | q.y | q.z | q.w) == 0) return;
        }
        for (int64_t i = i0; i < min(i0 + K, n); ++i)
            if (lab[i] != 0) flatten(i);
    }
}

template <class T>
static cudaError_t ccl_run(const T *img, uint32_t *lab, int64_t rows, int64_t cols, int64_t slice_rows, int64_t limit,
                           int *err, cudaStream_t s, int64_t *launches) {
    const int64_t n = rows * cols;
    const uint64_t tiles_x = (uint64_t)(cols + kTile - 1) / kTile, tiles = tiles_x * (uint64_t)((rows + kTile - 1) / kTile);
    constexpr int W = CclLocal<T>::WARPS;
    k_ccl_local<T><<<(unsigned)((tiles + W - 1) / W), W * 32, 0, s>>>(img, lab, (uint32_t)rows, (uint32_t)cols,
                                                                     (uint32_t)tiles_x, tiles, (uint32_t)slice_rows,
                                                                     limit, err);
    k_ccl_border<T><<<(unsigned)((tiles + 7) / 8), 256, 0, s>>>(img, lab, (uint32_t)rows, (uint32_t)cols,
                                                                (uint32_t)tiles_x, tiles, (uint32_t)slice_rows, limit,
                                                                err);
    const void *scanned = sizeof(T) == 1 ? static_cast<const void *>(img) : static_cast<const void *>(lab);
    const int64_t slice_n = slice_rows * cols;
    if (((uintptr_t)scanned & 15) == 0) {
        const int64_t k = sizeof(T) == 1 ? 16 : 4;
        k_ccl_flatten<T, true><<<(unsigned)((n + 256 * k - 1) / (256 * k)), 256, 0, s>>>(img, lab, n, slice_n, limit, err);
    } else {
        k_ccl_flatten<T, false><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(img, lab, n, slice_n, limit, err);
    }
    *launches += 3;
    return cudaGetLastError();
}

// Labels `rows x cols` pixels; with slice_rows < rows, every slice_rows rows
// form an independent image (a batch of slices labelled in one launch set).
cudaError_t ccl_launch(const void *img, bool is_bool, uint32_t *lab, int64_t rows, int64_t cols, int64_t slice_rows,
                       int64_t limit, int *err, cudaStream_t s, int64_t *launches) {
    if (rows <= 0 || cols <= 0) return cudaSuccess;
    if (slice_rows <= 0 || slice_rows > rows) slice_rows = rows;
    if (is_bool)
        return ccl_run<uint8_t>(static_cast<const uint8_t *>(img), lab, rows, cols, slice_rows, limit, err, s,
                                launches);
    return ccl_run<float>(static_cast<const float *>(img), lab, rows, cols, slice_rows, limit, err, s, launches);
}

// ---------------------------------------------------------------- bounding rectangles

// boxes[4 r .. 4 r + 3] = (min slow, min fast, max slow, max fast) over the pixels
// of the root of rank r < count (0-based).  VEC: four pixels of one row per thread
// (16-byte aligned labels, cols a multiple of 4), one update per run of equal labels.
template <bool VEC>
__global__ void __launch_bounds__(256)
    k_boxes(const uint32_t *__restrict__ lab, int64_t n, uint32_t cols, int64_t slice_n, const unsigned *__restrict__ rank,
            int *boxes, int64_t count) {
    constexpr int K = VEC ? 4 : 1;
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * K;
    if (i >= n) return;
    uint32_t l[K];
    if constexpr (VEC) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(lab + i));
        l[0] = q.x; l[1] = q.y; l[2] = q.z; l[3] = q.w;
        if ((q.x | q.y | q.z | q.w) == 0) return;
    } else {
        l[0] = lab[i];
        if (l[0] == 0) return;
    }
    const int64_t base = (i / slice_n) * slice_n;
    const uint32_t li = (uint32_t)(i - base);
    const int slow = (int)(li / cols), fast = (int)(li % cols);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (l[k] == 0 || (k > 0 && l[k] == l[k > 0 ? k - 1 : 0])) continue;   // the start of a run
        int e = k;
#pragma unroll
        for (int q = k + 1; q < K; ++q)
            if (e == q - 1 && l[q] == l[k]) e = q;
        const unsigned r = rank[base + l[k] - 1];
        if ((int64_t)r >= count) continue;
        int *b = boxes + 4 * (int64_t)r;
        atomicMin(b + 0, slow);
        atomicMin(b + 1, fast + k);
        atomicMax(b + 2, slow);
        atomicMax(b + 3, fast + e);
    }
}

__global__ void k_boxes_init(int *boxes, int64_t count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    boxes[4 * i + 0] = 0x7fffffff;
    boxes[4 * i + 1] = 0x7fffffff;
    boxes[4 * i + 2] = -1;
    boxes[4 * i + 3] = -1;
}

// ---------------------------------------------------------------- root compaction

constexpr int kRootThreads = 256;
constexpr int kRootItems = 16;                       // per thread
constexpr int kRootTile = kRootThreads * kRootItems; // elements per block

// The thread's 16 labels of a block, four consecutive ones at a time:
// f(j, label, is root) for element j = 4 (256 k + thread) + q of the block.  A
// root carries its own index (within its image of slice_n pixels) plus one; the
// index is followed from the block's start (one 64-bit division per block).
template <class F>
__device__ __forceinline__ void block_labels(const uint32_t *__restrict__ lab, int64_t n, int64_t slice_n, F &&f) {
    const int64_t base = (int64_t)blockIdx.x * kRootTile;
    const int64_t in_slice = base % slice_n;
    const bool vec = base + kRootTile <= n && ((uintptr_t)lab & 15) == 0;
#pragma unroll
    for (int k = 0; k < kRootItems / 4; ++k) {
        const int j = 4 * (kRootThreads * k + (int)threadIdx.x);
        uint32_t l[4] = {0, 0, 0, 0};
        if (vec) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(lab + base + j));
            l[0] = q.x; l[1] = q.y; l[2] = q.z; l[3] = q.w;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (base + j + q < n) l[q] = lab[base + j + q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (l[q] == 0) { f(j + q, 0u, false); continue; }
            int64_t at = in_slice + j + q;
            if (at >= slice_n) at = slice_n > kRootTile ? at - slice_n : at % slice_n;
            f(j + q, l[q], l[q] == (uint32_t)(at + 1));
        }
    }
}

__global__ void __launch_bounds__(kRootThreads)
    k_roots_count(const uint32_t *__restrict__ lab, int64_t n, int64_t slice_n, unsigned *counts) {
    __shared__ unsigned wsum[kRootThreads / 32];
    unsigned c = 0;
    block_labels(lab, n, slice_n, [&](int, uint32_t, bool root) { c += root; });
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < kRootThreads / 32; ++w) t += wsum[w];
        counts[blockIdx.x] = t;
    }
}

// Exclusive scan of `nb` block counts in place (one CTA, 8 counts per thread and
// round); total -> total[0], and with `flag` the error word it points at -> total[1].
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_roots_scan(unsigned *counts, int64_t nb, unsigned long long *total,
                                                            const int *flag) {
    __shared__ unsigned long long wsum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (int64_t off = 0; off < nb; off += kScanThreads * 8) {
        const int64_t i = off + (int64_t)threadIdx.x * 8;
        unsigned c[8];
        unsigned long long sum = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) { c[q] = i + q < nb ? counts[i + q] : 0u; sum += c[q]; }
        unsigned long long incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        if (w == 0) {
            unsigned long long ws = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long u = __shfl_up_sync(0xffffffffu, ws, o);
                if (lane >= o) ws += u;
            }
            wsum[lane] = ws;
        }
        __syncthreads();
        unsigned long long run = carry + (w > 0 ? wsum[w - 1] : 0ull) + incl - sum;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (i + q < nb) counts[i + q] = (unsigned)run;
            run += c[q];
        }
        carry += wsum[kScanThreads / 32 - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *total = carry;
        if (flag) total[1] = (unsigned long long)(unsigned)*flag;
    }
}

// Writes the 1-based linear index of every root, in increasing order, and (rank
// non-null) rank[i] = the root's position in that order.  offsets: the scanned
// counts; a block without roots is done at once.
__global__ void __launch_bounds__(kRootThreads)
    k_roots_write(const uint32_t *__restrict__ lab, int64_t n, int64_t slice_n, const unsigned *offsets, int64_t nb,
                  const unsigned long long *total, long long *out, int64_t cap, unsigned *rank) {
    __shared__ unsigned roots[kRootTile / 32];   // one bit per element of the block
    const unsigned first = offsets[blockIdx.x];
    const unsigned last = (int64_t)blockIdx.x + 1 < nb ? offsets[blockIdx.x + 1] : (unsigned)*total;
    if (first == last) return;
    if (threadIdx.x < kRootTile / 32) roots[threadIdx.x] = 0;
    __syncthreads();
    block_labels(lab, n, slice_n, [&](int j, uint32_t, bool root) {
        if (root) atomicOr(&roots[j >> 5], 1u << (j & 31));
    });
    __syncthreads();
    if (threadIdx.x < kRootTile / 32) {   // 128 threads, 32 elements each
        unsigned m = roots[threadIdx.x], pre = first;
        for (unsigned q = 0; q < threadIdx.x; ++q) pre += __popc(roots[q]);
        const int64_t base = (int64_t)blockIdx.x * kRootTile + threadIdx.x * 32;
        for (; m; m &= m - 1, ++pre) {
            const int64_t i = base + __ffs(m) - 1;
            if ((int64_t)pre < cap && out) out[pre] = (long long)(i + 1);
            if (rank) rank[i] = pre;
        }
    }
}

int64_t roots_blocks(int64_t n) { return (n + kRootTile - 1) / kRootTile; }

cudaError_t roots_count_launch(const uint32_t *lab, int64_t n, int64_t slice_n, unsigned *counts,
                               unsigned long long *total, const int *flag, cudaStream_t s, int64_t *launches) {
    const int64_t nb = roots_blocks(n);
    k_roots_count<<<(unsigned)nb, kRootThreads, 0, s>>>(lab, n, slice_n, counts);
    k_roots_scan<<<1, kScanThreads, 0, s>>>(counts, nb, total, flag);
    *launches += 2;
    return cudaGetLastError();
}

cudaError_t roots_write_launch(const uint32_t *lab, int64_t n, int64_t slice_n, const unsigned *offsets,
                               const unsigned long long *total, long long *out, int64_t cap, unsigned *rank,
                               cudaStream_t s, int64_t *launches) {
    const int64_t nb = roots_blocks(n);
    k_roots_write<<<(unsigned)nb, kRootThreads, 0, s>>>(lab, n, slice_n, offsets, nb, total, out, cap, rank);
    *launches += 1;
    return cudaGetLastError();
}

// Boxes of the roots of rank < count (their ranks are in `rank`, see k_roots_write).
cudaError_t boxes_launch(const uint32_t *lab, int64_t rows, int64_t cols, int64_t slice_rows, const unsigned *rank,
                         int *boxes, int64_t count, cudaStream_t s, int64_t *launches) {
    if (count > 0) k_boxes_init<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(boxes, count);
    const int64_t n = rows * cols, slice_n = slice_rows * cols;
    if (((uintptr_t)lab & 15) == 0 && cols % 4 == 0)
        k_boxes<true><<<(unsigned)((n / 4 + 255) / 256), 256, 0, s>>>(lab, n, (uint32_t)cols, slice_n, rank, boxes, count);
    else
        k_boxes<false><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(lab, n, (uint32_t)cols, slice_n, rank, boxes, count);
    *launches += 2;
    return cudaGetLastError();
}

}  // namespace ph
