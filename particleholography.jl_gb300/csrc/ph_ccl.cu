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
#include <type_traits>
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

// Each 32 x 32 tile on its own, one warp per tile, lane = column.  What bounds it is
// memory (read the image, write the labels) where most tiles are empty, as in a
// thresholded volume, and the latency of one warp's instructions in a small image.
// The tile's rows are read first (an empty tile writes zeros); then the rows are
// joined from the top, so that every pixel is given a root of the rows above:
//  - a pixel takes the root of the equal pixel above it, or of an upper neighbour on
//    a diagonal; a run of equal pixels takes that of its first pixel that has one, or
//    is a root itself at its first pixel;
//  - where a run meets a second root, the two trees are hooked, and the roots that
//    the lanes hold are found again.
// So the trees are about one level deep, and what a row costs does not depend on how
// many runs it holds: with lane = row, each lane walking its own runs, stripes at 512^2
// took 71 us, now 28 (256 threads per tile, pixel by pixel: 29), and 5 % noise at 2048^2
// 56 and 40 (72).  Inside a tile, row-major order is linear order, so a local
// root is the minimum index of its local component.  A row that starts a slice has no
// row above.
template <class T>
struct CclLocal {
    static constexpr int WARPS = sizeof(T) == 1 ? 8 : 4;
};

template <class T>
__global__ void __launch_bounds__(CclLocal<T>::WARPS * 32)
    k_ccl_local(const T *__restrict__ img, uint32_t *__restrict__ lab, uint32_t rows, uint32_t cols, uint32_t tiles_x,
                uint32_t tiles, uint32_t slice_rows, int64_t limit, int *err) {
    constexpr int WARPS = CclLocal<T>::WARPS;
    constexpr bool BOOL = sizeof(T) == 1;
    constexpr unsigned ALL = 0xffffffffu;
    __shared__ int s_parent[WARPS][kTile * kTile];
    __shared__ T s_value[BOOL ? 1 : WARPS][BOOL ? 1 : kTile * kTile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x * WARPS + warp;
    if (tile >= tiles) return;
    int *sp = s_parent[warp];
    T *sv = s_value[BOOL ? 0 : warp];
    const uint32_t y0 = tile / tiles_x * kTile, x0 = tile % tiles_x * kTile;
    const int nrows = (int)min((uint32_t)kTile, rows - y0);
    const bool xin = x0 + lane < cols;
    const size_t at = (size_t)y0 * cols + x0 + lane;   // pixel (0, lane) of the tile
    uint32_t mask = 0;                                 // lane r: the foreground of row r
#pragma unroll
    for (int r = 0; r < kTile; ++r) {
        const T q = (xin && r < nrows) ? img[at + (size_t)r * cols] : T(0);
        const uint32_t b = __ballot_sync(ALL, ccl_fg<T>(q));
        if (lane == r) mask = b;
        if constexpr (!BOOL) sv[r * kTile + lane] = q;
    }
    if (!__any_sync(ALL, mask != 0)) {
        if (xin)
            for (int r = 0; r < nrows; ++r) lab[at + (size_t)r * cols] = 0;
        return;
    }
    __syncwarp();
    const uint32_t yl = (y0 + lane) % slice_rows;   // lane r: the index of row r within its slice
    const uint32_t first = __shfl_sync(ALL, yl, 0);
    if (BOOL && __all_sync(ALL, mask == ALL && yl == first + lane)) {   // one component: no joining
        const uint32_t l = first * cols + x0 + 1u;
        for (int r = 0; r < kTile; ++r) lab[at + (size_t)r * cols] = l;
        return;
    }
    const uint32_t tops = __ballot_sync(ALL, yl == 0), filled = __ballot_sync(ALL, mask != 0);
    const uint32_t upto = ~0u >> (31 - lane);       // this lane and the ones before it
    int root = 0;                                   // of the pixel above, where that is foreground
    uint32_t up = 0;
    T above = T(0);
    for (uint32_t left_over = filled; left_over; left_over &= left_over - 1) {
        const int r = __ffs(left_over) - 1;
        const uint32_t m = __shfl_sync(ALL, mask, r);
        const T v = BOOL ? T(0) : sv[r * kTile + lane];
        if (((tops | ~(filled << 1)) >> r) & 1u) up = 0;   // the slice's first row, or an empty row above
        const bool fg = (m >> lane) & 1u;
        // the equal neighbours: above, above left, above right; the first pixels of the
        // runs, and the pixels that have an equal one above
        bool n = fg && ((up >> lane) & 1u), nw = fg && (((up << 1) >> lane) & 1u), ne = fg && (((up >> 1) >> lane) & 1u);
        uint32_t starts, held;
        if constexpr (BOOL) {
            starts = m & ~(m << 1);
            held = m & (up | (up << 1) | (up >> 1));
        } else {
            const T *sr = sv + r * kTile;
            const int left = max(lane - 1, 0), row_up = r > 0 ? kTile : 0;
            n = n && ccl_eq(above, v);
            nw = nw && ccl_eq(sr[left - row_up], v);
            ne = ne && ccl_eq(sr[min(lane + 1, 31) - row_up], v);
            starts = __ballot_sync(ALL, fg && !(((m << 1) >> lane) & 1u && ccl_eq(sr[left], v)));
            held = __ballot_sync(ALL, n || nw || ne);
        }
        const int rw = __shfl_up_sync(ALL, root, 1), re = __shfl_down_sync(ALL, root, 1);
        const bool has = n || nw || ne;
        const int cand = n ? root : nw ? rw : re;   // (an equal pixel above joins both diagonals)
        // the run of this pixel, [s, e), and the first pixel of it that has a root
        const int s = max(31 - __clz(starts & upto), 0);
        const uint32_t past = (starts | ~m) & ~upto;
        const uint32_t in_run = fg ? held & (past ? (1u << (__ffs(past) - 1)) - 1u : ALL) & (ALL << s) : 0u;
        const int from = __shfl_sync(ALL, cand, in_run ? __ffs(in_run) - 1 : lane);
        root = in_run ? from : r * kTile + s;
        sp[r * kTile + lane] = root;
        // a second root: of another pixel of the run, or this pixel's other diagonal
        const bool second = has && cand != root, other = !n && nw && ne && re != rw;
        if (__any_sync(ALL, second || other)) {
            const int before = __shfl_up_sync(ALL, cand, 1);   // (once for neighbours that share it)
            const bool shared = lane != s && ((held << 1) >> lane & 1u) && before == cand;
            __syncwarp();   // (the earlier rows' parents)
            if (second && !shared) ccl_lhook(sp, cand, root, limit, err);
            if (other) ccl_lhook(sp, re, root, limit, err);
            __syncwarp();
            if (fg) root = ccl_lroot(sp, root, limit, err);
        }
        up = m;
        above = v;
    }
    __syncwarp();
    for (int r0 = 0; r0 < nrows; r0 += 4) {   // (four rows' walks, nearly all of one step, side by side)
        int q[4], g[4];
        bool on[4];
        if (((filled >> r0) & 15u) == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (xin && r0 + i < nrows) lab[at + (size_t)(r0 + i) * cols] = 0;
            continue;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            on[i] = (__shfl_sync(ALL, mask, r0 + i) >> lane) & 1u;
            q[i] = on[i] ? sp[(r0 + i) * kTile + lane] : 0;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = on[i] ? sp[q[i]] : 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + i;
            const uint32_t yr = __shfl_sync(ALL, yl, r);
            if (g[i] != q[i]) q[i] = ccl_lroot(sp, g[i], limit, err);
            const uint32_t out = on[i] ? (yr - (uint32_t)(r - q[i] / kTile)) * cols + x0 + (uint32_t)(q[i] % kTile) + 1u : 0u;
            if (xin && r < nrows) lab[at + (size_t)r * cols] = out;
        }
    }
}

// ---- merge across tile borders: the pairs whose earlier neighbour lies in
// another tile (W, NW of the left column; NW, N, NE of the top row; NE of the
// right column) are hooked in the global parents.  One warp per tile, whose three
// sides are read together; or one per tile and side (gridDim.y = 3) where the tiles
// alone would not fill the device.  Within a warp, pairs whose current parents are
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
    k_ccl_border(const T *__restrict__ img, uint32_t *lab, uint32_t rows, uint32_t cols, uint32_t tiles_x, uint32_t tiles,
                 uint32_t slice_rows, int64_t limit, int *err) {
    const uint32_t tile = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= tiles) return;
    const int lane = threadIdx.x & 31;
    const uint32_t y0 = tile / tiles_x * kTile, x0 = tile % tiles_x * kTile;
    // lane = column of the top row, or row of the left or the right column
    bool fg[3];
    T v[3];
    bool any = false;
#pragma unroll
    for (int side = 0; side < 3; ++side) {
        const uint32_t y = y0 + (side == 0 ? 0 : lane), x = x0 + (side == 0 ? lane : side == 1 ? 0 : kTile - 1);
        const bool on = (gridDim.y == 1 || side == (int)blockIdx.y) && y < rows && x < cols && (side == 0 || lane > 0);
        v[side] = on ? img[(size_t)y * cols + x] : T(0);
        fg[side] = on && ccl_fg<T>(v[side]);
        any = any || fg[side];
    }
    if (!__any_sync(0xffffffffu, any)) return;
#pragma unroll
    for (int side = 0; side < 3; ++side) {
        if (!__any_sync(0xffffffffu, fg[side])) continue;
        const uint32_t y = y0 + (side == 0 ? 0 : lane), x = x0 + (side == 0 ? lane : side == 1 ? 0 : kTile - 1);
        const uint32_t yl = y % slice_rows;
        const size_t i = (size_t)y * cols + x, base = (size_t)(y - yl) * cols, u = i - cols;
        const bool up = fg[side] && yl != 0;
        if (side == 0) {
            ccl_hook_dedup(lab, fg[side] && lane == 0 && x > 0 && ccl_eq(img[i - 1], v[side]), base, i, i - 1, limit, err);
            ccl_hook_dedup(lab, up && x > 0 && ccl_eq(img[u - 1], v[side]), base, i, u - 1, limit, err);
            ccl_hook_dedup(lab, up && ccl_eq(img[u], v[side]), base, i, u, limit, err);
            ccl_hook_dedup(lab, up && x + 1 < cols && ccl_eq(img[u + 1], v[side]), base, i, u + 1, limit, err);
        } else if (side == 1) {
            ccl_hook_dedup(lab, fg[side] && x > 0 && ccl_eq(img[i - 1], v[side]), base, i, i - 1, limit, err);
            ccl_hook_dedup(lab, up && x > 0 && ccl_eq(img[u - 1], v[side]), base, i, u - 1, limit, err);
        } else {
            ccl_hook_dedup(lab, up && x + 1 < cols && ccl_eq(img[u + 1], v[side]), base, i, u + 1, limit, err);
        }
    }
}

// Every foreground pixel takes its root's label.  The foreground is found in the
// smaller array: the image where a pixel is one byte (K = 16 per thread, or 4 where 16
// would leave most of the device without a thread), else the labels (4 per thread);
// K-byte or 16-byte aligned, else K = 1.  A thread's pixels follow their parents
// together, so that the walks cost the latency of the deepest (one after the other
// they took 15 us of a 100^2 image's 40); a run of equal labels walks once.
template <class T, int K>
__global__ void __launch_bounds__(256)
    k_ccl_flatten(const T *__restrict__ img, uint32_t *lab, int64_t n, int64_t slice_n, int64_t limit, int *err) {
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * K;
    if (i >= n) return;
    uint32_t l[K], cur[K];
    const bool whole = i + K <= n;
    if constexpr (K > 1 && sizeof(T) == 1) {
        uint32_t word[K / 4] = {};
        if (whole) {
            if constexpr (K == 16) {
                const uint4 q = __ldg(reinterpret_cast<const uint4 *>(img + i));
                word[0] = q.x; word[1] = q.y; word[2] = q.z; word[3] = q.w;
                if ((q.x | q.y | q.z | q.w) == 0) return;
            } else {
                word[0] = __ldg(reinterpret_cast<const uint32_t *>(img + i));
                if (word[0] == 0) return;
            }
        }
        const bool aligned = ((uintptr_t)lab & 15) == 0;
#pragma unroll
        for (int w = 0; w < K / 4; ++w) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (word[w] != 0) {
                const uint32_t *at = lab + i + 4 * w;
                if (aligned) v = *reinterpret_cast<const uint4 *>(at);
                else v = make_uint4(at[0], at[1], at[2], at[3]);
            }
            l[4 * w] = v.x; l[4 * w + 1] = v.y; l[4 * w + 2] = v.z; l[4 * w + 3] = v.w;
        }
    } else if constexpr (K > 1) {
        if (whole) {
            const uint4 v = *reinterpret_cast<const uint4 *>(lab + i);
            if ((v.x | v.y | v.z | v.w) == 0) return;
            l[0] = v.x; l[1] = v.y; l[2] = v.z; l[3] = v.w;
        }
    } else {
        l[0] = lab[i];
    }
    const int64_t base = (i / slice_n) * slice_n;
    if (!whole || i + K > base + slice_n) {   // the array's end, or two slices
        for (int64_t j = i; j < i + K && j < n; ++j) {
            const uint32_t v = lab[j];
            if (v != 0) lab[j] = ccl_root(lab + (j / slice_n) * slice_n - 1, v, limit, err);
        }
        return;
    }
    // node of the slice -> its parent (roots do not change here, and whatever a pixel held
    // before is an ancestor of it, so reads may come from L1)
    uint32_t *p = lab + base - 1;
#pragma unroll
    for (int k = 0; k < K; ++k) cur[k] = l[k];
    bool walking = true;
    for (int64_t it = 0; walking; ++it) {
        if (it > limit) { atomicExch(err, 1); break; }
        walking = false;
        uint32_t next[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
            next[k] = l[k] != 0 && (k == 0 || l[k] != l[k > 0 ? k - 1 : 0]) ? __ldca(p + cur[k]) : cur[k];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            walking = walking || next[k] < cur[k];
            cur[k] = next[k];
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (k > 0 && l[k] == l[k > 0 ? k - 1 : 0]) cur[k] = cur[k > 0 ? k - 1 : 0];
        if (cur[k] != l[k]) lab[i + k] = cur[k];
    }
}

template <class T>
static cudaError_t ccl_run(const T *img, uint32_t *lab, int64_t rows, int64_t cols, int64_t slice_rows, int64_t limit,
                           int *err, cudaStream_t s, int64_t *launches) {
    const int64_t n = rows * cols;
    // (fewer than 2^32 pixels: fewer than 2^28 tiles)
    const uint32_t tiles_x = (uint32_t)((cols + kTile - 1) / kTile), tiles = tiles_x * (uint32_t)((rows + kTile - 1) / kTile);
    constexpr int W = CclLocal<T>::WARPS;
    k_ccl_local<T><<<(unsigned)((tiles + W - 1) / W), W * 32, 0, s>>>(img, lab, (uint32_t)rows, (uint32_t)cols,
                                                                     tiles_x, tiles, (uint32_t)slice_rows,
                                                                     limit, err);
    k_ccl_border<T><<<dim3((tiles + 7) / 8, tiles <= 3072 ? 3 : 1), 256, 0, s>>>(img, lab, (uint32_t)rows, (uint32_t)cols,
                                                                tiles_x, tiles, (uint32_t)slice_rows, limit,
                                                                err);
    const int64_t slice_n = slice_rows * cols;
    const auto flatten = [&](auto k) {
        constexpr int K = decltype(k)::value;
        k_ccl_flatten<T, K><<<(unsigned)((n + 256 * K - 1) / (256 * K)), 256, 0, s>>>(img, lab, n, slice_n, limit, err);
    };
    const uintptr_t at = sizeof(T) == 1 ? (uintptr_t)img : (uintptr_t)lab;
    if constexpr (sizeof(T) == 1) {
        if (n >= (1 << 20) && at % 16 == 0) flatten(std::integral_constant<int, 16>{});
        else if (at % 4 == 0) flatten(std::integral_constant<int, 4>{});
        else flatten(std::integral_constant<int, 1>{});
    } else {
        if (at % 16 == 0) flatten(std::integral_constant<int, 4>{});
        else flatten(std::integral_constant<int, 1>{});
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
// An update that the box already covers is left out: the values only grow outwards, so
// a value read earlier is as good (a component's pixels all update one box, and the
// atomics on it ran one after the other: 2048^2 of ones 11 ms pixel by pixel).
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
        const int4 now = __ldcg(reinterpret_cast<const int4 *>(b));
        if (slow < now.x) atomicMin(b + 0, slow);
        if (fast + k < now.y) atomicMin(b + 1, fast + k);
        if (slow > now.z) atomicMax(b + 2, slow);
        if (fast + e > now.w) atomicMax(b + 3, fast + e);
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
// counts; a block without roots is done at once.  Adjacent threads write adjacent
// roots (with 32 elements per thread, one after the other, dense roots cost more than
// the pass over the labels).
__global__ void __launch_bounds__(kRootThreads)
    k_roots_write(const uint32_t *__restrict__ lab, int64_t n, int64_t slice_n, const unsigned *offsets, int64_t nb,
                  const unsigned long long *total, long long *out, int64_t cap, unsigned *rank) {
    constexpr int WORDS = kRootTile / 32;
    __shared__ unsigned roots[WORDS], before[WORDS];   // one bit per element of the block; roots before its word
    __shared__ unsigned warp_sum[WORDS / 32];
    const unsigned first = offsets[blockIdx.x];
    const unsigned last = (int64_t)blockIdx.x + 1 < nb ? offsets[blockIdx.x + 1] : (unsigned)*total;
    if (first == last) return;
    if (threadIdx.x < WORDS) roots[threadIdx.x] = 0;
    __syncthreads();
    block_labels(lab, n, slice_n, [&](int j, uint32_t, bool root) {
        if (root) atomicOr(&roots[j >> 5], 1u << (j & 31));
    });
    __syncthreads();
    unsigned c = 0, incl = 0;
    if (threadIdx.x < WORDS) {   // (whole warps)
        c = incl = __popc(roots[threadIdx.x]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if ((threadIdx.x & 31) >= o) incl += u;
        }
        if ((threadIdx.x & 31) == 31) warp_sum[threadIdx.x >> 5] = incl;
    }
    __syncthreads();
    if (threadIdx.x < WORDS) {
        unsigned pre = first + incl - c;
        for (unsigned w = 0; w < threadIdx.x >> 5; ++w) pre += warp_sum[w];
        before[threadIdx.x] = pre;
    }
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRootTile;
    for (int j = threadIdx.x; j < kRootTile; j += kRootThreads) {
        const unsigned m = roots[j >> 5], bit = 1u << (j & 31);
        if (!(m & bit)) continue;
        const unsigned pre = before[j >> 5] + __popc(m & (bit - 1));
        if ((int64_t)pre < cap && out) out[pre] = (long long)(base + j + 1);
        if (rank) rank[base + j] = pre;
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

// Boxes of the roots of rank < count (their ranks are in `rank`, see k_roots_write); 16-byte aligned.
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
