// Kernel (c): tree links from the per-line depth sequence.
//
//   parent[i]       nearest previous content line with a smaller depth (PSV)
//   subtree_end[i]  nearest next content line with depth <= depth[i], else L
//   first_child[i]  next content line j if depth[j] > depth[i], else NONE
//   next_sibling[i] j = subtree_end[i] when parent[j] == parent[i], else NONE
// Blank lines: parent NONE, subtree_end i+1, no children, no sibling.
// Semantics: crates/oneline-core/src/links.rs:52-82 (sequential stack) and
// crates/oneline-simd/src/links.rs:135-180; first_child / next_sibling are
// derived from those links.
//
// Fast path (every content line has depth < 32; D = max depth + 1 levels),
// three kernels over tiles of 4096 lines (256 threads x 16 consecutive lines;
// of 1024 lines, 4 a thread, where that leaves at most kTreeFewTiles tiles: a
// thread's lines are a serial chain). With at most kTreeFewTiles tiles the
// second kernel is left out and every block of the third one scans the tiles'
// summaries itself; a single tile needs the third one alone:
//   summary : per tile and level k, the last and the first line of depth k;
//   scan    : per level, the exclusive prefix max (last line before the tile)
//             and suffix min (first line after it) over the tiles;
//   resolve : per level, the same scans over the threads of the tile give
//             every thread the last line of each depth before its run and the
//             first line of each depth after it. From these it rebuilds the
//             ancestor stack as a 32-bit level mask and walks its 16 lines
//             forward (parent in O(1) per line, the parent's depth kept in
//             registers), then the stack of following lines and walks backward
//             (subtree_end, next content line = first_child candidate, and
//             next_sibling: j = subtree_end[i] shares i's parent exactly when i
//             has no parent or its parent is shallower than j).
// Replaces crates/oneline-gpu/src/tree.wgsl:128-375 (seven passes).
//
// Any-depth path: each line searches left (strictly smaller) and right (smaller
// or equal), by halving windows of minima in shared memory inside its 1024
// lines, and through a 32-ary min tree in device memory past them.
#include <cuda_runtime.h>

#include "ol_common.cuh"
#include "ol_kernels.h"

namespace ol {

constexpr uint32_t TR_THREADS = 256;
static_assert(TR_THREADS * 16 == kTreeTile && TR_THREADS * 4 == kTreeSmallTile, "tree tiles");

__device__ __forceinline__ uint32_t mask_below(uint32_t d) { return d >= 32 ? 0xFFFFFFFFu : ((1u << d) - 1u); }
__device__ __forceinline__ uint32_t mask_le(uint32_t d) { return d >= 31 ? 0xFFFFFFFFu : ((2u << d) - 1u); }

// The RUN lines (4 or 16) of thread `tid` of tile `tile`: the level of each, or
// 0xFF for a blank line, four per word. Depths >= levels cannot reach this path
// (the host picks the any-depth path for them).
template <uint32_t RUN>
struct Run {
    uint32_t lv[RUN / 4];
    uint64_t first;
};

template <uint32_t RUN>
__device__ __forceinline__ Run<RUN> load_run(const TreeArgs &a, uint32_t tile, uint32_t tid) {
    Run<RUN> r;
    r.first = ((uint64_t)tile * TR_THREADS + tid) * RUN;
    uint32_t kd[RUN / 4], dp[RUN / 4];
    if (r.first + RUN <= a.L) {
        if (RUN == 16) {
            *reinterpret_cast<uint4 *>(kd) = *reinterpret_cast<const uint4 *>(a.kinds + r.first);
            *reinterpret_cast<uint4 *>(dp) = *reinterpret_cast<const uint4 *>(a.depth8 + r.first);
        } else {
            kd[0] = *reinterpret_cast<const uint32_t *>(a.kinds + r.first);
            dp[0] = *reinterpret_cast<const uint32_t *>(a.depth8 + r.first);
        }
    } else {
#pragma unroll
        for (uint32_t w = 0; w < RUN / 4; w++) {
            kd[w] = dp[w] = 0;  // past the end: blank
            for (uint32_t i = 0; i < 4; i++) {
                if (r.first + 4 * w + i >= a.L) break;
                kd[w] |= (uint32_t)a.kinds[r.first + 4 * w + i] << (8 * i);
                dp[w] |= (uint32_t)a.depth8[r.first + 4 * w + i] << (8 * i);
            }
        }
    }
    static_assert(KIND_BLANK == 0, "a blank line's kind byte is zero");
    const uint32_t top = (a.levels - 1) * 0x01010101u;
#pragma unroll
    for (uint32_t w = 0; w < RUN / 4; w++) r.lv[w] = __vminu4(dp[w], top) | ((zero_bytes(kd[w]) >> 7) * 0xFFu);
    return r;
}

template <uint32_t RUN>
__device__ __forceinline__ uint32_t level_of(const Run<RUN> &r, int i) {
    return (r.lv[i >> 2] >> (8 * (i & 3))) & 0xFFu;
}

// Dynamic shared memory of the summary and resolve kernels: D levels x 256
// threads of "last line + 1" (forward) followed by the same of "first line"
// (backward).
struct TreeSmem {
    uint32_t *fa, *fb;
    uint32_t D;
    __device__ uint32_t &a(uint32_t k, uint32_t t) { return fa[k * TR_THREADS + t]; }
    __device__ uint32_t &b(uint32_t k, uint32_t t) { return fb[k * TR_THREADS + t]; }
};
extern __shared__ __align__(16) uint32_t tree_dyn_smem[];

__device__ __forceinline__ TreeSmem tree_smem(uint32_t D) {
    TreeSmem s;
    s.fa = tree_dyn_smem;
    s.fb = tree_dyn_smem + D * TR_THREADS;
    s.D = D;
    return s;
}

// Pass 1: per tile and level, the last line (+1) and the first line of that depth.
template <uint32_t RUN>
__global__ void __launch_bounds__(TR_THREADS) tree_summary_kernel(TreeArgs a) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
    const uint32_t D = a.levels;
    TreeSmem sm = tree_smem(D);
    const Run<RUN> r = load_run<RUN>(a, tile, tid);
    for (uint32_t k = 0; k < D; k++) {
        sm.a(k, tid) = 0;
        sm.b(k, tid) = NONE;
    }
#pragma unroll
    for (int i = 0; i < (int)RUN; i++) {
        uint32_t d = level_of(r, i);
        if (d != 0xFF) sm.a(d, tid) = (uint32_t)(r.first + i + 1);
    }
#pragma unroll
    for (int i = RUN - 1; i >= 0; i--) {
        uint32_t d = level_of(r, i);
        if (d != 0xFF) sm.b(d, tid) = (uint32_t)(r.first + i);
    }
    __syncthreads();
    for (uint32_t k = warp; k < D; k += 8) {
        uint32_t mx = 0, mn = NONE;
#pragma unroll
        for (int j = 0; j < TR_THREADS / 32; j++) {
            mx = max(mx, sm.a(k, j * 32 + lane));
            mn = min(mn, sm.b(k, j * 32 + lane));
        }
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        mn = __reduce_min_sync(0xFFFFFFFFu, mn);
        if (lane == 0) {
            a.tile_last[(size_t)tile * kTreeLevels + k] = mx;
            a.tile_first[(size_t)tile * kTreeLevels + k] = mn;
        }
    }
}

// Pass 2: for each level (one block per level), exclusive prefix max of
// tile_last and exclusive suffix min of tile_first over the tiles.
__global__ void __launch_bounds__(1024) tree_scan_kernel(TreeArgs a) {
    __shared__ uint32_t s_max[32], s_min[32];
    const uint32_t k = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t T = a.n_tiles;
    const uint32_t per = (T + 1023) / 1024;
    const uint32_t lo = min(T, tid * per), hi = min(T, lo + per);
    // Up to kHeld tiles per thread (documents of up to 2^25 lines) are read
    // once, all loads in flight together, and kept in registers for the walks
    // below.
    constexpr uint32_t kHeld = 8;
    const bool held = per <= kHeld;  // uniform
    uint32_t vl[kHeld], vf[kHeld];
    uint32_t mx = 0, mn = NONE;
    if (held) {
#pragma unroll
        for (uint32_t i = 0; i < kHeld; i++) {
            const bool in = lo + i < hi;
            vl[i] = in ? a.tile_last[(size_t)(lo + i) * kTreeLevels + k] : 0u;
            vf[i] = in ? a.tile_first[(size_t)(lo + i) * kTreeLevels + k] : NONE;
        }
#pragma unroll
        for (uint32_t i = 0; i < kHeld; i++) {
            mx = max(mx, vl[i]);
            mn = min(mn, vf[i]);
        }
    } else {
        for (uint32_t t = lo; t < hi; t++) {
            mx = max(mx, a.tile_last[(size_t)t * kTreeLevels + k]);
            mn = min(mn, a.tile_first[(size_t)t * kTreeLevels + k]);
        }
    }
    // inclusive scans over threads: max forward, min backward
    uint32_t imx = mx, imn = mn;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t1 = __shfl_up_sync(0xFFFFFFFFu, imx, o);
        uint32_t t2 = __shfl_down_sync(0xFFFFFFFFu, imn, o);
        if ((int)lane >= o) imx = max(imx, t1);
        if (lane + o < 32) imn = min(imn, t2);
    }
    if (lane == 31) s_max[warp] = imx;
    if (lane == 0) s_min[warp] = imn;
    __syncthreads();
    uint32_t before = 0, after = NONE;  // warps before / after mine
    for (uint32_t w = 0; w < warp; w++) before = max(before, s_max[w]);
    for (uint32_t w = warp + 1; w < 32; w++) after = min(after, s_min[w]);
    // every lane takes part in both shuffles; lanes 0 / 31 discard the result
    const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, imx, 1);
    const uint32_t down = __shfl_down_sync(0xFFFFFFFFu, imn, 1);
    uint32_t ex_mx = max(before, lane == 0 ? 0u : up);
    uint32_t ex_mn = min(after, lane == 31 ? NONE : down);
    // walk my tiles: forward exclusive max, then backward exclusive min
    if (held) {
        uint32_t run = ex_mx;
#pragma unroll
        for (uint32_t i = 0; i < kHeld; i++) {
            if (lo + i < hi) a.in_last[(size_t)(lo + i) * kTreeLevels + k] = run;
            run = max(run, vl[i]);
        }
        run = ex_mn;
#pragma unroll
        for (int i = kHeld - 1; i >= 0; i--) {
            if (lo + i < hi) a.in_first[(size_t)(lo + i) * kTreeLevels + k] = run;
            run = min(run, vf[i]);
        }
        return;
    }
    uint32_t run = ex_mx;
    for (uint32_t t = lo; t < hi; t++) {
        a.in_last[(size_t)t * kTreeLevels + k] = run;
        run = max(run, a.tile_last[(size_t)t * kTreeLevels + k]);
    }
    run = ex_mn;
    for (uint32_t t = hi; t-- > lo;) {
        a.in_first[(size_t)t * kTreeLevels + k] = run;
        run = min(run, a.tile_first[(size_t)t * kTreeLevels + k]);
    }
}

// v to p[at .. at + W), W lines of which those below L exist; at is a multiple of
// W and the arrays are 256-byte aligned.
template <uint32_t W>
__device__ __forceinline__ void put_words(uint32_t *p, uint64_t at, uint32_t L, const uint32_t (&v)[W]) {
    if (at + W <= L) {
        if constexpr (W == 8)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + at), "r"(v[0]), "r"(v[1]),
                         "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                         : "memory");
        else
            *reinterpret_cast<uint4 *>(p + at) = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
        for (uint32_t q = 0; q < W; q++)
            if (at + q < L) p[at + q] = v[q];
    }
}

// Pass 3: every thread rebuilds the ancestor stack before its 16 lines and
// the stack of the lines after them, walks forward for parent (and the
// parent's depth, kept in registers) and backward for subtree_end,
// first_child and next_sibling.
// What bounds it is the serial chain of a thread's lines, and the stores: with 16
// bytes at a time every 32-byte sector was written in two halves; whole sectors
// at a time, and four blocks an SM without spills instead of five, took 72
// against 93 us for 11 M lines.
// FEW: at most kTreeFewTiles tiles, whose summaries are scanned here.
template <uint32_t RUN, bool FEW>
__global__ void __launch_bounds__(TR_THREADS, 4) tree_resolve_kernel(TreeArgs a) {
    constexpr uint32_t W = RUN < 8 ? RUN : 8;  // lines stored at a time
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
    const uint32_t D = a.levels;
    TreeSmem sm = tree_smem(D);
    const Run<RUN> r = load_run<RUN>(a, tile, tid);
    for (uint32_t k = 0; k < D; k++) {
        sm.a(k, tid) = 0;
        sm.b(k, tid) = NONE;
    }
#pragma unroll
    for (int i = 0; i < (int)RUN; i++) {
        uint32_t d = level_of(r, i);
        if (d != 0xFF) sm.a(d, tid) = (uint32_t)(r.first + i + 1);
    }
#pragma unroll
    for (int i = RUN - 1; i >= 0; i--) {
        uint32_t d = level_of(r, i);
        if (d != 0xFF) sm.b(d, tid) = (uint32_t)(r.first + i);
    }
    __syncthreads();
    // Per level: exclusive max over the threads before mine (seeded with the
    // tiles before this one) and exclusive min over the threads after mine
    // (seeded with the tiles after this one).
    // One warp per level; lane L holds the entries of threads 8L .. 8L+7 (two
    // 16-byte loads), reduces them, and one warp scan of the 32 lane values
    // gives each lane its seed.
    for (uint32_t k = warp; k < D; k += 8) {
        uint32_t in_last, in_first;
        if (!FEW) {
            in_last = a.in_last[(size_t)tile * kTreeLevels + k];
            in_first = a.in_first[(size_t)tile * kTreeLevels + k];
        } else {  // (a single tile has no summaries)
            in_last = 0;
            in_first = NONE;
#pragma unroll
            for (uint32_t i = 0; i < kTreeFewTiles / 32; i++) {
                const uint32_t t = i * 32 + lane;
                if (t < tile) in_last = max(in_last, a.tile_last[(size_t)t * kTreeLevels + k]);
                if (t > tile && t < a.n_tiles) in_first = min(in_first, a.tile_first[(size_t)t * kTreeLevels + k]);
            }
            in_last = __reduce_max_sync(0xFFFFFFFFu, in_last);
            in_first = __reduce_min_sync(0xFFFFFFFFu, in_first);
        }
        uint4 *ra = reinterpret_cast<uint4 *>(&sm.a(k, 8 * lane));
        uint4 *rb = reinterpret_cast<uint4 *>(&sm.b(k, 8 * lane));
        {
            const uint4 q0 = ra[0], q1 = ra[1];
            uint32_t v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint32_t inc = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) inc = max(inc, v[i]);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if ((int)lane >= o) inc = max(inc, t);
            }
            const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, inc, 1);
            uint32_t run = max(in_last, lane == 0 ? 0u : prev);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t t = v[i];
                v[i] = run;
                run = max(run, t);
            }
            ra[0] = make_uint4(v[0], v[1], v[2], v[3]);
            ra[1] = make_uint4(v[4], v[5], v[6], v[7]);
        }
        {
            const uint4 q0 = rb[0], q1 = rb[1];
            uint32_t v[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint32_t inc = NONE;
#pragma unroll
            for (int i = 0; i < 8; i++) inc = min(inc, v[i]);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_down_sync(0xFFFFFFFFu, inc, o);
                if (lane + o < 32) inc = min(inc, t);
            }
            const uint32_t next = __shfl_down_sync(0xFFFFFFFFu, inc, 1);
            uint32_t run = min(in_first, lane == 31 ? NONE : next);
#pragma unroll
            for (int i = 7; i >= 0; i--) {
                const uint32_t t = v[i];
                v[i] = run;
                run = min(run, t);
            }
            rb[0] = make_uint4(v[0], v[1], v[2], v[3]);
            rb[1] = make_uint4(v[4], v[5], v[6], v[7]);
        }
    }
    __syncthreads();

    // Forward: level k is on the ancestor stack iff its last line comes after
    // every line of smaller depth.
    uint32_t M = 0, runmax = 0;
    for (uint32_t k = 0; k < D; k++) {
        uint32_t v = sm.a(k, tid);
        if (v > runmax) {
            M |= 1u << k;
            runmax = v;
        }
    }
    uint32_t pdw[RUN / 4];  // parent depth bytes, 0xFF = none
#pragma unroll
    for (uint32_t w = 0; w < RUN / 4; w++) pdw[w] = 0xFFFFFFFFu;
    uint32_t par[W];
#pragma unroll
    for (int i = 0; i < (int)RUN; i++) {
        uint32_t d = level_of(r, i);
        uint32_t pv = NONE;
        if (d != 0xFF) {
            uint32_t low = M & mask_below(d);
            if (low) {
                uint32_t top = 31 - __clz(low);
                pv = sm.a(top, tid) - 1;
                pdw[i >> 2] = (pdw[i >> 2] & ~(0xFFu << (8 * (i & 3)))) | (top << (8 * (i & 3)));
            }
            M = low | (1u << d);
            sm.a(d, tid) = (uint32_t)(r.first + i + 1);
        }
        par[i % W] = pv;
        if (i % W == W - 1) put_words<W>(a.parent, r.first + i + 1 - W, a.L, par);
    }

    // Backward: level k is on the stack of following lines iff its first line
    // comes before every line of smaller depth; the highest level on it is the
    // next content line.
    M = 0;
    uint32_t runmin = NONE;
    for (uint32_t k = 0; k < D; k++) {
        uint32_t v = sm.b(k, tid);
        if (v < runmin) {
            M |= 1u << k;
            runmin = v;
        }
    }
    uint32_t se[W], fc[W], ns[W];
#pragma unroll
    for (int i = RUN - 1; i >= 0; i--) {
        uint64_t line = r.first + i;
        uint32_t d = level_of(r, i);
        uint32_t vse = (uint32_t)(line + 1), vfc = NONE, vns = NONE;
        if (d != 0xFF) {
            if (M) {
                uint32_t nb = 31 - __clz(M);
                if (nb > d) vfc = sm.b(nb, tid);
            }
            uint32_t le = M & mask_le(d);
            if (le) {
                uint32_t top = 31 - __clz(le);
                uint32_t j = sm.b(top, tid);
                vse = j;
                uint32_t pd = (pdw[i >> 2] >> (8 * (i & 3))) & 0xFF;
                if (pd == 0xFF || pd < top) vns = j;
            } else {
                vse = a.L;
            }
            M = (M & mask_below(d)) | (1u << d);
            sm.b(d, tid) = (uint32_t)line;
        }
        se[i % W] = vse;
        fc[i % W] = vfc;
        ns[i % W] = vns;
        if (i % W == 0) {
            if (a.subtree_end) put_words<W>(a.subtree_end, line, a.L, se);
            put_words<W>(a.first_child, line, a.L, fc);
            put_words<W>(a.next_sibling, line, a.L, ns);
        }
    }
}

uint32_t tree_tile_lines(uint32_t L) { return L <= kTreeFewTiles * kTreeSmallTile ? kTreeSmallTile : kTreeTile; }

template <uint32_t RUN, bool FEW>
static cudaError_t launch_tree_run(const TreeArgs &a, cudaStream_t st) {
    size_t smem = (size_t)a.levels * TR_THREADS * 4 * 2;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(tree_summary_kernel<RUN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tree_resolve_kernel<RUN, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    if (a.n_tiles > 1) {
        tree_summary_kernel<RUN><<<a.n_tiles, TR_THREADS, smem, st>>>(a); OL_LAUNCHED();
    }
    if (!FEW) {
        tree_scan_kernel<<<a.levels, 1024, 0, st>>>(a); OL_LAUNCHED();
    }
    tree_resolve_kernel<RUN, FEW><<<a.n_tiles, TR_THREADS, smem, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

// 1 MiB (21,000 lines, 17 levels) took 21.5 us in three kernels of 16 lines a
// thread: 10.9 us in two of 4.
cudaError_t launch_tree_fast(const TreeArgs &a, cudaStream_t st) {
    if (a.n_tiles == 0) return cudaSuccess;
    if (tree_tile_lines(a.L) == kTreeSmallTile) return launch_tree_run<4, true>(a, st);
    return a.n_tiles <= kTreeFewTiles ? launch_tree_run<16, true>(a, st) : launch_tree_run<16, false>(a, st);
}

// ------------------------------------------------------------ any depth ----
//
// What bounds it is latency: 400,000 lines (depths up to 60) took 92 us in seven
// kernels that searched the tree one load after the other, 34 us in three now.

constexpr uint32_t TD_LINES = 1024;  // lines (and threads) of a block: 32 chunks of 32

// A line's depth, or NONE for a blank line.
__device__ __forceinline__ uint32_t deep_key(const TreeDeepArgs &a, uint32_t i) {
    if (a.keys) return __ldg(a.keys + i);
    const uint32_t kind = __ldg(a.kinds + i), depth = __ldg(a.depth8 + i);
    return kind == KIND_BLANK ? NONE : depth;
}

// Minima of every 32 and every 1024 lines (levels 0 and 1).
__global__ void __launch_bounds__(TD_LINES) deep_min_kernel(TreeDeepArgs a) {
    __shared__ uint32_t chunk_min[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t i = (uint64_t)blockIdx.x * TD_LINES + tid;
    uint32_t m = __reduce_min_sync(0xFFFFFFFFu, i < a.L ? deep_key(a, (uint32_t)i) : NONE);
    if (lane == 0) {
        chunk_min[warp] = m;
        if (i < a.L) a.levels[0][i >> 5] = m;
    }
    __syncthreads();
    if (warp == 0) {
        m = __reduce_min_sync(0xFFFFFFFFu, chunk_min[lane]);
        if (lane == 0) a.levels[1][blockIdx.x] = m;
    }
}

// The levels above, one block.
__global__ void __launch_bounds__(TD_LINES) deep_top_kernel(TreeDeepArgs a) {
    for (uint32_t l = 2; l < a.n_levels; l++) {
        const uint32_t *src = a.levels[l - 1];
        for (uint32_t g = threadIdx.x; g < a.level_len[l]; g += TD_LINES) {
            uint32_t v = NONE;
#pragma unroll 8
            for (uint32_t c = 0; c < 32; c++)
                if (g * 32 + c < a.level_len[l - 1]) v = min(v, src[g * 32 + c]);
            a.levels[l][g] = v;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }

// Entry i of level l (lines: -1), or NONE past its end.
__device__ __forceinline__ uint32_t deep_value(const TreeDeepArgs &a, int32_t l, uint64_t i) {
    if (l < 0) return i < a.L ? deep_key(a, (uint32_t)i) : NONE;
    return i < a.level_len[l] ? a.levels[l][i] : NONE;
}

// Nearest line before block `pos` of 1024 lines with a depth < d, or NONE. The
// whole warp searches: 32 entries of a level at a time, up to the first level
// that has one, and down from there.
__device__ __forceinline__ uint32_t deep_prev_out(const TreeDeepArgs &a, uint32_t pos, uint32_t d) {
    const uint32_t lane = threadIdx.x & 31;
    for (int32_t lv = 1; lv < (int32_t)a.n_levels; lv++, pos >>= 5) {
        const uint32_t g = pos & ~31u;
        uint32_t m = __ballot_sync(0xFFFFFFFFu, g + lane < pos && a.levels[lv][g + lane] < d);
        if (!m) continue;
        uint32_t node = g + 31 - __clz(m);
        for (int32_t l = lv - 1; l >= -1; l--) {
            m = __ballot_sync(0xFFFFFFFFu, deep_value(a, l, (uint64_t)node * 32 + lane) < d);
            node = node * 32 + 31 - __clz(m);
        }
        return node;
    }
    return NONE;
}

// Nearest line after block `pos` of 1024 lines with a depth <= d, or NONE.
__device__ __forceinline__ uint32_t deep_next_out(const TreeDeepArgs &a, uint32_t pos, uint32_t d) {
    const uint32_t lane = threadIdx.x & 31;
    for (int32_t lv = 1; lv < (int32_t)a.n_levels; lv++, pos >>= 5) {
        const uint32_t g = pos & ~31u;
        uint32_t m = __ballot_sync(0xFFFFFFFFu, g + lane > pos && deep_value(a, lv, (uint64_t)g + lane) <= d);
        if (!m) continue;
        uint32_t node = g + __ffs(m) - 1;
        for (int32_t l = lv - 1; l >= -1; l--) {
            m = __ballot_sync(0xFFFFFFFFu, deep_value(a, l, (uint64_t)node * 32 + lane) <= d);
            node = node * 32 + __ffs(m) - 1;
        }
        return node;
    }
    return NONE;
}

// win[k][i]: the minimum of entries i .. i + 2^k - 1 of i's 32 (of those there
// are). The last entry before `pos` (0..32) below d, or NONE.
template <class Win>
__device__ __forceinline__ uint32_t win_prev(const Win &win, uint32_t base, uint32_t pos, uint32_t d) {
#pragma unroll
    for (int k = 4; k >= 0; k--)
        if (pos >= (1u << k) && win[k][base + pos - (1u << k)] >= d) pos -= 1u << k;
    // 32 entries are one more than the steps cover: the first one is left
    return pos && win[0][base + pos - 1] < d ? base + pos - 1 : NONE;
}

// The first entry from `pos` (0..32) on at most d, or NONE.
template <class Win>
__device__ __forceinline__ uint32_t win_next(const Win &win, uint32_t base, uint32_t pos, uint32_t d) {
#pragma unroll
    for (int k = 4; k >= 0; k--)
        if (pos + (1u << k) <= 32 && win[k][base + pos] > d) pos += 1u << k;
    return pos < 32 && win[0][base + pos] <= d ? base + pos : NONE;
}

__global__ void __launch_bounds__(TD_LINES) deep_links_kernel(TreeDeepArgs a) {
    __shared__ uint32_t win[5][TD_LINES];  // over the lines of each chunk
    __shared__ uint32_t top[5][32];        // over the chunks
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, base = tid & ~31u;
    const uint32_t line0 = blockIdx.x * TD_LINES;
    const uint64_t i = (uint64_t)line0 + tid;
    const uint32_t d = i < a.L ? deep_key(a, (uint32_t)i) : NONE;
    uint32_t m = d;
    win[0][tid] = m;
#pragma unroll
    for (int k = 1; k < 5; k++) {
        const uint32_t t = __shfl_down_sync(0xFFFFFFFFu, m, 1 << (k - 1));
        if (lane + (1u << (k - 1)) < 32) m = umin(m, t);
        win[k][tid] = m;
    }
    m = __reduce_min_sync(0xFFFFFFFFu, d);
    if (lane == 0) top[0][warp] = m;
    __syncthreads();
    if (warp == 0) {
        m = top[0][lane];
#pragma unroll
        for (int k = 1; k < 5; k++) {
            const uint32_t t = __shfl_down_sync(0xFFFFFFFFu, m, 1 << (k - 1));
            if (lane + (1u << (k - 1)) < 32) m = umin(m, t);
            top[k][lane] = m;
        }
    }
    __syncthreads();
    const bool line = d != NONE;  // blank lines and lanes past the end only help
    // A search that leaves the block depends on the depth alone: one for all lanes
    // of a warp that have it.
    auto outside = [&](bool need, uint32_t least, bool after, uint32_t &result) {
        for (uint32_t u; (u = __ballot_sync(0xFFFFFFFFu, need)) != 0;) {
            const uint32_t q = __shfl_sync(0xFFFFFFFFu, least, __ffs(u) - 1);
            const uint32_t r = after ? deep_next_out(a, blockIdx.x, q) : deep_prev_out(a, blockIdx.x, q);
            if (need && least == q) {
                result = r;
                need = false;
            }
        }
    };
    auto next = [&](uint32_t least) -> uint32_t {  // the next line with a depth <= least
        uint32_t j = win_next(win, base, lane + 1, least);
        if (j == NONE) {
            const uint32_t c = win_next(top, 0, warp + 1, least);
            if (c != NONE) j = win_next(win, c * 32, 0, least);
        }
        uint32_t r = j != NONE ? line0 + j : NONE;
        outside(line && j == NONE, least, true, r);
        return r;
    };
    // parent: the line before with a smaller depth
    uint32_t j = win_prev(win, base, lane, d);
    if (j == NONE) {
        const uint32_t c = win_prev(top, 0, warp, d);
        if (c != NONE) j = win_prev(win, c * 32, 32, d);
    }
    uint32_t p = j != NONE ? line0 + j : NONE;
    outside(line && d != 0 && j == NONE, d, false, p);
    const uint32_t e = next(d), c = next(NONE - 1);  // the subtree's end; the next content line
    if (i >= a.L) return;
    if (!line) {
        a.parent[i] = a.first_child[i] = a.next_sibling[i] = NONE;
        if (a.subtree_end) a.subtree_end[i] = (uint32_t)i + 1;
        return;
    }
    auto key_of = [&](uint32_t x) { return x - line0 < TD_LINES ? win[0][x - line0] : deep_key(a, x); };
    a.parent[i] = p;
    if (a.subtree_end) a.subtree_end[i] = e == NONE ? a.L : e;
    a.first_child[i] = c != NONE && c != e ? c : NONE;  // deeper than this line: before the end
    // the end has the same parent when it is deeper than this line's
    a.next_sibling[i] = e != NONE && (p == NONE || key_of(p) < key_of(e)) ? e : NONE;
}

cudaError_t launch_tree_deep(const TreeDeepArgs &a, cudaStream_t st) {
    if (a.L == 0) return cudaSuccess;
    const uint32_t blocks = (uint32_t)(((uint64_t)a.L + TD_LINES - 1) / TD_LINES);
    if (blocks > 1) {  // a single block searches its own lines only
        deep_min_kernel<<<blocks, TD_LINES, 0, st>>>(a); OL_LAUNCHED();
    }
    if (a.n_levels > 2) {
        deep_top_kernel<<<1, TD_LINES, 0, st>>>(a); OL_LAUNCHED();
    }
    deep_links_kernel<<<blocks, TD_LINES, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

}  // namespace ol
