// Node query filter: the lines of a range whose kind and depth match, in
// ascending order. Replaces filter_nodes / filter_fused
// (crates/oneline-gpu/src/shader.wgsl:136-193) and their slot atomics with a
// pass that marks and counts the matching lines of every block and one that
// writes them, so a truncated answer is the lowest max_out lines rather than an
// arbitrary subset. Between them the counts are scanned, by the writing blocks
// themselves when there are at most kQuerySelfScan of them.
//
// Filter semantics (shader.wgsl:152-160, query.rs:138-139): target_kind 0
// accepts every kind (so the reference cannot ask for Blank lines either), and
// target_depth 0xFFFFFFFF accepts every depth.
//
// A thread takes 16 lines: two 16-byte loads and byte compares instead of 16
// times two byte loads, once instead of in both passes. 5.5 M lines: 37 us in
// three kernels, 12 us in two.
#include <cuda_runtime.h>

#include "ol_common.cuh"
#include "ol_kernels.h"

namespace ol {

constexpr uint32_t QY_THREADS = 256;
constexpr uint32_t QY_PER_THREAD = 16;
constexpr uint32_t QY_LINES = QY_THREADS * QY_PER_THREAD;  // lines per block

uint32_t query_blocks(uint32_t lo, uint32_t hi) { return (uint32_t)(((uint64_t)hi - (lo & ~15u) + QY_LINES - 1) / QY_LINES); }
static_assert(kQueryMasks == QY_THREADS, "one mask a thread");

__device__ __forceinline__ bool query_match(const QueryArgs &a, uint32_t i) {
    uint32_t kind, depth8;
    if (a.nodes) {
        FlatNode nd = a.nodes[i];
        if (a.target_kind != 0 && nd.kind != a.target_kind) return false;
        return a.target_depth == NONE || nd.depth == a.target_depth;
    }
    kind = a.kinds[i];
    if (a.target_kind != 0 && kind != a.target_kind) return false;
    if (a.target_depth == NONE) return true;
    depth8 = a.depth8[i];
    if (depth8 < 255) return depth8 == a.target_depth;
    if (a.target_depth < 255) return false;
    // 255 or deeper: the exact depth from the text
    const uint32_t s = a.offsets[i];
    const uint32_t last_end = a.text[a.text_len - 1] == '\n' ? (uint32_t)(a.text_len - 1) : (uint32_t)a.text_len;
    const uint32_t e = i + 1 < a.lines ? a.offsets[i + 1] - 1 : last_end;
    FlatNode nd = classify_line(s, e, [&](uint32_t p) -> uint8_t { return __ldg(a.text + p); });
    return nd.depth == a.target_depth;
}

// The 16 lines from `first` (a multiple of 16) on: bit j = line first + j of
// [lo, hi) matches.
__device__ __forceinline__ uint32_t query_mask(const QueryArgs &a, uint32_t first, uint32_t hi) {
    uint32_t m = 0xFFFFu;  // lines of the range
    if (first < a.lo) m &= 0xFFFFu << (a.lo - first);
    if (first + 16 > hi) m &= (1u << (hi - first)) - 1u;  // first < hi
    if (!a.nodes && first + 16 <= a.lines && (a.target_depth < 255 || a.target_depth == NONE)) {
        if (a.target_kind > 255) return 0;
        if (a.target_kind) m &= eq_mask16(__ldg(reinterpret_cast<const uint4 *>(a.kinds + first)), a.target_kind * 0x01010101u);
        if (a.target_depth != NONE)
            m &= eq_mask16(__ldg(reinterpret_cast<const uint4 *>(a.depth8 + first)), a.target_depth * 0x01010101u);
        return m;
    }
    // materialised nodes, the document's last lines, depths of 255 and more
    uint32_t found = 0;
    for (uint32_t r = m; r; r &= r - 1) {
        const uint32_t j = __ffs(r) - 1;
        if (query_match(a, first + j)) found |= 1u << j;
    }
    return found;
}

__device__ __forceinline__ uint32_t qy_block_exclusive(uint32_t x, uint32_t *warp_sum, uint32_t *total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if ((int)lane >= o) inc += t;
    }
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < QY_THREADS / 32; w++) {
        before += w < warp ? warp_sum[w] : 0u;
        all += warp_sum[w];
    }
    if (total) *total = all;
    return before + inc - x;
}

// Block b: lines [4096 b, 4096 b + 4096) of those from lo rounded down to 16.
__global__ void __launch_bounds__(QY_THREADS) query_count_kernel(QueryArgs a) {
    __shared__ uint32_t warp_sum[QY_THREADS / 32];
    const uint32_t hi = a.hi_dev ? *a.hi_dev : a.hi;
    const uint64_t first = (uint64_t)(a.lo & ~15u) + (uint64_t)blockIdx.x * QY_LINES + threadIdx.x * QY_PER_THREAD;
    const uint32_t m = first < hi ? query_mask(a, (uint32_t)first, hi) : 0u;
    a.masks[(size_t)blockIdx.x * QY_THREADS + threadIdx.x] = (uint16_t)m;
    uint32_t total;
    qy_block_exclusive(__popc(m), warp_sum, &total);
    if (threadIdx.x == 0) a.counts[blockIdx.x] = total;
}

__global__ void __launch_bounds__(QY_THREADS) query_write_kernel(QueryArgs a) {
    __shared__ uint32_t warp_sum[QY_THREADS / 32], before_sum[QY_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t mine = a.counts[blockIdx.x];
    const bool last = blockIdx.x + 1 == gridDim.x;
    if (mine == 0 && !(a.bases == nullptr && last)) return;  // uniform
    uint32_t base = 0;
    if (a.bases) {
        base = a.bases[blockIdx.x];
    } else {
        uint32_t before = 0;
        for (uint32_t b = tid; b < blockIdx.x; b += QY_THREADS) before += a.counts[b];
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        if (lane == 0) before_sum[warp] = before;
        __syncthreads();
#pragma unroll
        for (uint32_t w = 0; w < QY_THREADS / 32; w++) base += before_sum[w];
        if (last && tid == 0) *a.total = base + mine;
    }
    if (mine == 0 || base >= a.max_out) return;  // uniform
    uint32_t m = a.masks[(size_t)blockIdx.x * QY_THREADS + tid];
    uint32_t r = base + qy_block_exclusive(__popc(m), warp_sum, nullptr);
    const uint32_t first = (a.lo & ~15u) + blockIdx.x * QY_LINES + tid * QY_PER_THREAD;
    for (; m && r < a.max_out; m &= m - 1) a.out[r++] = first + __ffs(m) - 1;
}

cudaError_t launch_query(const QueryArgs &a, cudaStream_t st) {
    if (a.hi <= a.lo) return cudaSuccess;
    const uint32_t blocks = query_blocks(a.lo, a.hi);
    query_count_kernel<<<blocks, QY_THREADS, 0, st>>>(a); OL_LAUNCHED();
    QueryArgs w = a;
    if (blocks <= kQuerySelfScan) {
        w.bases = nullptr;
    } else {
        cudaError_t e = launch_scan_columns(a.counts, a.bases, a.total, blocks, 1, scan_ld(blocks), st);
        if (e != cudaSuccess) return e;
    }
    query_write_kernel<<<blocks, QY_THREADS, 0, st>>>(w); OL_LAUNCHED();
    return cudaGetLastError();
}

}  // namespace ol
