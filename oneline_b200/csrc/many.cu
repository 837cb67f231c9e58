// Kernel (e): dictionary search. Every (pattern, offset) at which one of a set
// of patterns (4..64 bytes, up to 65,536 of them) occurs, ordered by
// (pattern, offset) like ManyPatterns::find_all_par
// (crates/oneline-simd/src/search.rs:259-282). Replaces the reference's
// window-filter kernels and host sort (crates/oneline-gpu/src/many.rs:391-646).
//
// The compiled set (runtime_many.cu) deduplicates the patterns. In oneline text
// most dictionary hits lie in and around runs of one byte (indent markers,
// rules), so the patterns of up to four run bytes c that start with c^3 are
// kept apart:
//   * runs c^k: found with bit masks, without looking at any position alone;
//   * c^r rest (r >= 3, rest starting with another byte): found from the end of
//     a run, once for all r: a trie over the rests, whose nodes list (r, pattern).
// All other patterns are in a trie whose depth-4 nodes are reached through a
// hash table keyed by a position's first four bytes. Where a trie continues with
// a run byte several times (a line break, then indent markers), the node where
// that begins lists the nodes of the run, so that a walk takes it in one step,
// by the run's length in the text. A filter of those keys, and of c c c
// rest[0] for the run ends, sits in shared memory (16 KiB), copied there once
// per block with a bulk TMA copy (cp.async.bulk, no multicast).
//
// dict_match_kernel: persistent warps take slices of the text in turn. Every
// position is filtered (16 a lane, from registers), the candidates are queued
// and walked 32 at a time, one per lane; nodes with patterns are queued in turn
// and their hits written 32 nodes at a time. Every hit is found by the warp
// whose slice holds its start.
//   * heavy patterns (chosen per search from a sample of the text) set bits in
//     a bitmap: the slice's words are gathered in shared memory and stored once;
//   * light patterns append (u, offset) keys through a per-warp buffer, and
//     count themselves.
// Before it, the same kernel counts hits on a sample of the text, and
// dict_plan_kernel picks the heavy patterns from the counts, on the device.
// After it, a column scan of the heavy hits per tile gives every heavy hit its
// rank; a radix sort orders the light keys; a single-block pass gives every
// pattern id its first output slot; the emit kernels write each hit once per id
// that holds the same bytes (duplicates are reported once per id).
#include <cuda_runtime.h>

#include <algorithm>

#include "ol_common.cuh"
#include "ol_kernels.h"

namespace ol {

// Two blocks of 20 warps fit an SM (registers and shared memory, the filter in
// each block): 597 us against 659 with four of 8 warps (64 MiB, 10,000
// patterns). A text whose slices are all walked at once by blocks of four warps
// is spread over the chip in those: a text whose slices are at most 24 a SM (100
// patterns, 1 MiB, is 100 us with either; 2 MiB 107 against 109 in large blocks, and
// with 96 a SM 115).
constexpr uint32_t DM_THREADS = 640;
constexpr uint32_t DM_SMALL_THREADS = 128, DM_SMALL_WARPS_PER_SM = 24;
constexpr uint32_t DM_QCAP = 64;                          // per-warp candidate queue
constexpr uint32_t DM_FILTER_WORDS = 1u << (kDictFilterBits - 5);
constexpr uint32_t kMbarSpins = 1u << 24;
constexpr uint32_t DM_LIGHT = 32;                         // per-warp buffer of light keys
constexpr uint32_t DM_EVENTS = 64;                        // per-warp queue of nodes with hits
constexpr uint32_t DM_POW = 7;                            // run masks of 1, 2, 4, .., 64 bytes
// A warp's work item: SLICE text positions (staged with the longest pattern
// after them) and their SLICE / 32 heavy-bitmap words per heavy pattern.
template <uint32_t SLICE>
struct DictWarp {
    static constexpr uint32_t kWords = SLICE / 32;
    static constexpr uint32_t kRunWords = kWords + 2;  // the slice and the 64 positions after it
    static constexpr uint32_t kText = SLICE + kDictHalo;
    static_assert(kText % 16 == 0 && kDictWordsPerTile % kWords == 0 && kDictTile % SLICE == 0, "slice geometry");
    alignas(16) uint8_t text[kText];
    alignas(16) uint32_t bits[kDictMaxHeavy][kWords];  // heavy pattern h starts at the positions of the set bits
    unsigned long long light[DM_LIGHT];
    // bit p of words 2..: position p holds the run byte (two words of 0 before, two after)
    uint32_t run[kDictMaxRuns][kRunWords + 4];
    uint32_t pow[DM_POW][kRunWords + 1];        // one run byte's: 2^i of it start at the position (a word of 0 after)
    unsigned long long ev_starts[DM_EVENTS];    // DictEvent
    uint32_t ev_at[DM_EVENTS];
    uint32_t n_light, n_events;
    uint16_t queue[DM_QCAP];
};
template <uint32_t SLICE>
struct DictSmem {
    uint32_t filter[DM_FILTER_WORDS];
    uint32_t heavy_run[kDictMaxHeavy];  // the heavy run patterns: (j << 16) | (k << 8) | heavy index
    uint32_t n_heavy_run;
    alignas(8) unsigned long long bar;
    DictWarp<SLICE> w[DM_THREADS / 32];  // as many as the block has warps

    static size_t bytes(uint32_t threads) {
        return sizeof(DictSmem) - (DM_THREADS - threads) / 32 * sizeof(DictWarp<SLICE>);
    }
};

// ---------------------------------------------------------------- TMA bulk --

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

// Global -> shared bulk copy (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity) {
    for (uint32_t i = 0; i < kMbarSpins; i++) {
        uint32_t ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// ------------------------------------------------------------ trie walk ----

__device__ __forceinline__ uint32_t dict_child(const DictSet &s, const uint4 &nd, uint32_t b) {
    if (nd.y & kDictDenseFlag) return __ldg(s.dense + (size_t)nd.w * 256 + b);
    const uint32_t n = nd.y & kDictEdgeMask;
    if (n == 0) return NONE;
    uint32_t e0 = nd.z & 0xFFu;
    if (e0 == b) return nd.z >> 8;
    if (n == 1 || b < e0) return NONE;
    if (n == 2) return (nd.w & 0xFFu) == b ? nd.w >> 8 : NONE;
    for (uint32_t i = 0; i < n - 1; i++) {
        uint32_t e = __ldg(s.extra + nd.w + i);
        uint32_t eb = e & 0xFFu;
        if (eb == b) return e >> 8;
        if (eb > b) break;
    }
    return NONE;
}

__device__ __forceinline__ uint32_t dict_probe(const DictSet &s, uint32_t key) {
    const uint32_t mask = (1u << s.table_bits) - 1u;
    uint32_t slot = dict_table_h(key, s.table_bits);
    for (uint32_t i = 0; i <= s.max_probe; i++) {
        uint2 e = __ldg(s.table + slot);
        if (e.y == NONE) return NONE;
        if (e.x == key) return e.y;
        slot = (slot + 1) & mask;
    }
    return NONE;
}

// ------------------------------------------------------------- matching ----

// The unique pattern of entry x, (heavy index + 1, or 0) << 16 | u, starts at
// slice position p (absolute: pos): counts (count mode), a bit of the heavy
// pattern's bitmap words, or a light key.
template <uint32_t SLICE>
__device__ __forceinline__ void dict_emit(const DictMatchArgs &a, DictWarp<SLICE> &w, uint32_t x, uint32_t p, uint64_t pos) {
    const uint32_t u = x & 0xFFFFu, hv = (x >> 16) & 0xFFu;
    if (a.count_only) {
        const uint32_t peers = __match_any_sync(__activemask(), u);
        if ((peers & ((1u << (threadIdx.x & 31)) - 1u)) == 0) atomicAdd(a.counts + u, (uint32_t)__popc(peers));
        return;
    }
    if (hv) {
        atomicOr(&w.bits[hv - 1][p >> 5], 1u << (p & 31));
        return;
    }
    atomicAdd(a.counts + u, 1u);
    const unsigned long long key = ((unsigned long long)u << a.off_bits) | pos;
    const uint32_t at = atomicAdd(&w.n_light, 1u);
    if (at < DM_LIGHT) {
        w.light[at] = key;
    } else {  // the buffer is full until the walk's lanes meet again
        const uint32_t slot = atomicAdd(a.light_n, 1u);
        if (slot < a.light_cap) a.light_keys[slot] = key;
    }
}

// The whole warp moves the buffered light keys to the search's list when at
// least `least` are there.
template <uint32_t SLICE>
__device__ __forceinline__ void dict_flush(const DictMatchArgs &a, DictWarp<SLICE> &w, uint32_t least) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    const uint32_t n = min(w.n_light, DM_LIGHT);
    if (n < least) return;  // uniform
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(a.light_n, n);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    for (uint32_t i = lane; i < n; i += 32)
        if (base + i < a.light_cap) a.light_keys[base + i] = w.light[i];
    __syncwarp();
    if (lane == 0) w.n_light = 0;
    __syncwarp();
}

// Hits of one node: patterns outs[o], outs[o + 1], ... start r before slice
// position e for the set bits r of `starts` in turn; with `same`, all at e.
// Packed: at = (same << 31) | (o << 11) | e.
constexpr uint32_t kEventSame = 0x80000000u;

template <uint32_t SLICE>
__device__ __forceinline__ void dict_hits(const DictMatchArgs &a, DictWarp<SLICE> &w, unsigned long long starts, uint32_t at,
                                          uint64_t s0) {
    const uint32_t e = at & 0x7FFu;
    const uint32_t *o = a.outs + ((at & ~kEventSame) >> 11);
    uint32_t next = __ldg(o);  // a step ahead (the entry after the last is not used)
    for (; starts; starts &= starts - 1) {
        const uint32_t entry = next, p = (at & kEventSame) ? e : e + 1 - __ffsll(starts);
        next = __ldg(++o);
        dict_emit(a, w, entry, p, s0 + p);
    }
}

// A node's hits at once, when the queue is full until the walk's lanes meet
// again. Out of line: the walk's code has to stay small (inlined with its
// callers, the match kernel waited for instructions more than for anything
// but memory).
template <uint32_t SLICE>
__device__ __noinline__ void dict_hits_now(const DictMatchArgs &a, DictWarp<SLICE> &w, unsigned long long starts, uint32_t at,
                                           uint64_t s0) {
    dict_hits(a, w, starts, at, s0);
}

template <uint32_t SLICE>
__device__ __forceinline__ void dict_push(const DictMatchArgs &a, DictWarp<SLICE> &w, unsigned long long starts, uint32_t at,
                                          uint64_t s0) {
    const uint32_t i = atomicAdd(&w.n_events, 1u);
    if (i < DM_EVENTS) {
        w.ev_starts[i] = starts;
        w.ev_at[i] = at;
    } else {
        dict_hits_now(a, w, starts, at, s0);
    }
}

// The whole warp writes the hits of the queued nodes, one per lane, when at
// least `least` are queued.
template <uint32_t SLICE>
__device__ __forceinline__ void dict_drain(const DictMatchArgs &a, DictWarp<SLICE> &w, uint32_t least, uint64_t s0) {
    __syncwarp();
    const uint32_t n = min(w.n_events, DM_EVENTS);
    if (n < least) return;  // uniform
    for (uint32_t i = threadIdx.x & 31; i < n; i += 32) dict_hits(a, w, w.ev_starts[i], w.ev_at[i], s0);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) w.n_events = 0;
    if (!a.count_only) dict_flush(a, w, DM_LIGHT / 2);
    __syncwarp();
}

// Length of the run of run byte j that starts at slice position p (which holds
// it), as far as the masks go.
template <uint32_t SLICE>
__device__ __forceinline__ uint32_t dict_run_from(const DictWarp<SLICE> &w, uint32_t j, uint32_t p) {
    const uint32_t *rw = w.run[j] + 2 + (p >> 5);
    const uint32_t lo = __funnelshift_r(rw[0], rw[1], p & 31);
    if (lo != 0xFFFFFFFFu) return __ffs(~lo) - 1;
    const uint32_t hi = __funnelshift_r(rw[1], rw[2], p & 31);
    return 32 + (hi != 0xFFFFFFFFu ? __ffs(~hi) - 1 : 32);
}

// Every hit of the candidate at slice position p. Hits must end by `lim` (the
// end of the text, or of the position's document in a batch).
//   * c c c x of a run byte c, x another: the run's end e = p + 3 is walked, for
//     the starts that lie in the slice, 3 to R (the run's length back to the
//     slice's start) before e;
//   * any other four bytes: the table gives the depth-4 node.
template <uint32_t SLICE>
__device__ __forceinline__ void dict_walk(const DictMatchArgs &a, DictWarp<SLICE> &w, uint32_t p, uint64_t s0, uint64_t lim,
                                          uint32_t &levels) {
    const uint32_t *tw = reinterpret_cast<const uint32_t *>(w.text);
    const uint32_t key = __funnelshift_r(tw[p >> 2], tw[(p >> 2) + 1], (p & 3) * 8);
    if (s0 + p + kDictMinLen > lim) return;
    uint32_t j = a.set.n_runs;
    if (((key ^ (key >> 8)) & 0xFFFFu) == 0)  // three equal bytes
        for (j = 0; j < a.set.n_runs && ((a.set.run_bytes >> (8 * j)) & 0xFFu) != (key & 0xFFu);) j++;
    // The text from slice position e on is matched against a trie from node v,
    // t bytes so far; a node's patterns start r before e: r = 0, or the starts
    // that lie in the slice, r0 to R.
    uint32_t v, e = p, t = kDictMinLen, r0 = 0;
    unsigned long long starts = 1;
    if (j < a.set.n_runs) {
        const uint32_t *rw = w.run[j] + (p >> 5);  // words p/32 - 2 .. p/32
        const uint32_t hi = __funnelshift_r(rw[1], rw[2], p & 31), lo = __funnelshift_r(rw[0], rw[1], p & 31);
        const uint32_t back = hi != 0xFFFFFFFFu ? __clz(~hi) : 32 + __clz(~lo);  // (__clz(0) = 32)
        e = p + 3;
        t = 1;
        r0 = e > SLICE + 2 ? e - SLICE + 1 : 3u;  // at most 63: see the candidates past the slice
        starts = (~0ull >> (kDictMaxLen - 1 - min(3 + back, kDictMaxLen - 1))) & (~0ull << r0);
        v = __ldg(a.set.dense + (size_t)a.set.run_root[j] * 256 + (key >> 24));
    } else {
        v = dict_probe(a.set, key);
    }
    const uint32_t end = (uint32_t)min(lim - s0, (uint64_t)(SLICE + 2 * kDictMaxLen));  // lim, as a slice position
    while (v != NONE) {
        const uint4 nd = __ldg(a.set.nodes + v);
        levels++;
        if (nd.x != NONE) {
            if (nd.x & kDictOneFlag) {
                dict_push(a, w, 1ull, ((nd.x & ~kDictOneFlag) << 11) | e, s0);
            } else {  // of the list's entries only those that count
                const uint4 l = __ldg(a.set.lists + nd.x);
                const unsigned long long all = ((unsigned long long)l.y << 32) | l.x, m = all & starts;
                if (m) dict_push(a, w, m, ((l.z + __popcll(all & ((m & (0 - m)) - 1))) << 11) | e, s0);
            }
        }
        if (t + r0 >= kDictMaxLen || e + t >= end) break;
        const uint32_t b = w.text[e + t];
        if ((nd.y & kDictPathFlag) && b == ((a.set.run_bytes >> (8 * ((nd.y >> 28) & 3u))) & 0xFFu)) {
            // the node's run: K nodes, the patterns of those passed by, then on from the last one reached
            const uint32_t *path = a.set.paths + ((nd.y >> 9) & 0x7FFFFu);
            const uint32_t D = min(min(__ldg(path), min(kDictMaxLen - t, end - e - t)),
                                   dict_run_from(w, (nd.y >> 28) & 3u, e + t));
            const unsigned long long all = ((unsigned long long)__ldg(path + 2) << 32) | __ldg(path + 1);
            const uint32_t n = __popcll(all & ((1ull << (D - 1)) - 1));  // D >= 1: b is the run byte
            if (n) dict_push(a, w, (1ull << n) - 1, kEventSame | (__ldg(path + 3) << 11) | e, s0);
            v = __ldg(path + 3 + D);
            t += D;
            continue;
        }
        v = dict_child(a.set, nd, b);
        t++;
    }
}

// 16-bit mask of the positions lo .. lo + 15 below n.
__device__ __forceinline__ uint32_t below16(uint32_t n, uint32_t lo) {
    return n <= lo ? 0u : n - lo >= 16 ? 0xFFFFu : (1u << (n - lo)) - 1u;
}

// The pattern run_byte(j)^k over the slice's word i: bit b is set where it
// starts. pow[q] holds the starts of runs of 2^q: with 2^q <= k < 2^(q+1) a run
// of k is one of 2^q here and one k - 2^q further on.
template <uint32_t SLICE>
__device__ __forceinline__ uint32_t dict_run_word(const DictWarp<SLICE> &w, uint32_t k, uint32_t i) {
    const uint32_t q = 31 - __clz(k), s = k - (1u << q);  // k = 4..64: s <= 31
    return w.pow[q][i] & __funnelshift_r(w.pow[q][i], w.pow[q][i + 1], s);
}

// End of the document holding pos (pos itself when pos lies between
// documents), searching forward from hint, the first document ending after the
// slice start.
__device__ __forceinline__ uint64_t dict_limit(const DictMatchArgs &a, uint64_t pos, uint32_t hint) {
    if (!a.seg_end) return a.text_len;
    uint32_t i = hint;
    while (i < a.n_seg && a.seg_end[i] <= pos) i++;
    if (i == a.n_seg || a.seg_start[i] > pos) return pos;
    return a.seg_end[i];
}

// Each warp takes slices of SLICE positions in turn: it stages the slice (plus
// the longest pattern) in its own shared memory, filters all positions 32 at a
// time, queues the candidates and walks them 32 at a time (one per lane), so
// walks run on full warps; then it finds the run patterns from the run bytes'
// masks and stores the heavy patterns' words of the slice. Warps never wait for
// one another.
template <uint32_t SLICE>
__global__ void __launch_bounds__(DM_THREADS, 2) dict_match_kernel(const __grid_constant__ DictMatchArgs a) {
    using Warp = DictWarp<SLICE>;
    constexpr uint32_t DM_SLICES_PER_TILE = kDictTile / SLICE;
    extern __shared__ __align__(16) uint8_t dyn_smem[];
    DictSmem<SLICE> &sm = *reinterpret_cast<DictSmem<SLICE> *>(dyn_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;

    // The filter, once per block, by a bulk copy.
    if (tid == 0) mbar_init(&sm.bar, 1);
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&sm.bar, DM_FILTER_WORDS * 4);
        bulk_copy_g2s(sm.filter, a.set.filter, DM_FILTER_WORDS * 4, &sm.bar);
    }
    bool ok = mbar_wait(&sm.bar, 0);
    // (A separate statement: folded into the wait's result, the test hook
    // made the whole match kernel 47% slower, 19.8 against 13.5 ms per GiB.)
    if (a.force_timeout) ok = false;
    if (warp == 0) {
        const uint32_t x = !a.count_only && lane < a.plan->n_heavy ? a.heavy_run[lane] : 0u;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, x != 0);
        if (x) sm.heavy_run[__popc(m & lt)] = (x << 8) | lane;
        if (lane == 0) sm.n_heavy_run = __popc(m);
    }
    if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicOr(a.error, OL_DEVERR_TIMEOUT);
        mbar_wait(&sm.bar, 0);  // let the copy land before the block exits
        return;
    }

    const uint64_t N = a.text_len;
    const uint32_t n_words = a.n_tiles * kDictWordsPerTile;
    const uint32_t per_tile = DM_SLICES_PER_TILE / a.slices;  // items of a tile, of a.slices slices each
    const uint32_t n_items = ((a.n_tiles + a.tile_stride - 1) / a.tile_stride) * per_tile;
    const uint32_t H = a.count_only ? 0u : a.plan->n_heavy, n_runs = a.set.n_runs, run_bytes = a.set.run_bytes;
    const uint32_t n_run_light = a.count_only ? a.n_run_light : a.plan->n_run_light;
    uint32_t cands = 0, levels = 0;  // per lane, for the search statistics
    Warp &w = sm.w[warp];
    uint8_t *text = w.text;
    uint16_t *queue = w.queue;
    const uint32_t *tw = reinterpret_cast<const uint32_t *>(text);
    if (lane == 0) w.n_light = w.n_events = 0;
    if (lane < kDictMaxRuns) {
        w.run[lane][0] = w.run[lane][1] = 0;
        w.run[lane][Warp::kRunWords + 2] = w.run[lane][Warp::kRunWords + 3] = 0;
    }
    for (uint32_t i = lane; i < DM_POW; i += 32) w.pow[i][Warp::kRunWords] = 0;
    if (lane < H && H)
        for (uint32_t i = 0; i < Warp::kWords; i += 4) *reinterpret_cast<uint4 *>(&w.bits[lane][i]) = make_uint4(0, 0, 0, 0);

    // item by item, slice by slice; `found`: the item's hits of heavy pattern `lane`
    for (uint32_t item = blockIdx.x * n_warps + warp, nth = 0, found = 0; item < n_items;) {
        const uint32_t tile = (item / per_tile) * a.tile_stride;
        const uint32_t slice = tile * DM_SLICES_PER_TILE + (item % per_tile) * a.slices + nth;
        const uint64_t s0 = (uint64_t)slice * SLICE;  // slices past the text only write zero words
        constexpr uint32_t kPieces = SLICE / 16, kMine = (kPieces + 31) / 32;  // 16-byte pieces; a lane's
        uint4 v[kMine];
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < kMine; i++) {
            const uint32_t piece = i * 32 + lane;
            v[i] = ld_stream16(a.text + s0 + piece * 16);  // (SLICE = 256: up to 256 bytes past the slice)
            if (piece < Warp::kText / 16) *reinterpret_cast<uint4 *>(&text[piece * 16]) = v[i];
        }
        if (kMine * 32 + lane < Warp::kText / 16)
            *reinterpret_cast<uint4 *>(&text[(kMine * 32 + lane) * 16]) = ld_stream16(a.text + s0 + (kMine * 32 + lane) * 16);
        // bytes of the text from the slice start on, as far as they matter here
        const uint32_t have = N > s0 ? (uint32_t)min(N - s0, (uint64_t)(SLICE + 64)) : 0u;
        __syncwarp();
        uint32_t hint = 0;
        if (a.seg_end) {  // first document ending after the slice start
            uint32_t lo = 0, hi = a.n_seg;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.seg_end[mid] <= s0)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            hint = lo;
        }
        // The run bytes' masks over the slice and the 64 positions after it.
#pragma unroll 1
        for (uint32_t j = 0; j < n_runs; j++) {
            const uint32_t c = (run_bytes >> (8 * j)) & 0xFFu;
#pragma unroll
            for (uint32_t i = 0; i < kMine; i++) {
                const uint32_t piece = i * 32 + lane;
                uint32_t m = eq_mask16(v[i], c * 0x01010101u) & below16(have, piece * 16);
                m |= __shfl_down_sync(0xFFFFFFFFu, m, 1) << 16;
                if (!(lane & 1) && piece < kPieces) w.run[j][2 + piece / 2] = m;
            }
            const uint32_t q = SLICE + lane;
            const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, text[q] == c && q < have);
            const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, text[q + 32] == c && q + 32 < have);
            if (lane < 2) w.run[j][2 + Warp::kWords + lane] = lane ? m1 : m0;
        }
        __syncwarp();
        // Candidates, lane by lane: bit q of cm is position piece * 16 + q.
        uint32_t cm[kMine];
#pragma unroll
        for (uint32_t i = 0; i < kMine; i++) {
            const uint32_t piece = i * 32 + lane;
            const uint32_t *pw = tw + (piece < kPieces ? piece * 4 : 0);
            uint32_t m = 0, x = pw[0];
#pragma unroll 1
            for (uint32_t q = 0; q < 16; q += 4) {  // (rolled: the code has to stay small)
                const uint32_t y = *++pw;
#pragma unroll
                for (uint32_t b = 0; b < 4; b++) {
                    const uint32_t key = b ? __funnelshift_r(x, y, 8 * b) : x;
                    const uint32_t f = sm.filter[dict_filter_word(key)], g = dict_filter_bits(key);
                    m |= ((f >> (g >> 27)) & (f >> ((g >> 22) & 31)) & (f >> ((g >> 17) & 31)) & 1u) << (q + b);
                }
                x = y;
            }
            m &= piece < kPieces ? below16(have > 3 ? have - 3 : 0u, piece * 16) : 0u;  // four bytes of text
#pragma unroll 1
            for (uint32_t j = 0; j < n_runs; j++) {  // c^4: inside a run, the masks find those
                const uint32_t *rw = w.run[j] + 2 + (piece < kPieces ? piece / 2 : 0);
                const uint32_t r = __funnelshift_r(rw[0], rw[1], (piece & 1) * 16);
                m &= ~(r & (r >> 1) & (r >> 2) & (r >> 3));
            }
            cm[i] = m;
        }
        // The end of a run that covers the slice's last position and ends at
        // least 3 further on is one more candidate, past the slice.
        uint32_t tail = 0;
#pragma unroll 1
        for (uint32_t j = 0; j < n_runs; j++) {
            if (!(w.run[j][Warp::kWords + 1] >> 31)) continue;  // uniform, and so is what follows
            const uint32_t f = dict_run_from(w, j, SLICE);
            // (f = 63: a start in the slice would need a pattern of 64 run bytes and a rest)
            if (f >= 3 && f + 1 < kDictMaxLen) tail = SLICE + f - 3;  // of one run byte at most
        }
        for (uint32_t qn = 0, at = 0, last = 0; !last;) {
            while (qn < 32 && !last) {  // each lane's lowest candidate, until the queue holds a full round
                uint32_t mine = cm[0];
#pragma unroll
                for (uint32_t i = 1; i < kMine; i++) mine = at == i ? cm[i] : mine;
                const uint32_t any = __ballot_sync(0xFFFFFFFFu, mine != 0);
                if (any) {
                    if (mine) queue[qn + __popc(any & lt)] = (uint16_t)((at * 32 + lane) * 16 + __ffs(mine) - 1);
                    qn += __popc(any);
#pragma unroll
                    for (uint32_t i = 0; i < kMine; i++)
                        if (at == i) cm[i] = mine & (mine - 1);
                } else if (++at == kMine) {
                    if (tail && lane == 0) queue[qn] = (uint16_t)tail;
                    qn += tail != 0;
                    tail = 0;
                    last = qn <= 32;
                    if (!last) at = kMine - 1;
                }
            }
            __syncwarp();
            const uint32_t n = min(qn, 32u);
            if (lane < n) {  // one candidate per lane
                const uint32_t p = queue[lane];
                dict_walk(a, w, p, s0, dict_limit(a, s0 + p, hint), levels);
                cands++;
            }
            __syncwarp();
            const uint16_t keep = lane + 32 < qn ? queue[lane + 32] : (uint16_t)0;
            __syncwarp();
            if (lane + 32 < qn) queue[lane] = keep;
            qn -= n;
            dict_drain(a, w, last ? 1 : DM_EVENTS / 2, s0);
        }
        // Run patterns, one run byte after the other.
#pragma unroll 1
        for (uint32_t j = 0; j < n_runs; j++) {
            bool any = false;
            for (uint32_t i = lane; i < Warp::kRunWords; i += 32) w.pow[0][i] = w.run[j][i + 2];
#pragma unroll
            for (uint32_t q = 1; q < DM_POW; q++) {
                __syncwarp();
                for (uint32_t i = lane; i < Warp::kRunWords; i += 32) {
                    const uint32_t x = w.pow[q - 1][i], y = w.pow[q - 1][i + 1];
                    const uint32_t z = x & (q == 6 ? y : __funnelshift_r(x, y, 1u << (q - 1)));
                    w.pow[q][i] = z;
                    if (q == 2) any |= i < Warp::kWords && z != 0;
                }
                if (q == 2 && !__any_sync(0xFFFFFFFFu, any)) break;  // no run of four
            }
            if (!__any_sync(0xFFFFFFFFu, any)) continue;
            __syncwarp();
            const uint32_t n_hr = sm.n_heavy_run;
            for (uint32_t i = lane; i < n_hr * Warp::kWords; i += 32) {  // (pattern, word) pairs
                const uint32_t x = sm.heavy_run[i / Warp::kWords];
                if ((x >> 16) == j) w.bits[x & 0xFFu][i % Warp::kWords] = dict_run_word(w, (x >> 8) & 0xFFu, i % Warp::kWords);
            }
            // the light ones (all of them in count mode)
            for (uint32_t n = 0; n < n_run_light; n++) {
                const uint32_t x = __ldg(a.run_light + n);  // (j << 24) | (k << 16) | u
                if ((x >> 24) != j) continue;
                const uint32_t u = x & 0xFFFFu;
                uint32_t sum = 0;
                for (uint32_t i = lane; i < Warp::kWords; i += 32) {
                    uint32_t m = dict_run_word(w, (x >> 16) & 0xFFu, i);
                    sum += __popc(m);
                    if (a.count_only) continue;
                    for (; m; m &= m - 1) {
                        const uint32_t p = i * 32 + __ffs(m) - 1;
                        dict_emit(a, w, u, p, s0 + p);
                    }
                }
                if (a.count_only) {
                    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
                    if (lane == 0 && sum) atomicAdd(a.counts + u, sum);
                } else {
                    dict_flush(a, w, DM_LIGHT / 2);
                }
            }
        }
        __syncwarp();
        // lane h stores heavy pattern h's words of the slice (contiguous, 16-byte stores) and clears them
        if (lane < H) {
            uint4 *dst = reinterpret_cast<uint4 *>(a.bitmap + (size_t)lane * n_words + (size_t)slice * Warp::kWords);
            uint4 *src = reinterpret_cast<uint4 *>(w.bits[lane]);
#pragma unroll
            for (uint32_t i = 0; i < Warp::kWords / 4; i++) {
                const uint4 x = src[i];
                found += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
                dst[i] = x;
                src[i] = make_uint4(0, 0, 0, 0);
            }
        }
        if (++nth == a.slices) {
            if (found) atomicAdd(a.heavy_counts + (size_t)lane * a.heavy_ld + tile, found);  // (lane < H)
            nth = found = 0;
            item += gridDim.x * n_warps;
        }
    }
    if (!a.count_only) dict_flush(a, w, 1);
    if (a.stats) {  // candidates walked and trie nodes visited
        const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, cands), l = __reduce_add_sync(0xFFFFFFFFu, levels);
        if (lane == 0) {
            atomicAdd(a.stats, (unsigned long long)c);
            atomicAdd(a.stats + 1, (unsigned long long)l);
        }
    }
}

template <uint32_t SLICE>
static cudaError_t launch_match(const DictMatchArgs &args, int sm_count, uint32_t blocks_per_sm, cudaStream_t st) {
    DictMatchArgs a = args;
    uint64_t n_items = (uint64_t)((a.n_tiles + a.tile_stride - 1) / a.tile_stride) * (kDictTile / SLICE);
    const bool small = n_items <= (uint64_t)sm_count * DM_SMALL_WARPS_PER_SM;
    const uint32_t threads = small ? DM_SMALL_THREADS : DM_THREADS, warps = threads / 32;
    const size_t smem = DictSmem<SLICE>::bytes(threads);
    cudaError_t e = cudaFuncSetAttribute(dict_match_kernel<SLICE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(DictSmem<SLICE>));
    if (e != cudaSuccess) return e;
    uint64_t grid = (n_items + warps - 1) / warps;
    if (!small || blocks_per_sm) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dict_match_kernel<SLICE>, threads, smem);
        if (e != cudaSuccess) return e;
        if (blocks_per_sm) per_sm = std::min<int>(per_sm, (int)blocks_per_sm);
        grid = std::min<uint64_t>(grid, (uint64_t)std::max(per_sm, 1) * sm_count);
    }
    // items of several slices, as long as every warp gets a few dozen of them:
    // the heavy hits of an item are counted in registers
    a.slices = 1;
    while (a.slices < 8 && a.slices * 2 * SLICE <= kDictTile && n_items >= grid * warps * 32) {
        a.slices *= 2;
        n_items /= 2;
    }
    dict_match_kernel<SLICE><<<(uint32_t)grid, threads, smem, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

// slice: text positions per warp work item (256, 512 or 1024); blocks_per_sm:
// resident blocks per SM of the persistent grid (0: as many as fit).
cudaError_t launch_dict_match(const DictMatchArgs &a, int sm_count, cudaStream_t st, uint32_t slice,
                              uint32_t blocks_per_sm) {
    if (a.n_tiles == 0) return cudaSuccess;
    // half the serial work per warp where the text leaves most of the chip idle
    if (slice == 512 && (uint64_t)((a.n_tiles + a.tile_stride - 1) / a.tile_stride) * (kDictTile / 256) <=
                            (uint64_t)sm_count * DM_SMALL_WARPS_PER_SM)
        slice = 256;
    switch (slice) {
        case 256: return launch_match<256>(a, sm_count, blocks_per_sm, st);
        case 1024: return launch_match<1024>(a, sm_count, blocks_per_sm, st);
        default: return launch_match<512>(a, sm_count, blocks_per_sm, st);
    }
}

// ------------------------------------------------------------------ plan ----

constexpr uint32_t DP_THREADS = 1024;

// One block picks the heavy patterns from the sample counts: the (at most 32)
// most frequent of those at or above `least`, lower u first among equals. (Of
// more than 1024 such patterns any 1024 are looked at: which patterns are heavy
// changes nothing but the time.) Then the lists that the match pass reads.
__global__ void __launch_bounds__(DP_THREADS) dict_plan_kernel(DictPlanArgs a) {
    __shared__ uint32_t cand_u[DP_THREADS], cand_n[DP_THREADS], n_cand, n_light_runs;
    __shared__ unsigned long long light;
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        n_cand = n_light_runs = 0;
        light = 0;
    }
    if (tid < kDictMaxHeavy) a.heavy_run[tid] = a.heavy_u[tid] = 0;
    __syncthreads();
    unsigned long long below = 0;
    for (uint32_t u = tid; u < a.set.n_u; u += DP_THREADS) {
        const uint32_t n = a.sample_counts[u];
        a.heavy_of_u[u] = 0xFF;
        uint32_t at = DP_THREADS;
        if (n >= a.least) at = atomicAdd(&n_cand, 1u);
        if (at < DP_THREADS) {
            cand_u[at] = u;
            cand_n[at] = n;
        } else {
            below += n;
        }
    }
    if (below) atomicAdd(&light, below);
    __syncthreads();
    const uint32_t c = min(n_cand, DP_THREADS);
    if (tid < c) {
        uint32_t rank = 0;
        for (uint32_t i = 0; i < c; i++)
            rank += cand_n[i] > cand_n[tid] || (cand_n[i] == cand_n[tid] && cand_u[i] < cand_u[tid]);
        if (rank < kDictMaxHeavy) {
            a.heavy_u[rank] = cand_u[tid];
            a.heavy_of_u[cand_u[tid]] = (uint8_t)rank;
        } else {
            atomicAdd(&light, (unsigned long long)cand_n[tid]);
        }
    }
    __syncthreads();  // heavy_of_u is complete (one block: its own global writes)
    for (uint32_t i = tid; i < a.n_runs; i += DP_THREADS) {
        const uint32_t x = a.runs[i];
        const uint32_t h = a.heavy_of_u[x & 0xFFFFu];
        if (h != 0xFFu)
            a.heavy_run[h] = x >> 16;
        else
            a.run_light[atomicAdd(&n_light_runs, 1u)] = x;
    }
    for (uint32_t i = tid; i < a.set.n_outs; i += DP_THREADS) {
        const uint32_t u = a.set.outs[i];
        a.outs[i] = (((a.heavy_of_u[u] + 1u) & 0xFFu) << 16) | u;
    }
    __syncthreads();
    if (tid == 0) {
        a.plan->n_heavy = min(c, kDictMaxHeavy);
        a.plan->n_run_light = n_light_runs;
        a.plan->light_sample = light;
    }
}

cudaError_t launch_dict_plan(const DictPlanArgs &a, cudaStream_t st) {
    dict_plan_kernel<<<1, DP_THREADS, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

// ------------------------------------------------------- block-wide sums ----

constexpr uint32_t DH_THREADS = 256;

// Block sum / exclusive scan helpers for 256 threads.
__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t x, uint32_t *warp_sum, uint32_t *total) {
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
    for (uint32_t w = 0; w < DH_THREADS / 32; w++) {
        uint32_t ws = warp_sum[w];
        before += w < warp ? ws : 0u;
        all += ws;
    }
    __syncthreads();
    if (total) *total = all;
    return before + inc - x;
}

// ---------------------------------------------------- light-key radix sort --
//
// LSD radix sort of the keys, 8 bits a pass, over as many bits as a key has
// (offset bits and pattern bits next to each other). Keys differ, so the order
// is one. A block ranks 4096 keys in shared memory, a warp 512 of them in order
// (lanes with the same digit by __match_any_sync), and writes them digit by
// digit: runs of 16 keys on average, where single keys were scattered before
// (4.3 M keys: a pass takes
// 12 + 4 + 50 us, 21 + 9 + 60 before).

constexpr uint32_t DS_THREADS = 256;
constexpr uint32_t DS_WARPS = DS_THREADS / 32;
constexpr uint32_t DS_STEPS = kDictSortBlock / DS_THREADS;  // keys per lane

uint32_t dict_sort_blocks(uint32_t n) { return (n + kDictSortBlock - 1) / kDictSortBlock; }

__global__ void __launch_bounds__(DS_THREADS) dict_sort_hist_kernel(const unsigned long long *__restrict__ keys,
                                                                     uint32_t n, uint32_t shift, uint32_t *hist,
                                                                     uint32_t ld) {
    __shared__ uint32_t sh[256];
    sh[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < DS_STEPS; i++) {
        const uint32_t idx = blockIdx.x * kDictSortBlock + i * DS_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&sh[(uint32_t)(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ld + blockIdx.x] = sh[threadIdx.x];
}

// Ranks of `n` keys (at most 512 per warp) by digit: on return rank[i] is key
// i's place in the block's order, and start[d] the first place of digit d.
// cursor: 256 words per warp. The whole block calls (NT threads).
template <uint32_t NT, uint32_t STEPS>
__device__ __forceinline__ void sort_ranks(const unsigned long long (&key)[STEPS], uint32_t first, uint32_t n, uint32_t shift,
                                           uint16_t (*cursor)[256], uint32_t *start, uint32_t *warp_sum,
                                           uint32_t (&rank)[STEPS]) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
    for (uint32_t d = lane; d < 256; d += 32) cursor[warp][d] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < STEPS; i++) {
        const bool valid = first + i * 32 + lane < n;
        const uint32_t vm = __ballot_sync(0xFFFFFFFFu, valid);
        uint32_t d = 0, peers = 0;
        if (valid) {
            d = (uint32_t)(key[i] >> shift) & 255u;
            peers = __match_any_sync(vm, d);
            rank[i] = cursor[warp][d] + __popc(peers & lt);  // in the warp, among the digit's keys
        }
        __syncwarp();
        if (valid && (peers & lt) == 0) cursor[warp][d] += (uint16_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // digit d (thread d): the warps' counts become their first places among the digit's keys
    uint32_t total = 0;
    if (tid < 256) {
#pragma unroll 8
        for (uint32_t w = 0; w < NT / 32; w++) {
            const uint32_t c = cursor[w][tid];
            cursor[w][tid] = (uint16_t)total;
            total += c;
        }
        uint32_t inc = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        if (lane == 31) warp_sum[warp] = inc;
        start[tid] = inc - total;
    }
    __syncthreads();
    if (tid < 256)
        for (uint32_t w = 0; w < warp; w++) start[tid] += warp_sum[w];
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < STEPS; i++) {
        const uint32_t d = (uint32_t)(key[i] >> shift) & 255u;
        if (first + i * 32 + lane < n) rank[i] += start[d] + cursor[warp][d];
    }
}

__global__ void __launch_bounds__(DS_THREADS) dict_sort_scatter_kernel(const unsigned long long *__restrict__ in,
                                                                        unsigned long long *__restrict__ out,
                                                                        uint32_t n, uint32_t shift,
                                                                        const uint32_t *__restrict__ base,
                                                                        const uint32_t *__restrict__ totals,
                                                                        uint32_t ld) {
    __shared__ unsigned long long sorted[kDictSortBlock];
    __shared__ uint16_t cursor[DS_WARPS][256];
    __shared__ uint32_t start[256], to[256], warp_sum[DS_WARPS];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t b0 = blockIdx.x * kDictSortBlock, m = min(n - b0, kDictSortBlock), first = warp * (DS_STEPS * 32);
    unsigned long long key[DS_STEPS];
#pragma unroll
    for (uint32_t i = 0; i < DS_STEPS; i++) {
        const uint32_t j = first + i * 32 + lane;
        key[i] = j < m ? in[b0 + j] : 0ull;
    }
    // the digits' first places in the output: totals before the digit, and the blocks before this one
    to[tid] = block_exclusive_256(totals[tid], warp_sum, nullptr) + base[(size_t)tid * ld + blockIdx.x];
    uint32_t rank[DS_STEPS];
    sort_ranks<DS_THREADS, DS_STEPS>(key, first, m, shift, cursor, start, warp_sum, rank);
#pragma unroll
    for (uint32_t i = 0; i < DS_STEPS; i++)
        if (first + i * 32 + lane < m) sorted[rank[i]] = key[i];
    __syncthreads();
    for (uint32_t j = tid; j < m; j += DS_THREADS) {
        const unsigned long long k = sorted[j];
        const uint32_t d = (uint32_t)(k >> shift) & 255u;
        out[to[d] + j - start[d]] = k;
    }
}

cudaError_t launch_dict_sort(unsigned long long *keys, unsigned long long *tmp, uint32_t n, uint32_t key_bits,
                             uint32_t *hist, uint32_t *totals, unsigned long long **sorted, cudaStream_t st) {
    const uint32_t blocks = dict_sort_blocks(n), ld = scan_ld(blocks);
    uint32_t *counts = hist, *bases = hist + (size_t)256 * ld;
    unsigned long long *src = keys, *dst = tmp;
    for (uint32_t shift = 0; shift < key_bits && n > 1; shift += 8) {
        dict_sort_hist_kernel<<<blocks, DS_THREADS, 0, st>>>(src, n, shift, counts, ld); OL_LAUNCHED();
        cudaError_t e = launch_scan_columns(counts, bases, totals, blocks, 256, ld, st);
        if (e != cudaSuccess) return e;
        dict_sort_scatter_kernel<<<blocks, DS_THREADS, 0, st>>>(src, dst, n, shift, bases, totals, ld); OL_LAUNCHED();
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        std::swap(src, dst);
    }
    *sorted = src;
    return cudaSuccess;
}

// ------------------------------------------------------------------ ids ----

constexpr uint32_t DI_THREADS = 1024;

// One block: per id its count and first output slot (u64 exclusive scan in id
// order), the total, and per unique pattern the start of its light keys.
__device__ __forceinline__ void dict_ids(const DictEmitArgs &a) {
    __shared__ unsigned long long wsum64[DI_THREADS / 32];
    __shared__ uint32_t wsum32[DI_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto count_of_u = [&](uint32_t u) -> uint32_t {
        uint32_t h = a.heavy_of_u[u];
        return h == 0xFFu ? a.light_count[u] : a.heavy_totals[h];
    };
    // ids
    {
        const uint32_t per = (a.n_ids + DI_THREADS - 1) / DI_THREADS;
        const uint32_t lo = min(a.n_ids, tid * per), hi = min(a.n_ids, lo + per);
        unsigned long long sum = 0;
        for (uint32_t i = lo; i < hi; i++) sum += count_of_u(a.u_of_id[i]);
        unsigned long long inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        if (lane == 31) wsum64[warp] = inc;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (uint32_t w = 0; w < DI_THREADS / 32; w++) {
            before += w < warp ? wsum64[w] : 0ull;
            all += wsum64[w];
        }
        unsigned long long run = before + inc - sum;
        for (uint32_t i = lo; i < hi; i++) {
            uint32_t c = count_of_u(a.u_of_id[i]);
            a.id_counts[i] = c;
            a.id_base[i] = run;
            run += c;
        }
        if (tid == 0) *a.total = all;
    }
    __syncthreads();
    // light key starts per unique pattern
    {
        const uint32_t per = (a.n_u + DI_THREADS - 1) / DI_THREADS;
        const uint32_t lo = min(a.n_u, tid * per), hi = min(a.n_u, lo + per);
        uint32_t sum = 0;
        for (uint32_t u = lo; u < hi; u++) sum += a.heavy_of_u[u] == 0xFFu ? a.light_count[u] : 0u;
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        if (lane == 31) wsum32[warp] = inc;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t w = 0; w < warp; w++) before += wsum32[w];
        uint32_t run = before + inc - sum;
        for (uint32_t u = lo; u < hi; u++) {
            a.light_base[u] = run;
            run += a.heavy_of_u[u] == 0xFFu ? a.light_count[u] : 0u;
        }
    }
}

__global__ void __launch_bounds__(DI_THREADS) dict_ids_kernel(DictEmitArgs a) { dict_ids(a); }

// A search with few light keys: one block sorts them (all passes in shared
// memory) and places the ids; with more keys than it takes it leaves them and
// the caller sorts. A 256 KiB text and 40 patterns took 19 launches for this.
__global__ void __launch_bounds__(DI_THREADS) dict_sort_ids_kernel(DictEmitArgs a, unsigned long long *keys, uint32_t key_bits) {
    extern __shared__ __align__(16) uint8_t dyn_smem[];
    constexpr uint32_t STEPS = kDictSortBlock / DI_THREADS;
    unsigned long long *sorted = reinterpret_cast<unsigned long long *>(dyn_smem);
    uint16_t(*cursor)[256] = reinterpret_cast<uint16_t(*)[256]>(sorted + kDictSortBlock);
    __shared__ uint32_t start[256], warp_sum[8];
    const uint32_t lane = threadIdx.x & 31, first = (threadIdx.x >> 5) * (STEPS * 32);
    const uint32_t n = *a.light_n_dev;
    if (n > 1 && n <= kDictSortBlock) {
        unsigned long long key[STEPS];
#pragma unroll
        for (uint32_t i = 0; i < STEPS; i++) {
            const uint32_t j = first + i * 32 + lane;
            key[i] = j < n ? keys[j] : 0ull;
        }
        for (uint32_t shift = 0; shift < key_bits; shift += 8) {
            uint32_t rank[STEPS];
            sort_ranks<DI_THREADS, STEPS>(key, first, n, shift, cursor, start, warp_sum, rank);
#pragma unroll
            for (uint32_t i = 0; i < STEPS; i++)
                if (first + i * 32 + lane < n) sorted[rank[i]] = key[i];
            __syncthreads();
#pragma unroll
            for (uint32_t i = 0; i < STEPS; i++) {
                const uint32_t j = first + i * 32 + lane;
                key[i] = j < n ? sorted[j] : 0ull;
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < STEPS; i++)
            if (first + i * 32 + lane < n) keys[first + i * 32 + lane] = key[i];
    }
    dict_ids(a);
}

cudaError_t launch_dict_sort_ids(const DictEmitArgs &a, unsigned long long *keys, uint32_t key_bits, cudaStream_t st) {
    const size_t smem = kDictSortBlock * 8 + (DI_THREADS / 32) * 256 * 2;
    cudaError_t e = cudaFuncSetAttribute(dict_sort_ids_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    dict_sort_ids_kernel<<<1, DI_THREADS, smem, st>>>(a, keys, key_bits); OL_LAUNCHED();
    return cudaGetLastError();
}

cudaError_t launch_dict_ids(const DictEmitArgs &a, cudaStream_t st) {
    dict_ids_kernel<<<1, DI_THREADS, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

// ----------------------------------------------------------------- emit ----

// One hit into output slot `slot`: a ManyHit {pattern, offset u32}, or the
// (pattern u32, offset u64) pair of arrays. Streaming stores: the emission
// never reads them back.
__device__ __forceinline__ void put_hit(const DictEmitArgs &a, unsigned long long slot, uint32_t id, uint32_t off) {
    if (a.hit_off) {
        __stcs(a.hit_pat + slot, id);
        __stcs(a.hit_off + slot, (unsigned long long)off);
    } else {
        __stcs(&a.hits[slot], make_uint2(id, off));
    }
}

// Heavy hits: a warp expands the 512 bitmap words of one tile of one heavy
// pattern (a tile without hits, known from the match pass's counts, is left at
// once), 128 words a round, four a lane: one scan of the lanes' popcounts gives
// every hit its rank, each lane lists its words' hits in the warp's buffer, and
// the warp writes them to consecutive slots, for one id after the other. Four
// words a lane instead of one make a round's scan, and its longest lane, count
// for four times the hits.
// What bounds it is the writing of 8 bytes a hit: a plain fill runs at 7.1 TB/s
// in one region, but the ids of one unique pattern are as many regions written
// at a time, and a kernel that only stores reaches 4.9 TB/s into 12 of them
// this way. 256 MiB, 10,000 patterns, 7.7 GB of hits: 2.28 ms with one word a
// lane and the block's words read twice, 1.79 ms (4.3 TB/s) now. Blocks of one,
// two or four tiles that list first and write one stretch per id then took 1.81
// to 2.0 ms; listing again for every one to four ids, 1.8 to 3.3 ms.
// The ids of a unique pattern and their first output slots are read once per
// block into shared memory (up to DH_MAX_DUPS of them).
constexpr uint32_t DH_MAX_DUPS = 64;
constexpr uint32_t DH_BUF = 1024;  // hits listed at a time

// A run of n listed hits of one id into consecutive slots, by one warp; four
// stores in flight per lane.
template <bool PAIR>
__device__ __forceinline__ void put_run(const DictEmitArgs &a, unsigned long long slot, uint32_t id, uint32_t text0,
                                        const uint16_t *buf, uint32_t n) {
    uint2 *hits = a.hits + slot;
    uint32_t *pat = a.hit_pat + slot;
    unsigned long long *off = a.hit_off + slot;
    auto put = [&](uint32_t j, uint32_t x) {
        if (PAIR) {
            __stcs(pat + j, id);
            __stcs(off + j, (unsigned long long)x);
        } else {
            __stcs(hits + j, make_uint2(id, x));
        }
    };
    uint32_t j = threadIdx.x & 31;
    for (; j + 96 < n; j += 128) {
        uint32_t x[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) x[i] = text0 + buf[j + 32 * i];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) put(j + 32 * i, x[i]);
    }
    for (; j < n; j += 32) put(j, text0 + buf[j]);
}

template <bool PAIR>
__global__ void __launch_bounds__(DH_THREADS, 6) dict_emit_heavy_kernel(DictEmitArgs a) {
    __shared__ uint32_t dup_id[DH_MAX_DUPS];
    __shared__ unsigned long long dup_base[DH_MAX_DUPS];
    __shared__ uint16_t hit_buf[DH_THREADS / 32][DH_BUF];  // per warp: hit offsets in the tile, in order
    const uint32_t h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x * (DH_THREADS / 32) + warp;
    if (h >= a.plan->n_heavy) return;
    const uint32_t u = a.heavy_u[h];
    const uint32_t d0 = a.dup_start[u], n_dup = a.dup_start[u + 1] - d0;
    const bool cached = n_dup <= DH_MAX_DUPS;
    if (cached && threadIdx.x < n_dup) {
        const uint32_t id = __ldg(a.dup_ids + d0 + threadIdx.x);
        dup_id[threadIdx.x] = id;
        dup_base[threadIdx.x] = a.id_base[id];
    }
    __syncthreads();
    if (tile >= a.n_tiles || a.heavy_counts[(size_t)h * a.ld + tile] == 0) return;  // uniform over the warp
    uint16_t *buf = hit_buf[warp];
    unsigned long long rank = a.heavy_bases[(size_t)h * a.ld + tile];
    constexpr uint32_t kRounds = kDictWordsPerTile / 128;
    const uint4 *col = reinterpret_cast<const uint4 *>(a.bitmap + ((size_t)h * a.n_tiles + tile) * kDictWordsPerTile);
    uint4 words[kRounds];
#pragma unroll
    for (uint32_t r = 0; r < kRounds; r++) words[r] = __ldcs(col + r * 32 + lane);
#pragma unroll
    for (uint32_t r = 0; r < kRounds; r++) {
        const uint32_t x[4] = {words[r].x, words[r].y, words[r].z, words[r].w};
        const uint32_t cnt = __popc(x[0]) + __popc(x[1]) + __popc(x[2]) + __popc(x[3]);
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        const uint32_t all = __shfl_sync(0xFFFFFFFFu, inc, 31);
        // all lanes at once when the buffer holds their hits, else eight lanes
        // (at most 1024 hits) after the other
        const uint32_t step = all <= DH_BUF ? 32 : 8;
        for (uint32_t g = 0; g < 32 && all; g += step) {
            const uint32_t before = g ? __shfl_sync(0xFFFFFFFFu, inc, g - 1) : 0u;
            const uint32_t T = __shfl_sync(0xFFFFFFFFu, inc, g + step - 1) - before;
            if (lane >= g && lane < g + step) {
                uint32_t at = inc - cnt - before;
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    const uint32_t base = (r * 128 + lane * 4 + i) * 32;
                    for (uint32_t bits = x[i]; bits; bits &= bits - 1) buf[at++] = (uint16_t)(base + __ffs(bits) - 1);
                }
            }
            __syncwarp();
            for (uint32_t d = 0; d < n_dup; d++) {
                const uint32_t id = cached ? dup_id[d] : __ldg(a.dup_ids + d0 + d);
                const unsigned long long slot = (cached ? dup_base[d] : a.id_base[id]) + rank;
                const uint32_t n = slot >= a.max_hits ? 0u : (uint32_t)min((unsigned long long)T, a.max_hits - slot);
                put_run<PAIR>(a, slot, id, tile * kDictTile, buf, n);
            }
            __syncwarp();  // the buffer is filled again
            rank += T;
        }
    }
}

__global__ void dict_emit_light_kernel(DictEmitArgs a) {
    const uint32_t n = *a.light_n_dev;
    if (n > a.light_max) return;  // unsorted (dict_sort_ids_kernel): the caller emits once more
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const unsigned long long key = a.light_keys[k];
        const uint32_t u = (uint32_t)(key >> a.off_bits), off = (uint32_t)(key & ((1ull << a.off_bits) - 1));
        const uint32_t rank = k - a.light_base[u];
        const uint32_t d0 = a.dup_start[u], d1 = a.dup_start[u + 1];
        for (uint32_t d = d0; d < d1; d++) {
            const uint32_t id = a.dup_ids[d];
            const unsigned long long slot = a.id_base[id] + rank;
            if (slot < a.max_hits) put_hit(a, slot, id, off);
        }
    }
}

cudaError_t launch_dict_emit(const DictEmitArgs &a, cudaStream_t st) {
    if (a.max_hits == 0) return cudaSuccess;
    if (a.n_heavy && a.n_tiles) {
        dim3 grid((a.n_tiles + DH_THREADS / 32 - 1) / (DH_THREADS / 32), a.n_heavy);
        if (a.hit_off) {
            dict_emit_heavy_kernel<true><<<grid, DH_THREADS, 0, st>>>(a); OL_LAUNCHED();
        } else {
            dict_emit_heavy_kernel<false><<<grid, DH_THREADS, 0, st>>>(a); OL_LAUNCHED();
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (a.light_max) {
        dict_emit_light_kernel<<<(a.light_max + 255) / 256, 256, 0, st>>>(a); OL_LAUNCHED();
        return cudaGetLastError();
    }
    return cudaSuccess;
}

}  // namespace ol
