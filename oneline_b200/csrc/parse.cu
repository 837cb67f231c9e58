// Kernel (a)+(b): newline scan fused with per-line classification.
//
// The text is read once and no block ever waits on another:
//   1. parse_stage_kernel: per 16 KiB tile, the newline count (asynchronous
//      16-byte copies, exact byte SWAR, popc, warp scans), the
//      newline positions in order, and the classification of every line
//      starting in the tile from shared memory, staged as one word per line
//      in the tile's slot; also the tile's first newline and deepest line;
//   2. the staged lines are written at their line indices:
//      * up to kParseFinishTiles tiles, parse_finish_kernel, one block per
//        tile: it sums the counts of the tiles before its own itself and
//        parses a tile with more lines than a slot holds again, in place;
//      * larger texts: scan_columns_kernel (every tile's first line index),
//        parse_copy_kernel (one warp per tile) and parse_redo_kernel (the
//        tiles with more lines than a slot holds).
// A single pass with a decoupled look-back was measured slower here: the
// look-back chain fell behind the tile rate. A line that runs past the tile
// plus a 256-byte halo (at most one per tile) is classified in step 2 from
// global memory; it ends at the first newline of the tiles after its own.
//
// Replaces crates/oneline-gpu/src/scan.wgsl:20-237 (three passes + a host read
// of the line count) and shader.wgsl:34-134 (one thread per line, byte loads
// from global memory). Semantics: crates/oneline-simd/src/lib.rs:49-66 (line
// starts) and crates/oneline-simd/src/line.rs:8-81 (classification).
#include <cuda_runtime.h>

#include <algorithm>

#include "ol_common.cuh"
#include "ol_kernels.h"

namespace ol {

constexpr uint32_t PT_THREADS = 256;
constexpr uint32_t PT_WARPS = PT_THREADS / 32;
constexpr uint32_t PT_STEPS = 4;                          // 16-byte pieces per thread
constexpr uint32_t PT_TILE = PT_THREADS * 16 * PT_STEPS;  // 16384
constexpr uint32_t PT_HALO = 256;
constexpr uint32_t PT_LIST = 1024;                        // newline positions listed per round

static_assert(PT_TILE == kParseTile && PT_HALO == kParseHalo, "tile geometry");
static_assert(PT_LIST == kParseSlotCap && kParseFinishTiles % PT_THREADS == 0, "slot and finish geometry");

struct ParseSmem {
    alignas(16) uint8_t text[PT_TILE + PT_HALO + 32];  // +32: reads of 16 unaligned bytes may run past
    uint16_t nl[PT_LIST + 1];                 // newline positions of the current round, ascending
    uint32_t warp_tot[PT_WARPS];              // newlines of each warp's 2 KiB
    uint32_t halo_first;                      // first newline in the halo (local), or NONE
    uint32_t long_idx, long_start;  // the line left to classify_long (long_start: tile-local), or NONE
};

// Staged form: a tile's lines as one word each, (start, kind, depth8) or a
// marker, in its slot of PT_LIST words.
constexpr uint32_t kSlotNone = 0xFFFFFFFFu;  // a final '\n' that starts no line
constexpr uint32_t kSlotLong = 1u << 26;     // the line runs past the halo: classify_long
constexpr uint32_t kFirstUnlisted = PT_TILE;  // tile_first of a tile with newlines that were not listed
__device__ __forceinline__ uint32_t slot_word(uint32_t s, uint32_t kind, uint32_t depth) {
    return s | (kind << 15) | (min(depth, 255u) << 18);  // s <= 16384: 15 bits
}

// 4 bytes of shared memory from any byte offset.
__device__ __forceinline__ uint32_t lds4(const uint8_t *base, uint32_t off) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(base) + (off >> 2);
    return __funnelshift_r(w[0], w[1], (off & 3) * 8);
}

// parse_line (crates/oneline-simd/src/line.rs:8-44) for a line held in shared
// memory at tile-local [s, e), e = its '\n' or the text end; the bytes from e
// to e+3 are readable. The prefix is read as alternating runs: a run of '|'
// sixteen bytes per step, then a run of blanks; it continues only while another
// '|' follows the blanks. The usual line, one blank or none before its content,
// needs no look at single bytes.
__device__ __forceinline__ uint32_t classify_smem(const uint8_t *t, uint32_t s, uint32_t e, uint32_t &depth_out) {
    uint32_t eff = e;
    while (eff > s && t[eff - 1] == '\r') eff--;
    uint32_t c = s, depth = 0;
    uint32_t w = lds4(t, c);
    if (s < eff && (w & 0xFFu) == '|') {
        for (;;) {
            // run of '|' (stops at a non-'|' byte, at the latest at eff)
            for (;;) {
                const uint32_t *q = reinterpret_cast<const uint32_t *>(t) + (c >> 2);
                const uint32_t sh = (c & 3) * 8, a0 = q[0], a1 = q[1], a2 = q[2], a3 = q[3], a4 = q[4];
                uint32_t x = __funnelshift_r(a0, a1, sh) ^ 0x7C7C7C7Cu, at = 0;
                if (!x) x = __funnelshift_r(a1, a2, sh) ^ 0x7C7C7C7Cu, at = 4;
                if (!x) x = __funnelshift_r(a2, a3, sh) ^ 0x7C7C7C7Cu, at = 8;
                if (!x) x = __funnelshift_r(a3, a4, sh) ^ 0x7C7C7C7Cu, at = 12;
                if (x) at += (__ffs(x) - 1) >> 3;
                else at = 16;
                depth += at;
                c += at;
                if (at < 16) break;
            }
            // run of blanks; the prefix goes on only if a '|' follows it
            w = lds4(t, c);
            if (c >= eff || !is_blank((uint8_t)w)) break;
            const uint8_t next = (uint8_t)(w >> 8);
            if (c + 1 < eff && next != '|' && !is_blank(next)) {
                c++;
                w >>= 8;
                break;
            }
            uint32_t b = c + 1;
            while (b < eff && is_blank(t[b])) b++;
            c = b;
            if (b < eff && t[b] == '|') continue;
            w = lds4(t, c);
            break;
        }
    } else if (s < eff && is_blank((uint8_t)w)) {
        while (c < eff && is_blank(t[c])) c++;
        w = lds4(t, c);
    }
    depth_out = depth;
    if (c >= eff) return KIND_BLANK;
    return classify3((uint8_t)w, (uint8_t)(w >> 8), (uint8_t)(w >> 16), eff - c);
}

// 32-bit mask of the positions lo .. lo + 31 below n.
__device__ __forceinline__ uint32_t below32(uint32_t n, uint32_t lo) {
    return n <= lo ? 0u : n - lo >= 32 ? 0xFFFFFFFFu : (1u << (n - lo)) - 1u;
}

// Exact newline mask of a 16-byte piece: bit b = byte b. ('\n' is below 0x80, so
// three operations a word tell it from every byte.)
__device__ __forceinline__ uint32_t newline_mask(const uint4 &v) {
    auto bits = [](uint32_t w) {  // high bit of every newline byte
        const uint32_t y = ((w ^ 0x0A0A0A0Au) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
        return ~(y | w) & 0x80808080u;
    };
    return gather16(bits(v.x), bits(v.y), bits(v.z), bits(v.w));
}

// The last tile from t0 on with as many newlines before it as t0 has: the first
// tile with a newline, or the text's last one. The prefix sums ascend, so the
// whole warp narrows the range 32-fold a round trip (four for 4 GiB).
__device__ __forceinline__ uint32_t last_of_equal_base(const ParseArgs &a, uint32_t t0) {
    const uint32_t lane = threadIdx.x & 31, base = a.tile_base[t0];
    uint32_t lo = t0, hi = a.n_tiles;  // tile_base[lo] == base; from hi on it is not, or there is no tile
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, t = lo + lane * step;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, t < hi && a.tile_base[t] == base);
        lo += (31 - __clz(m)) * step;  // (lane 0 always has it)
        hi = min(hi, lo + step);
    }
    return lo;
}

// The first newline at or past tile t0, or N: the whole warp scans the tiles'
// first newlines, 256 tiles in one round trip. Where those have none, a larger
// text's prefix sums (complete before any pass that asks) lead to the tile that
// has one: 256 at a time all the way took 387 us to parse 1 GiB that is one line,
// 219 so.
__device__ __forceinline__ uint32_t next_newline(const ParseArgs &a, uint32_t t0) {
    const uint32_t lane = threadIdx.x & 31;
    while (t0 < a.n_tiles) {
        uint32_t v[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t t = t0 + i * 32 + lane;
            v[i] = t < a.n_tiles ? a.tile_first[t] : NONE;
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, v[i] != NONE);
            if (m) {
                const uint32_t l = __ffs(m) - 1, first = __shfl_sync(0xFFFFFFFFu, v[i], l);
                uint32_t at = (t0 + i * 32 + l) * PT_TILE;
                if (first != kFirstUnlisted) return at + first;
                for (;; at += 32) {  // ends: the tile has a newline
                    const uint32_t nl = __ballot_sync(0xFFFFFFFFu, __ldg(a.text + at + lane) == '\n');
                    if (nl) return at + __ffs(nl) - 1;
                }
            }
        }
        t0 += 256;
        if (a.n_tiles > kParseFinishTiles && t0 < a.n_tiles) t0 = last_of_equal_base(a, t0);
    }
    return (uint32_t)a.text_len;
}

// Line idx, which starts at s in `tile` and runs past the tile's halo: its
// bytes come from global memory. The whole warp calls; lane 0 classifies.
__device__ __forceinline__ void classify_long(const ParseArgs &a, uint32_t tile, uint32_t idx, uint32_t s) {
    const uint32_t e = next_newline(a, tile + 1);
    if ((threadIdx.x & 31) != 0 || idx >= a.line_cap) return;
    const uint8_t *t = a.text;
    const FlatNode nd = classify_line(s, e, [t](uint32_t p) -> uint8_t { return __ldg(t + p); });
    a.kinds[idx] = (uint8_t)nd.kind;
    a.depth8[idx] = (uint8_t)min(nd.depth, 255u);
    if (nd.kind != KIND_BLANK) atomicMax(&a.stats->max_content_depth, nd.depth);
}

// One tile: the block loads tile b, lists its newlines in position order
// (warp popc scans) and classifies every line that starts after one of them
// (plus line 0 for tile 0) from shared memory. Consecutive threads take
// consecutive lines. A line that runs past the tile plus a 256-byte halo is
// left to classify_long.
//   STAGE: the tile's newline count goes to tile_count and its lines, by
//     tile-local rank, to its slot (a tile with more lines than a slot holds
//     is flagged for the other form instead);
//   else: nl_base newlines come before the tile, and offsets, kinds and
//     depth8 are written in place.
template <bool STAGE>
__device__ __forceinline__ void parse_tile(const ParseArgs &a, ParseSmem &sm, uint32_t tile, uint32_t nl_base) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t t0 = (uint64_t)tile * PT_TILE;
    const uint64_t N = a.text_len;
    // bytes of this tile (and halo) that belong to the text
    const uint32_t valid = N - t0 >= PT_TILE + PT_HALO ? PT_TILE + PT_HALO : (uint32_t)(N - t0);

    // 1. The tile and its halo into shared memory, 16 bytes a copy, without a stop
    //    in registers: the pass needs 32 of them and runs eight blocks an SM
    //    (through registers six: 113 against 101 us per 256 MiB).
#pragma unroll
    for (uint32_t k = 0; k < PT_STEPS; k++) cp_async16(&sm.text[k * 4096 + tid * 16], a.text + t0 + k * 4096 + tid * 16);
    if (tid < PT_HALO / 16) cp_async16(&sm.text[PT_TILE + tid * 16], a.text + t0 + PT_TILE + tid * 16);
    if (tid == 0) {
        sm.long_idx = NONE;
        *reinterpret_cast<uint4 *>(&sm.text[PT_TILE + PT_HALO]) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(&sm.text[PT_TILE + PT_HALO + 16]) = make_uint4(0, 0, 0, 0);
    }
    cp_async_wait();
    __syncthreads();  // (a) text in shared memory

    // 2. Newlines of the thread's 64 consecutive bytes, and their rank: one count
    //    and one scan per thread, and ranks in thread order. (Four strided pieces
    //    a thread, straight from the loads, took twice the instructions: a scan
    //    each, and a list of 32 totals.)
    const uint32_t mine = tid * 64;
    uint32_t m0, m1;  // bit b: byte mine + b, mine + 32 + b
    {
        const uint4 *own = reinterpret_cast<const uint4 *>(&sm.text[mine]);
        m0 = newline_mask(own[0]) | (newline_mask(own[1]) << 16);
        m1 = newline_mask(own[2]) | (newline_mask(own[3]) << 16);
    }
    if (valid < PT_TILE) {  // uniform: the last tile
        m0 &= below32(valid, mine);
        m1 &= below32(valid, mine + 32);
    }
    const uint32_t cnt = __popc(m0) + __popc(m1);
    uint32_t rank = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, rank, o);
        if ((int)lane >= o) rank += t;
    }
    if (lane == 31) sm.warp_tot[warp] = rank;
    rank -= cnt;
    if (warp == 0) {  // the halo's first newline
        uint32_t m = tid < PT_HALO / 16 ? newline_mask(*reinterpret_cast<const uint4 *>(&sm.text[PT_TILE + tid * 16])) : 0u;
        const uint32_t lo = PT_TILE + tid * 16;
        if (valid < PT_TILE + PT_HALO) m &= below32(valid, lo);
        const uint32_t first = __reduce_min_sync(0xFFFFFFFFu, m ? lo + __ffs(m) - 1 : NONE);
        if (tid == 0) sm.halo_first = first;
    }
    __syncthreads();  // (b) totals and halo_first visible
    const uint32_t t8 = lane < PT_WARPS ? sm.warp_tot[lane] : 0u;
    const uint32_t n_nl = __reduce_add_sync(0xFFFFFFFFu, t8);
    rank += __reduce_add_sync(0xFFFFFFFFu, lane < warp ? t8 : 0u);

    const uint32_t off = tile == 0 ? 1u : 0u;
    const uint32_t n_lines = n_nl + off;
    if (STAGE) {
        const bool over = n_lines > a.slot_cap;
        if (tid == 0) {
            a.tile_count[tile] = n_nl;
            a.slot_over[tile] = over ? 1 : 0;
            if (over || n_lines == 0) a.tile_first[tile] = over ? kFirstUnlisted : NONE;
        }
        if (over) return;  // uniform
    }
    const uint32_t halo_first = sm.halo_first;
    uint32_t *slot = STAGE ? a.slot + (size_t)tile * a.slot_cap : nullptr;
    uint32_t my_max = 0;

    // Lines are classified in rounds of PT_LIST (one round unless the tile
    // holds more than 1024 newlines): list the round's newline positions, then
    // classify and write the round's lines.
    for (uint32_t r0 = 0; r0 < n_lines; r0 += PT_LIST) {
        const int32_t w0 = (int32_t)r0 - (int32_t)off;  // rank of nl[0]
        int32_t rk = (int32_t)rank - w0;
        if (rk <= (int32_t)PT_LIST && rk + (int32_t)cnt > 0) {  // some of the thread's are in the round
            auto list = [&](uint32_t m, uint32_t lo) {  // the warp runs as many rounds as its busiest lane has newlines
                for (; m; m &= m - 1, rk++)
                    if (STAGE || (rk >= 0 && rk <= (int32_t)PT_LIST)) sm.nl[rk] = (uint16_t)(lo + __ffs(m) - 1);
            };
            list(m0, mine);
            list(m1, mine + 32);
        }
        __syncthreads();  // (c) list ready
        if (STAGE && tid == 0) a.tile_first[tile] = n_nl ? sm.nl[off] : NONE;

        const uint32_t r_end = min(n_lines, r0 + PT_LIST);
        for (uint32_t j = r0 + tid; j < r_end; j += PT_THREADS) {
            int32_t q = (int32_t)j - (int32_t)off;  // newline that precedes the line (-1: none)
            uint32_t s = q < 0 ? 0u : sm.nl[q - w0] + 1u;  // tile-local
            if (s >= valid) {  // the final '\n' starts no line
                if (STAGE) slot[j] = kSlotNone;
                continue;
            }
            uint32_t idx = nl_base + j + 1 - off;
            if (!STAGE) {
                if (idx >= a.line_cap) {
                    atomicOr(&a.stats->error, OL_DEVERR_CAPACITY);
                    continue;
                }
                a.offsets[idx] = (uint32_t)t0 + s;
            }
            uint32_t e;
            if ((uint32_t)(q + 1) < n_nl) e = sm.nl[q + 1 - w0];
            else if (halo_first != NONE) e = halo_first;
            else if (valid < PT_TILE + PT_HALO) e = valid;  // the text ends in the staged bytes
            else {
                // runs past the halo (the tile's last line)
                if (STAGE) {
                    slot[j] = s | kSlotLong;
                } else {
                    sm.long_idx = idx;
                    sm.long_start = s;
                }
                continue;
            }
            uint32_t depth;
            uint32_t kind = classify_smem(sm.text, s, e, depth);
            if (STAGE) {
                slot[j] = slot_word(s, kind, depth);
            } else {
                a.kinds[idx] = (uint8_t)kind;
                a.depth8[idx] = (uint8_t)min(depth, 255u);
            }
            if (kind != KIND_BLANK) my_max = max(my_max, depth);
        }
        // (d) the next round overwrites the list; in place, long_idx and long_start are complete
        if (!STAGE || r0 + PT_LIST < n_lines) __syncthreads();
    }
    my_max = __reduce_max_sync(0xFFFFFFFFu, my_max);
    if (STAGE) {
        if (lane == 0) a.tile_depth[tile * 8 + warp] = (uint16_t)my_max;  // at most the staged bytes: below 2^16
    } else {
        if (warp == 0 && sm.long_idx != NONE) classify_long(a, tile, sm.long_idx, (uint32_t)t0 + sm.long_start);
        if (lane == 0 && my_max) atomicMax(&a.stats->max_content_depth, my_max);
    }
}

// Pass 1: every tile counts its newlines and stages its lines; the block of
// tile 0 resets the document's counters, which only pass 2 adds to. Block b
// first asks L2 to prefetch the tile kPrefetchTilesAhead further on (when this
// launch covers it), which a block that starts soon will read.
__global__ void __launch_bounds__(PT_THREADS, 8) parse_stage_kernel(ParseArgs a) {
    __shared__ ParseSmem sm;
    const uint32_t tile = a.first_tile + blockIdx.x;
    if (threadIdx.x == 0 && blockIdx.x + kPrefetchTilesAhead < gridDim.x)  // inside this launch's tiles
        prefetch_l2(a.text + (uint64_t)(tile + kPrefetchTilesAhead) * kParseTile, kParseTile);
    if (tile == 0 && threadIdx.x < sizeof(DocStats) / 4) reinterpret_cast<uint32_t *>(a.stats)[threadIdx.x] = 0;
    parse_tile<true>(a, sm, tile, 0);
}

// A staged line word at line index idx: offsets, kinds and depth8. A long line
// (kSlotLong) is left to the caller, which gets its start in `at`.
__device__ __forceinline__ void put_line(const ParseArgs &a, uint32_t t0, uint32_t w, uint32_t idx, uint2 &at) {
    if (w == kSlotNone) return;
    if (idx >= a.line_cap) {
        atomicOr(&a.stats->error, OL_DEVERR_CAPACITY);
        return;
    }
    const uint32_t s = t0 + (w & 0x7FFFu);
    a.offsets[idx] = s;
    if (w & kSlotLong) {
        at = make_uint2(idx, s);
        return;
    }
    a.kinds[idx] = (uint8_t)((w >> 15) & 7u);
    a.depth8[idx] = (uint8_t)((w >> 18) & 0xFFu);
}

// The deepest staged line of a tile.
__device__ __forceinline__ uint32_t tile_depth_of(const ParseArgs &a, uint32_t tile) {
    const uint4 d = reinterpret_cast<const uint4 *>(a.tile_depth)[tile];
    const uint32_t m = __vmaxu2(__vmaxu2(d.x, d.y), __vmaxu2(d.z, d.w));
    return max(m & 0xFFFFu, m >> 16);
}

// L = 1 + newlines before the last byte, from the last tile's.
__device__ __forceinline__ void put_line_count(const ParseArgs &a, uint32_t nl_base, uint32_t n_nl) {
    a.stats->line_count = 1u + nl_base + n_nl - (a.text[a.text_len - 1] == '\n');
}

// Pass 2 of a text of at most kParseFinishTiles tiles, block b for tile b. The
// counts before it are at most 4 KiB of L2 reads, all in flight at once, so
// the scan needs no launch of its own, nor do the dense tiles and long lines:
// two launches for the whole parse instead of five. At 1 MiB (64 tiles) the
// passes after the stage pass took 14.6 us of kernels and four launches of
// 3.9 us each on the host.
__global__ void __launch_bounds__(PT_THREADS, 6) parse_finish_kernel(ParseArgs a) {
    __shared__ ParseSmem sm;
    __shared__ uint32_t warp_sum[PT_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
    uint32_t before = 0;
#pragma unroll
    for (uint32_t i = 0; i < kParseFinishTiles / PT_THREADS; i++) {
        const uint32_t t = i * PT_THREADS + tid;
        before += t < tile ? a.tile_count[t] : 0u;
    }
    const bool over = a.slot_over[tile];
    const uint32_t depth = tile_depth_of(a, tile);
    const uint32_t off = tile == 0 ? 1u : 0u, n_nl = a.tile_count[tile], n_lines = n_nl + off;
    const uint32_t *slot = a.slot + (size_t)tile * a.slot_cap;
    uint32_t ws[kParseSlotCap / PT_THREADS];
#pragma unroll
    for (uint32_t r = 0; r < kParseSlotCap / PT_THREADS; r++) {
        const uint32_t j = r * PT_THREADS + tid;
        ws[r] = !over && j < n_lines ? slot[j] : kSlotNone;
    }
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    if (lane == 0) warp_sum[warp] = before;
    __syncthreads();
    uint32_t nl_base = 0;
#pragma unroll
    for (uint32_t w = 0; w < PT_THREADS / 32; w++) nl_base += warp_sum[w];
    if (tid == 0 && tile == a.n_tiles - 1) put_line_count(a, nl_base, n_nl);
    if (over) {  // uniform: more lines than the slot holds
        parse_tile<false>(a, sm, tile, nl_base);
        return;
    }
    if (tid == 0 && depth) atomicMax(&a.stats->max_content_depth, depth);
    uint2 at = make_uint2(NONE, 0);
#pragma unroll
    for (uint32_t r = 0; r < kParseSlotCap / PT_THREADS; r++)
        put_line(a, tile * PT_TILE, ws[r], nl_base + r * PT_THREADS + tid + 1 - off, at);
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, at.x != NONE);
    if (m) {
        const uint32_t l = __ffs(m) - 1;
        classify_long(a, tile, __shfl_sync(0xFFFFFFFFu, at.x, l), __shfl_sync(0xFFFFFFFFu, at.y, l));
    }
}

// Pass 2 of a larger text, after the scan of the counts: one warp per tile.
constexpr uint32_t PC_TILES = 8;    // tiles per block
constexpr uint32_t PC_FLIGHT = 4;   // 12 (one round trip a tile) measured 62 against 54 us per GiB
__global__ void __launch_bounds__(256) parse_copy_kernel(ParseArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x * PC_TILES + (threadIdx.x >> 5);
    if (tile >= a.n_tiles) return;
    const uint32_t off = tile == 0 ? 1u : 0u;
    const uint32_t n_nl = a.tile_count[tile], nl_base = a.tile_base[tile];
    const uint32_t n_lines = n_nl + off;
    if (tile == a.n_tiles - 1 && lane == 0) put_line_count(a, nl_base, n_nl);
    if (a.slot_over[tile]) return;  // parse_redo_kernel
    const uint32_t *slot = a.slot + (size_t)tile * a.slot_cap;
    uint2 at = make_uint2(NONE, 0);
    for (uint32_t j0 = 0; j0 < n_lines; j0 += PC_FLIGHT * 32) {
        uint32_t ws[PC_FLIGHT];  // independent loads in flight per lane
#pragma unroll
        for (uint32_t r = 0; r < PC_FLIGHT; r++) {
            const uint32_t j = j0 + r * 32 + lane;
            ws[r] = j < n_lines ? __ldg(slot + j) : kSlotNone;
        }
#pragma unroll
        for (uint32_t r = 0; r < PC_FLIGHT; r++)
            put_line(a, tile * PT_TILE, ws[r], nl_base + j0 + r * 32 + lane + 1 - off, at);
    }
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, at.x != NONE);
    if (m) {
        const uint32_t l = __ffs(m) - 1;
        classify_long(a, tile, __shfl_sync(0xFFFFFFFFu, at.x, l), __shfl_sync(0xFFFFFFFFu, at.y, l));
    }
}

// Pass 3 of a larger text: the tiles with more lines than a slot holds, parsed
// again in place now that their first line index is known, and the document's
// deepest line. Block b looks through tiles b, b + grid, ...: one atomic a
// block. (One a warp and tile of the stage pass, all on one address, made that
// pass 438 us per GiB in some processes and 704 us in others, on one box; it
// now takes 457 us in all.) The grid is as many blocks as run at a time: a dense
// tile is a long chain of rounds (32 MiB of newlines: 360 us with 512 blocks, 282
// so; of two-byte lines 164 and 132).
constexpr uint32_t kRedoGrid = 148 * 6;
__global__ void __launch_bounds__(PT_THREADS, 6) parse_redo_kernel(ParseArgs a) {
    __shared__ ParseSmem sm;
    __shared__ uint32_t list[PT_THREADS], n_list, deepest;
    if (threadIdx.x == 0) deepest = 0;
    uint32_t depth = 0;
    for (uint32_t i0 = blockIdx.x; i0 < a.n_tiles; i0 += gridDim.x * PT_THREADS) {
        if (threadIdx.x == 0) n_list = 0;
        __syncthreads();
        const uint64_t tile = i0 + (uint64_t)gridDim.x * threadIdx.x;
        if (tile < a.n_tiles) {
            if (a.slot_over[tile]) list[atomicAdd(&n_list, 1u)] = (uint32_t)tile;
            else depth = max(depth, tile_depth_of(a, (uint32_t)tile));
        }
        __syncthreads();
        const uint32_t n = n_list;
        for (uint32_t i = 0; i < n; i++) {
            parse_tile<false>(a, sm, list[i], a.tile_base[list[i]]);
            __syncthreads();  // shared memory is reused by the next tile
        }
    }
    depth = __reduce_max_sync(0xFFFFFFFFu, depth);
    if ((threadIdx.x & 31) == 0) atomicMax(&deepest, depth);
    __syncthreads();
    if (threadIdx.x == 0 && deepest) atomicMax(&a.stats->max_content_depth, deepest);
}

// FlatNode of every line from the text and a complete offsets array (used for
// GpuParser::parse(input, offsets) and to materialise nodes of a resident
// document). One thread per line, bytes from global memory (read-only path).
// With `count`, there are *count lines, at most L.
__global__ void classify_lines_kernel(const uint8_t *__restrict__ text, uint64_t N, const uint32_t *__restrict__ offsets,
                                      uint32_t L, const uint32_t *__restrict__ count, FlatNode *__restrict__ nodes,
                                      uint32_t *__restrict__ depth32) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (count) L = min(L, *count);
    if (i >= L) return;
    uint32_t s = offsets[i];
    uint32_t last_end = text[N - 1] == '\n' ? (uint32_t)(N - 1) : (uint32_t)N;
    uint32_t e = i + 1 < L ? offsets[i + 1] - 1 : last_end;
    FlatNode nd = classify_line(s, e, [text](uint32_t p) -> uint8_t { return __ldg(text + p); });
    if (nodes) nodes[i] = nd;
    if (depth32) depth32[i] = nd.kind == KIND_BLANK ? NONE : nd.depth;
}

// ------------------------------------------------------------------ host ----

cudaError_t launch_parse(const ParseArgs &a, cudaStream_t st) {
    if (a.n_tiles == 0) return cudaSuccess;
    cudaError_t e = launch_parse_tiles(a, 0, a.n_tiles, st);
    return e == cudaSuccess ? launch_parse_end(a, st) : e;
}

cudaError_t launch_parse_tiles(const ParseArgs &a, uint32_t t0, uint32_t t1, cudaStream_t st) {
    if (a.slot_cap != kParseSlotCap) return cudaErrorInvalidValue;  // a slot is listed in one round
    t1 = std::min(t1, a.n_tiles);
    if (t0 >= t1) return cudaSuccess;
    ParseArgs r = a;
    r.first_tile = t0;
    parse_stage_kernel<<<t1 - t0, PT_THREADS, 0, st>>>(r); OL_LAUNCHED();
    return cudaGetLastError();
}

cudaError_t launch_parse_end(const ParseArgs &a, cudaStream_t st) {
    if (a.n_tiles == 0) return cudaSuccess;
    if (a.n_tiles <= kParseFinishTiles) {
        parse_finish_kernel<<<a.n_tiles, PT_THREADS, 0, st>>>(a); OL_LAUNCHED();
        return cudaGetLastError();
    }
    cudaError_t e = launch_scan_columns(a.tile_count, a.tile_base, nullptr, a.n_tiles, 1, scan_ld(a.n_tiles), st);
    if (e != cudaSuccess) return e;
    parse_copy_kernel<<<(a.n_tiles + PC_TILES - 1) / PC_TILES, 256, 0, st>>>(a); OL_LAUNCHED();
    parse_redo_kernel<<<std::min(a.n_tiles, kRedoGrid), PT_THREADS, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

cudaError_t launch_classify_lines(const uint8_t *text, uint64_t N, const uint32_t *offsets, uint32_t L, FlatNode *nodes,
                                  uint32_t *depth32, cudaStream_t st, const uint32_t *count) {
    if (L == 0) return cudaSuccess;
    classify_lines_kernel<<<(L + 255) / 256, 256, 0, st>>>(text, N, offsets, L, count, nodes, depth32); OL_LAUNCHED();
    return cudaGetLastError();
}

}  // namespace ol
