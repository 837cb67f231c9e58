// Kernel (a)+(b): newline scan fused with per-line classification.
//
// The text is read once and no block ever waits on another:
//   1. parse_stage_kernel: per 16 KiB tile, the newline count (16-byte
//      coalesced vector loads, exact byte SWAR, popc, warp scans), the
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
constexpr uint32_t PT_STEPS = 4;                          // 16-byte pieces per thread
constexpr uint32_t PT_TILE = PT_THREADS * 16 * PT_STEPS;  // 16384
constexpr uint32_t PT_HALO = 256;
constexpr uint32_t PT_LIST = 1024;                        // newline positions listed per round

static_assert(PT_TILE == kParseTile && PT_HALO == kParseHalo, "tile geometry");
static_assert(PT_LIST == kParseSlotCap && kParseFinishTiles % PT_THREADS == 0, "slot and finish geometry");

struct ParseSmem {
    alignas(16) uint8_t text[PT_TILE + PT_HALO + 16];  // +16: word reads may run 3 bytes past
    uint16_t nl[PT_LIST + 1];        // newline positions of the current round, ascending
    uint32_t warp_tot[PT_STEPS][8];  // newline count per (step, warp)
    uint32_t warp_base[PT_STEPS][8];
    uint32_t halo_first;             // first newline in the halo (local), or NONE
    uint32_t tile_nl;                // newlines in the tile
    uint32_t long_idx, long_start;   // the line left to classify_long (long_start: tile-local), or NONE
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

// High bit of every byte of w equal to '|'.
__device__ __forceinline__ uint32_t pipe_bits(uint32_t w) { return zero_bytes(w ^ 0x7C7C7C7Cu); }

// parse_line (crates/oneline-simd/src/line.rs:8-44) for a line held in shared
// memory at tile-local [s, e), e = its '\n' or the text end; the bytes from e
// to e+3 are readable. The prefix is read as alternating runs: a run of '|'
// four bytes per step (byte SWAR), then a run of blanks; it continues only
// while another '|' follows the blanks.
__device__ __forceinline__ uint32_t classify_smem(const uint8_t *t, uint32_t s, uint32_t e, uint32_t &depth_out) {
    uint32_t eff = e;
    while (eff > s && t[eff - 1] == '\r') eff--;
    uint32_t c = s, depth = 0;
    if (s < eff && t[s] == '|') {
        for (;;) {
            // run of '|' (stops at a non-'|' byte, at the latest at eff)
            for (;;) {
                uint32_t other = ~pipe_bits(lds4(t, c)) & 0x80808080u;
                if (other) {
                    uint32_t nb = (__ffs(other) - 8) >> 3;
                    depth += nb;
                    c += nb;
                    break;
                }
                depth += 4;
                c += 4;
            }
            // run of blanks; the prefix goes on only if a '|' follows it
            uint32_t b = c;
            while (b < eff && is_blank(t[b])) b++;
            if (b < eff && t[b] == '|') {
                c = b;
                continue;
            }
            c = b;
            break;
        }
    } else {
        while (c < eff && is_blank(t[c])) c++;
    }
    depth_out = depth;
    if (c >= eff) return KIND_BLANK;
    uint32_t w = lds4(t, c);
    return classify3((uint8_t)w, (uint8_t)(w >> 8), (uint8_t)(w >> 16), eff - c);
}

// Exact '\n' bits (high bit of each byte) of a 16-byte piece at tile-local lo;
// bytes at or past `valid` are cleared.
__device__ __forceinline__ void newline_bits(const uint4 &v, uint32_t lo, uint32_t valid, uint32_t z[4]) {
    const uint32_t NL4 = 0x0A0A0A0Au;
    z[0] = zero_bytes(v.x ^ NL4);
    z[1] = zero_bytes(v.y ^ NL4);
    z[2] = zero_bytes(v.z ^ NL4);
    z[3] = zero_bytes(v.w ^ NL4);
    if (lo + 16 > valid) {
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            uint32_t b0 = lo + 4 * i;  // bytes b0..b0+3; keep those < valid
            uint32_t keep = b0 >= valid ? 0u : (valid - b0 >= 4 ? 4u : valid - b0);
            z[i] &= keep == 4 ? 0xFFFFFFFFu : ((1u << (8 * keep)) - 1u);
        }
    }
}

// The first newline at or past tile t0, or N: the whole warp scans the tiles'
// first newlines, 256 tiles per round trip.
__device__ __forceinline__ uint32_t next_newline(const ParseArgs &a, uint32_t t0) {
    const uint32_t lane = threadIdx.x & 31;
    for (; t0 < a.n_tiles; t0 += 256) {
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

    // 1. Coalesced 16-byte loads: step k covers [t0 + k*4096, +4096), lane-major.
    uint4 v[PT_STEPS];
#pragma unroll
    for (uint32_t k = 0; k < PT_STEPS; k++) v[k] = ld_stream16(a.text + t0 + k * 4096 + tid * 16);
    uint4 vh = make_uint4(0, 0, 0, 0);
    if (tid < PT_HALO / 16) vh = ld_stream16(a.text + t0 + PT_TILE + tid * 16);
    if (tid == 0) {
        sm.halo_first = NONE;
        sm.long_idx = NONE;
        *reinterpret_cast<uint4 *>(&sm.text[PT_TILE + PT_HALO]) = make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (uint32_t k = 0; k < PT_STEPS; k++) *reinterpret_cast<uint4 *>(&sm.text[k * 4096 + tid * 16]) = v[k];
    if (tid < PT_HALO / 16) *reinterpret_cast<uint4 *>(&sm.text[PT_TILE + tid * 16]) = vh;

    // 2. Newline bits and their ranks within the warp: steps (0,1) and (2,3)
    //    packed in 16-bit fields.
    uint32_t nlm[PT_STEPS];  // bit b: byte b of the thread's piece in step k is a newline
    uint32_t cnt[PT_STEPS];
#pragma unroll
    for (uint32_t k = 0; k < PT_STEPS; k++) {
        uint32_t z[4];
        newline_bits(v[k], k * 4096 + tid * 16, valid, z);
        nlm[k] = gather16(z[0], z[1], z[2], z[3]);
        cnt[k] = __popc(nlm[k]);
    }
    uint32_t c01 = cnt[0] | (cnt[1] << 16), c23 = cnt[2] | (cnt[3] << 16);
    uint32_t i01 = c01, i23 = c23;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t1 = __shfl_up_sync(0xFFFFFFFFu, i01, o);
        uint32_t t2 = __shfl_up_sync(0xFFFFFFFFu, i23, o);
        if ((int)lane >= o) {
            i01 += t1;
            i23 += t2;
        }
    }
    const uint32_t r01 = i01 - c01, r23 = i23 - c23;
    if (lane == 31) {
        sm.warp_tot[0][warp] = i01 & 0xFFFF;
        sm.warp_tot[1][warp] = i01 >> 16;
        sm.warp_tot[2][warp] = i23 & 0xFFFF;
        sm.warp_tot[3][warp] = i23 >> 16;
    }
    __syncthreads();  // (a) halo_first initialised, warp totals visible
    if (tid < PT_HALO / 16) {
        const uint32_t lo = PT_TILE + tid * 16;
        uint32_t first = NONE;
        uint32_t zh[4];
        newline_bits(vh, lo, valid, zh);
#pragma unroll
        for (int i = 3; i >= 0; i--)
            if (zh[i]) first = lo + 4 * i + ((__ffs(zh[i]) - 8) >> 3);
        for (int o = 8; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0x0000FFFFu, first, o));
        if (tid == 0) sm.halo_first = first;
    }
    if (warp == 1) {
        // 32 (step, warp) totals in position order: index = k*8 + w.
        uint32_t c = sm.warp_tot[lane >> 3][lane & 7], inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        sm.warp_base[lane >> 3][lane & 7] = inc - c;
        if (lane == 31) sm.tile_nl = inc;
    }
    __syncthreads();  // (b) bases and halo_first visible

    const uint32_t off = tile == 0 ? 1u : 0u;
    const uint32_t n_nl = sm.tile_nl;
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
#pragma unroll
        for (uint32_t k = 0; k < PT_STEPS; k++) {
            uint32_t rr = (k & 1) ? ((k < 2 ? r01 : r23) >> 16) : ((k < 2 ? r01 : r23) & 0xFFFF);
            int32_t rk = (int32_t)(sm.warp_base[k][warp] + rr) - w0;
            if (rk > (int32_t)PT_LIST) continue;
            // one loop over the piece's 16-bit newline mask: the warp runs as
            // many rounds as its busiest lane has newlines in this piece
            uint32_t m = nlm[k];
            while (m) {
                const uint32_t b = __ffs(m) - 1;
                m &= m - 1;
                if (rk >= 0 && rk <= (int32_t)PT_LIST) sm.nl[rk] = (uint16_t)(k * 4096 + tid * 16 + b);
                rk++;
            }
        }
        __syncthreads();  // (c) list ready
        if (STAGE && tid == 0) a.tile_first[tile] = n_nl ? sm.nl[0] : NONE;

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
        __syncthreads();  // (d) the next round may overwrite the list
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
__global__ void __launch_bounds__(PT_THREADS, 6) parse_stage_kernel(ParseArgs a) {
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
// now takes 457 us in all.)
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
__global__ void classify_lines_kernel(const uint8_t *__restrict__ text, uint64_t N, const uint32_t *__restrict__ offsets,
                                      uint32_t L, FlatNode *__restrict__ nodes, uint32_t *__restrict__ depth32) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
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
    parse_redo_kernel<<<std::min(a.n_tiles, 512u), PT_THREADS, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

cudaError_t launch_classify_lines(const uint8_t *text, uint64_t N, const uint32_t *offsets, uint32_t L, FlatNode *nodes,
                                  uint32_t *depth32, cudaStream_t st) {
    if (L == 0) return cudaSuccess;
    classify_lines_kernel<<<(L + 255) / 256, 256, 0, st>>>(text, N, offsets, L, nodes, depth32); OL_LAUNCHED();
    return cudaGetLastError();
}

}  // namespace ol
