// Kernel (d): substring search, every overlapping occurrence, ascending.
//
// Up to eight patterns are searched in one pass over the text; CTA b owns the
// 16 KiB tile b and stages it, plus a halo of (longest pattern - 1) bytes, in
// shared memory with asynchronous 16-byte copies (in the stage pass, after asking
// L2 to prefetch the tile kPrefetchTilesAhead further on, which a block that
// starts soon will read). Every 16-byte piece is compared with each pattern of
// up to 4 bytes at all sixteen starts at once (byte SWAR on the piece shifted by
// 1, 2 and 3 bytes, built once for all patterns), which decides it; of 5 to 7 bytes
// the first two are looked for like that, and the pieces that have them are queued
// and compared whole. Longer patterns are looked for by their anchor words: four
// consecutive 4-byte words of the pattern, one of which lies on a 4-byte boundary
// of the text in every occurrence. A shared hash map of those words is tested once
// per aligned text word, for all patterns together; a word found there gives the
// one start it can belong to, which is queued per warp and verified word by word,
// 32 at a time, one per lane. Where in the pattern the anchor words lie is chosen
// by how rare such words are in text. A run c^m is decided from the masks of c at 64 positions; any other
// pattern whose anchor words cannot but be runs of one byte (which made nearly
// every piece of indented text a candidate) is looked for by its rarest four
// bytes, at all starts like a short one. An occurrence must end inside the text (the
// buffer is zero padded: a pattern ending in NUL must not match the padding).
// Recomputing form, three launches, no block waits on another:
//   1. search_count_kernel: matches per (tile, pattern);
//   2. scan_columns_kernel: per pattern, the first output slot of every tile
//      and the total;
//   3. search_write_kernel: tiles with matches recompute them for the patterns
//      that have some and write every pattern's first max_out offsets in
//      ascending order, the whole block writing one contiguous range per
//      pattern: no host sort, and a truncated result is the lowest max_out
//      offsets.
// Patterns longer than kSearchMaxStagedPattern run alone (np = 1) and read
// their halo and verification bytes from global memory.
//
// Semantics: crates/oneline-simd/src/search.rs:88-114 (every overlapping
// occurrence, ascending). Replaces crates/oneline-gpu/src/search.wgsl:101-173
// (4-byte window filter, slot atomics, host sort).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "ol_common.cuh"
#include "ol_kernels.h"

namespace ol {

constexpr uint32_t SR_THREADS = 256;
constexpr uint32_t SR_STEPS = 4;
constexpr uint32_t SR_PIECES = SR_THREADS * SR_STEPS;  // 16-byte pieces per tile
constexpr uint32_t SR_QCAP = 96;                       // per-warp queue of starts to verify
static_assert(SR_THREADS * 16 * SR_STEPS == kSearchTile, "search tile");

// Patterns of at least kAnchorMin bytes are filtered by their anchor words:
// every occurrence at start s covers the 4-byte-aligned text word at
// a = 4 * floor((s + r0) / 4) + 4 (1 <= a - s - r0 <= 4, and a + 4 <= s + r0 + 8
// <= s + len), which equals the pattern's bytes [a - s, a - s + 4): one of four
// anchor words, r = a - s = r0 + 1 .. r0 + 4. Each start has one such word, and
// a text word that equals anchor r can only belong to the start a - r. A 2^15-bit
// map of the anchors' hashes, shared by all patterns of the launch, tells which
// aligned text words may be one; those are compared exactly.
constexpr uint32_t kAnchorMin = 8;
constexpr uint32_t kAnchorBits = 15;
constexpr uint32_t kAnchorReach = 240;  // largest r0 (or window offset): at most 16 pieces past the tile
constexpr uint32_t kPoorAnchor = 20;    // anchor_place: a word of this weight is mostly one byte repeated
constexpr uint32_t kRunMask = 48;       // runs of up to this length are decided from the masks of four pieces

__host__ __device__ __forceinline__ uint32_t anchor_hash(uint32_t w) {
    return (w * 0x9E3779B1u) >> (32 - kAnchorBits);
}

struct alignas(16) PatMeta {  // a SearchPatMeta, copied from the kernel parameters 16 bytes a lane
    uint4 pre;  // bytes 0..3 of the pattern, each replicated into a word (unused ones 0); of a window pattern: its
                // rarest two so, and the window r0..r0 + 3 as a word
    uint4 anc;  // anchor words r = r0 + 1 .. r0 + 4
    uint32_t len;
    uint32_t r0;
    uint32_t last4;  // the last four bytes (len >= 4)
    uint32_t pair;   // window patterns: the place of those two in the window
};
static_assert(sizeof(PatMeta) == 48 && sizeof(SearchPatMeta) == 48, "copied as three 16-byte pieces");

struct SearchSmem {
    alignas(16) uint8_t text[kSearchTile + kSearchMaxStagedPattern + 16];  // stage pass: output staging after use
    uint32_t anchor_map[(1u << kAnchorBits) / 32];
    uint32_t queue[SR_THREADS / 32][SR_QCAP];  // (pattern << 16) | start, per warp
    PatMeta pat[kSearchMaxPatterns];
    const uint8_t *ptr[kSearchMaxPatterns];
    uint32_t count[kSearchMaxPatterns];
    uint32_t active;  // stage pass: patterns with matches in this tile (bit mask)
};

// 4 bytes of the tile-local text from any offset: from shared memory when
// staged, else from global memory (the buffer is padded).
__device__ __forceinline__ uint32_t text4(const SearchArgs &a, const SearchSmem &sm, uint32_t off, bool staged, uint64_t t0) {
    const uint8_t *base = staged ? sm.text : a.text + t0;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(base) + (off >> 2);
    return __funnelshift_r(w[0], w[1], (off & 3) * 8);
}

// Clears the starts of the piece at tile-local lo that lie past N - m (they
// cannot match; the zero padding must not complete a pattern ending in NUL).
__device__ __forceinline__ void keep_valid_starts(uint64_t N, uint32_t m, uint64_t t0, uint32_t lo, uint32_t &c0,
                                                  uint32_t &c1, uint32_t &c2, uint32_t &c3) {
    const int64_t last_ok = (int64_t)N - (int64_t)m - (int64_t)t0;
    uint32_t keep[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int64_t room = last_ok - (int64_t)(lo + 4 * i) + 1;  // valid starts in word i
        keep[i] = room <= 0 ? 0u : (room >= 4 ? 0xFFFFFFFFu : ((1u << (8 * room)) - 1u));
    }
    c0 &= keep[0];
    c1 &= keep[1];
    c2 &= keep[2];
    c3 &= keep[3];
}

// Whether pattern pm (at least eight bytes) occurs at tile start s: its last
// four bytes first (patterns that begin with a run match a long way into
// another run), then four at a time.
__device__ __forceinline__ bool verify_start(const SearchArgs &a, const SearchSmem &sm, uint32_t p, uint32_t s,
                                             bool staged, uint64_t t0) {
    const PatMeta &pm = sm.pat[p];
    const uint32_t m = pm.len;
    if (t0 + s + m > a.text_len) return false;
    if (text4(a, sm, s + m - 4, staged, t0) != pm.last4) return false;
    const uint32_t *pw = reinterpret_cast<const uint32_t *>(sm.ptr[p]);  // 16-byte aligned
    for (uint32_t j = 0; j + 4 < m; j += 4)
        if (text4(a, sm, s + j, staged, t0) != pw[j >> 2]) return false;
    return true;
}

// Loads tile b (plus the halo) into shared memory, and from the kernel
// parameters the anchor map (warp 0), the pattern table (warp 1) and the pattern
// pointers (warp 2): one warp with all three, eight lanes each copying a table
// entry word by word, kept the block waiting (256 MiB, 8 patterns: 119.8 against
// 116.5 us). The caller's __syncthreads publishes them.
__device__ __forceinline__ void load_tile(const SearchArgs &a, SearchSmem &sm, uint64_t t0) {
    const uint32_t tid = threadIdx.x;
    const bool staged = a.halo <= kSearchMaxStagedPattern;
#pragma unroll
    for (uint32_t k = 0; k < SR_STEPS; k++) cp_async16(&sm.text[k * 4096 + tid * 16], a.text + t0 + k * 4096 + tid * 16);
    const uint32_t halo = staged ? a.halo : 0u;
    for (uint32_t o = tid * 16; o < halo; o += SR_THREADS * 16)
        cp_async16(&sm.text[kSearchTile + o], a.text + t0 + kSearchTile + o);
    // 16 bytes past the halo: zeros when staged; unstaged, the bytes right
    // after the tile (the filter looks 3 bytes ahead; the text is padded)
    if (tid == 0)
        *reinterpret_cast<uint4 *>(&sm.text[kSearchTile + halo]) =
            staged ? make_uint4(0, 0, 0, 0) : ld_stream16(a.text + t0 + kSearchTile);
    if (tid < 32) {
        uint4 *am = reinterpret_cast<uint4 *>(sm.anchor_map);
        for (uint32_t o = tid; o < (1u << kAnchorBits) / 128; o += 32) am[o] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        if (tid < a.n_anchor) {
            const uint32_t h = a.anchor_hash[tid];
            atomicOr(&sm.anchor_map[h >> 5], 1u << (h & 31));
        }
    } else if (tid < 64) {
        const uint32_t i = tid - 32;
        if (i < a.np * 3) reinterpret_cast<uint4 *>(sm.pat)[i] = reinterpret_cast<const uint4 *>(a.meta)[i];
    } else if (tid < 96) {
        const uint32_t i = tid - 64;
        if (i < a.np) {
            sm.ptr[i] = a.pat[i] ? a.pat[i] : a.pat_bytes + a.pat_at[i];
            sm.count[i] = 0;
        }
    }
    cp_async_wait();
}

// Whether one of the sixteen bytes is zero, without telling which.
__device__ __forceinline__ bool any_zero_byte(const uint32_t (&x)[4]) {
    uint32_t z = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) z |= (x[i] - 0x01010101u) & ~x[i];
    return (z & 0x80808080u) != 0;
}

// The starts of pattern p (5 to 7 bytes) in a piece, whole: its first four bytes at
// the sixteen starts at once, then the last four at the starts that are left.
__device__ __forceinline__ uint32_t mid_starts(const SearchArgs &a, const SearchSmem &sm, uint32_t p, uint32_t piece,
                                            bool tail_tile, uint64_t t0) {
    const uint32_t *t = reinterpret_cast<const uint32_t *>(&sm.text[piece * 16]), m = sm.pat[p].len;
    const uint4 pre = sm.pat[p].pre;
    uint32_t c[4], g, ok = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
        c[i] = zero_bytes((t[i] ^ pre.x) | (__funnelshift_r(t[i], t[i + 1], 8) ^ pre.y) |
                          (__funnelshift_r(t[i], t[i + 1], 16) ^ pre.z) | (__funnelshift_r(t[i], t[i + 1], 24) ^ pre.w));
    if (tail_tile) keep_valid_starts(a.text_len, m, t0, piece * 16, c[0], c[1], c[2], c[3]);
    for (g = gather16(c[0], c[1], c[2], c[3]); g; g &= g - 1) {
        const uint32_t b = __ffs(g) - 1;
        if (text4(a, sm, piece * 16 + b + m - 4, true, t0) == sm.pat[p].last4) ok |= 1u << b;
    }
    return ok;
}

// Adds the match at tile start `start` to a pattern's masks, 16 starts each
// (verified starts of one piece may come from several lanes).
__device__ __forceinline__ void set_match(uint16_t *masks, uint32_t start) {
    atomicOr(reinterpret_cast<uint32_t *>(masks) + (start >> 5), 1u << (start & 31));
}

// The starts of run pattern p (one byte m times) in a lane's piece: the mask of
// the sixteen, from e, the piece's mask of the byte. Longer runs than the masks
// of four pieces show: their candidates are next to each other and in one run,
// whose end is looked for once for all of them, sixteen bytes at a time.
__device__ __forceinline__ uint32_t run_starts(const SearchArgs &a, const SearchSmem &sm, uint32_t p, uint32_t e, uint32_t piece,
                                            uint64_t t0) {
    const uint32_t lane = threadIdx.x & 31, m = sm.pat[p].len, c = sm.pat[p].pre.x;
    // the masks of the three pieces after mine (lanes 0..2 have those after the warp's)
    uint32_t more = 0;
    if (lane < 3) more = eq_mask16(*reinterpret_cast<const uint4 *>(&sm.text[(piece + 32) * 16]), c);
    unsigned long long x = e;
#pragma unroll
    for (uint32_t j = 1; j < 4; j++) {
        const uint32_t in = __shfl_sync(0xFFFFFFFFu, e, (lane + j) & 31), past = __shfl_sync(0xFFFFFFFFu, more, (lane + j) & 31);
        x |= (unsigned long long)(lane + j < 32 ? in : past) << (16 * j);
    }
    // starts of runs of n: of 2, 4, .. by doubling, then of n as two that overlap
    const uint32_t n = min(m, kRunMask);
    uint32_t have = 1;
    for (; have * 2 <= n; have *= 2) x &= x >> have;
    x &= x >> (n - have);
    uint32_t g = (uint32_t)x & 0xFFFFu;
    if (m > kRunMask && g) {
        // where the run ends, from the piece on, as far as it matters to the sixteen
        const uint32_t last = 31 - __clz(g);
        uint32_t end = last + kRunMask;
        if (last == 15) {
            const uint32_t far = m + 15;
            for (end = kRunMask; end < far; end += 16) {
                const uint32_t ne = 0xFFFFu ^ eq_mask16(*reinterpret_cast<const uint4 *>(&sm.text[piece * 16 + end]), c);
                if (ne) {
                    end += __ffs(ne) - 1;
                    break;
                }
            }
        }
        const uint32_t ok = end < m ? 0u : end - m + 1;  // starts that the run has room for
        g &= ok >= 16 ? 0xFFFFu : (1u << ok) - 1u;
    }
    const int64_t room = (int64_t)a.text_len - m - (int64_t)t0 - piece * 16 + 1;  // valid starts from the piece's
    return g & (room <= 0 ? 0u : room >= 16 ? 0xFFFFu : (1u << room) - 1u);
}

// Finds every start of the patterns in `mask` in the tile (staged in shared
// memory). Every lane takes its four pieces, one per step, and builds once for
// all patterns the windows of the piece shifted by 1, 2 and 3 bytes (the word
// after the piece comes from the next lane, or from shared memory for lane 31).
// Patterns of at most 4 bytes are decided at all sixteen starts at once; their
// matches go to pieces(p, piece, 16-bit mask). Patterns of 8 bytes and more share
// one test of the piece's four aligned words against the anchor map, whose cost
// does not grow with the number of patterns. What needs more than that comes after the
// steps, in loops that are not unrolled (inside the steps, where everything is
// there four times, it made the stage pass 680 us per GiB instead of 480): words
// found in the map, pieces with the first two bytes of a pattern of 5 to 7, the
// patterns without good anchors (runs, decided from masks of 64 positions, and
// those compared by four bytes). Their starts, or pieces, are queued per warp,
// verified 32 at a time, one per lane, and counted or set in `match`.
// Returns the patterns whose starts the lane verified.
// PLAIN: there are patterns of at most 4 bytes and with good anchors only. Without
// the other kinds' code, though it is not run, the graph of parse, tree and search
// over 1 GiB takes 1064 and 1325 us for two sets of eight such patterns, 1102 and
// 1340 with it.
// The pattern loops are not unrolled (the step loop is): with up to eight
// patterns a fully unrolled body outgrows the instruction cache.
template <bool COUNT, bool PLAIN, class Pieces>
__device__ __forceinline__ uint32_t filter_tile(const SearchArgs &a, SearchSmem &sm, uint32_t mask, uint64_t t0,
                                                uint16_t (*match)[SR_PIECES], Pieces pieces) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool tail_tile = t0 + kSearchTile + a.halo + 16 > a.text_len;
    // patterns in `mask` by how they are found: whole (up to 4 bytes), by anchors, by
    // their rarest four bytes, as runs, by their first two bytes (5 to 7 bytes)
    const uint32_t shorts = a.len_class[0] & mask, anchored = a.len_class[1] & mask, windows = PLAIN ? 0u : a.len_class[2] & mask,
                   runs = PLAIN ? 0u : a.len_class[3] & mask, mids = PLAIN ? 0u : a.len_class[4] & mask,
                   rare = PLAIN ? 0u : a.rare_runs & mask;
    auto in_map = [&](uint32_t x) {
        const uint32_t h = anchor_hash(x);
        return (sm.anchor_map[h >> 5] >> (h & 31)) & 1u;
    };
    uint32_t flagged = 0;  // bit 4k + i: word i of my piece of step k is in the map
    uint32_t begun = 0;    // bit 4p + k: my piece of step k has pattern p's first two bytes (mids)
#pragma unroll
    for (uint32_t k = 0; k < SR_STEPS; k++) {
        const uint32_t piece = k * SR_THREADS + tid;
        const uint4 vk = *reinterpret_cast<const uint4 *>(&sm.text[piece * 16]);
        if (shorts | mids) {  // uniform
            uint32_t w4 = __shfl_down_sync(0xFFFFFFFFu, vk.x, 1);
            if (lane == 31) w4 = *reinterpret_cast<const uint32_t *>(&sm.text[(piece + 1) * 16]);
            const uint32_t w[5] = {vk.x, vk.y, vk.z, vk.w, w4};
            uint32_t s1[4], s2[4], s3[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                s1[i] = __funnelshift_r(w[i], w[i + 1], 8);
                s2[i] = __funnelshift_r(w[i], w[i + 1], 16);
                s3[i] = __funnelshift_r(w[i], w[i + 1], 24);
            }
#pragma unroll 1
            for (uint32_t bits = shorts; bits; bits &= bits - 1) {
                const uint32_t p = __ffs(bits) - 1;
                const uint4 pre = sm.pat[p].pre;
                const uint32_t m = sm.pat[p].len;
                uint32_t x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = w[i] ^ pre.x;
                if (m > 1)
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] |= s1[i] ^ pre.y;
                if (m > 2)
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] |= s2[i] ^ pre.z;
                if (m > 3)
#pragma unroll
                    for (int i = 0; i < 4; i++) x[i] |= s3[i] ^ pre.w;
                uint32_t c0 = zero_bytes(x[0]), c1 = zero_bytes(x[1]), c2 = zero_bytes(x[2]), c3 = zero_bytes(x[3]);
                if (tail_tile) keep_valid_starts(a.text_len, m, t0, piece * 16, c0, c1, c2, c3);
                if (c0 | c1 | c2 | c3) pieces(p, piece, gather16(c0, c1, c2, c3));
            }
#pragma unroll 1
            for (uint32_t bits = mids; bits; bits &= bits - 1) {
                const uint32_t p = __ffs(bits) - 1;
                const uint2 pre = *reinterpret_cast<const uint2 *>(&sm.pat[p].pre);
                uint32_t x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = (w[i] ^ pre.x) | (s1[i] ^ pre.y);
                begun |= (any_zero_byte(x) ? 1u : 0u) << (4 * p + k);
            }
        }
        if (anchored | rare)  // uniform
            flagged |= (in_map(vk.x) | (in_map(vk.y) << 1) | (in_map(vk.z) << 2) | (in_map(vk.w) << 3)) << (4 * k);
    }
    if (!(anchored | windows | runs | mids)) return 0;  // uniform

    const bool staged = a.halo <= kSearchMaxStagedPattern;
    uint32_t found = 0;
    uint32_t *queue = sm.queue[warp];
    uint32_t queued = 0;  // the same in all lanes
    // Verifies the queued starts.
    auto drain = [&]() {
        __syncwarp();
        for (uint32_t i = lane; i < queued; i += 32) {
            const uint32_t e = queue[i], p = e >> 16, start = e & 0xFFFFu;
            if ((mids >> p) & 1u) {  // a piece
                const uint32_t g = mid_starts(a, sm, p, start, tail_tile, t0);
                if (g) pieces(p, start, g);
                continue;
            }
            if (!verify_start(a, sm, p, start, staged, t0)) continue;
            found |= 1u << p;
            if (COUNT)
                atomicAdd(&sm.count[p], 1u);
            else
                set_match(match[p], start);
        }
        __syncwarp();
        queued = 0;
    };
    // Queues each lane's (p, start) if `ok` and the start lies in the tile (one before it has wrapped).
    auto queue_start = [&](uint32_t p, uint32_t start, bool ok) {
        ok = ok && start < kSearchTile;
        const uint32_t who = __ballot_sync(0xFFFFFFFFu, ok);
        if (ok) queue[queued + __popc(who & ((1u << lane) - 1u))] = (p << 16) | start;
        queued += __popc(who);
        if (queued > SR_QCAP - 32) drain();
    };
    // Queues pattern p's starts first + bit, for the set bits of each lane's g.
    auto queue_starts = [&](uint32_t p, uint32_t g, uint32_t first) {
        while (__any_sync(0xFFFFFFFFu, g != 0)) {
            queue_start(p, first + __ffs(g) - 1, g != 0);
            g &= g - 1;
        }
    };
    // Pieces with the first two bytes of a pattern of 5 to 7.
#pragma unroll 1
    for (uint32_t bits = mids; bits; bits &= bits - 1) {
        const uint32_t p = __ffs(bits) - 1, mine = (begun >> (4 * p)) & 15u;
        if (!__any_sync(0xFFFFFFFFu, mine != 0)) continue;
#pragma unroll 1
        for (uint32_t k = 0; k < SR_STEPS; k++) queue_start(p, k * SR_THREADS + tid, (mine >> k) & 1u);
    }
    // Runs of rare bytes are looked for only where the warp's pieces, or the words
    // right after them, have a word in the map.
    uint32_t others = windows | runs;
    if (rare) {  // uniform
        bool some = flagged != 0;
        if (lane == 31)
            for (uint32_t k = 0; k < SR_STEPS; k++)
                some |= in_map(*reinterpret_cast<const uint32_t *>(&sm.text[(k * SR_THREADS + tid + 1) * 16]));
        if (!__any_sync(0xFFFFFFFFu, some)) others &= ~rare;
    }
    // Words in the map, against every pattern's anchors: those of the lane's
    // pieces, then (a round more) of the words past the tile, of starts in it.
    // Most often one lane or two have one; then the warp takes a word at a time
    // and each lane compares it with one anchor. Only where more lanes have one
    // than there are patterns does each lane take its own through all patterns
    // (always so: 116 us for 256 MiB and 8 patterns, 106 for 100 MB of nested text
    // with longer ones; now 103 and 88).
    if (anchored) {
        const uint32_t anchor = reinterpret_cast<const uint32_t *>(&sm.pat[lane >> 2].anc)[lane & 3];
        const uint32_t anchor_r = sm.pat[lane >> 2].r0 + 1 + (lane & 3);
        const bool mine = (anchored >> (lane >> 2)) & 1u;
#pragma unroll 1
        for (uint32_t past = 0; past < 2; past++) {
            if (past) {
                if ((tid & ~31u) >= a.anchor_words) break;  // whole warps
                flagged = tid < a.anchor_words && in_map(*reinterpret_cast<const uint32_t *>(&sm.text[kSearchTile + tid * 4]));
            }
            while (const uint32_t with = __ballot_sync(0xFFFFFFFFu, flagged != 0)) {
                if (__popc(with) <= __popc(anchored)) {  // one word, lane 4p + i for anchor i of pattern p
                    const uint32_t from = __ffs(with) - 1, b = __ffs(__shfl_sync(0xFFFFFFFFu, flagged, from)) - 1;
                    const uint32_t t = (tid & ~31u) + from;
                    const uint32_t at = past ? kSearchTile + t * 4 : ((b >> 2) * SR_THREADS + t) * 16 + (b & 3) * 4;
                    queue_start(lane >> 2, at - anchor_r, *reinterpret_cast<const uint32_t *>(&sm.text[at]) == anchor && mine);
                    if (lane == from) flagged &= flagged - 1;
                    continue;
                }
                const uint32_t b = __ffs(flagged) - 1;  // (NONE without one)
                const uint32_t at = !flagged ? 0u : past ? kSearchTile + tid * 4 : ((b >> 2) * SR_THREADS + tid) * 16 + (b & 3) * 4;
                const uint32_t x = *reinterpret_cast<const uint32_t *>(&sm.text[at]);
#pragma unroll 1
                for (uint32_t bits = anchored; bits; bits &= bits - 1) {
                    const uint32_t p = __ffs(bits) - 1;
                    const uint4 c = sm.pat[p].anc;
                    // anchor r0 + 1 + i: start at - r0 - 1 - i, bit 3 - i from at - r0 - 4
                    const uint32_t g = (x == c.x ? 8u : 0u) | (x == c.y ? 4u : 0u) | (x == c.z ? 2u : 0u) | (x == c.w ? 1u : 0u);
                    queue_starts(p, flagged ? g : 0u, at - sm.pat[p].r0 - 4);
                }
                flagged &= flagged - 1;
            }
        }
    }
    // The other patterns, piece by piece (windows: the pieces past the tile too). A
    // window is looked for by its rarest two bytes: by its first byte, which is
    // most often the common one, a pattern like "||||||||a" took 102 us in 64 MiB of
    // "|" and 70 in outline text; now 41 and 41.
    if (others) {  // the same in all lanes
#pragma unroll 1
        for (uint32_t base = tid & ~31u; base < a.window_pieces; base += SR_THREADS) {  // whole warps
            const uint32_t piece = base + lane;
            const uint4 v = *reinterpret_cast<const uint4 *>(&sm.text[piece * 16]);
            uint32_t w4 = __shfl_down_sync(0xFFFFFFFFu, v.x, 1);
            if (lane == 31) w4 = *reinterpret_cast<const uint32_t *>(&sm.text[(piece + 1) * 16]);
#pragma unroll 1
            for (uint32_t bits = others; bits; bits &= bits - 1) {
                const uint32_t p = __ffs(bits) - 1;
                const uint4 pre = sm.pat[p].pre;
                if ((runs >> p) & 1u) {  // of eight and more: it holds an aligned word of it, in the piece or right after
                    if (base >= SR_PIECES ||
                        !__any_sync(0xFFFFFFFFu, v.x == pre.x || v.y == pre.x || v.z == pre.x || v.w == pre.x || w4 == pre.x))
                        continue;
                    const uint32_t g = run_starts(a, sm, p, eq_mask16(v, pre.x), piece, t0);
                    if (g) pieces(p, piece, g);
                    continue;
                }
                // the window's rarest two bytes, in any of the sixteen places: a zero byte in one of four words
                const uint32_t x[4] = {(v.x ^ pre.x) | (__funnelshift_r(v.x, v.y, 8) ^ pre.y),
                                       (v.y ^ pre.x) | (__funnelshift_r(v.y, v.z, 8) ^ pre.y),
                                       (v.z ^ pre.x) | (__funnelshift_r(v.z, v.w, 8) ^ pre.y),
                                       (v.w ^ pre.x) | (__funnelshift_r(v.w, w4, 8) ^ pre.y)};
                if (!__any_sync(0xFFFFFFFFu, any_zero_byte(x))) continue;
                const uint32_t r0 = sm.pat[p].r0, pair = sm.pat[p].pair;
                uint32_t ok = 0;
                if (piece < SR_PIECES + (r0 + pair + 15) / 16) {  // where they are: the window's four bytes
                    for (uint32_t g = gather16(zero_bytes(x[0]), zero_bytes(x[1]), zero_bytes(x[2]), zero_bytes(x[3])); g; g &= g - 1) {
                        const uint32_t b = __ffs(g) - 1, off = piece * 16 + b - pair;
                        if (off < kSearchTile + 512 && text4(a, sm, off, true, t0) == pre.z) ok |= 1u << b;
                    }
                }
                queue_starts(p, ok, piece * 16 - pair - r0);
            }
        }
    }
    if (queued) drain();
    return found;
}

// Pass 1: matches of every pattern in every tile (counts only). NP = a.np.
template <uint32_t NP>
__global__ void __launch_bounds__(SR_THREADS) search_count_kernel(const __grid_constant__ SearchArgs a) {
    __shared__ SearchSmem sm;
    const uint32_t tid = threadIdx.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * kSearchTile;
    load_tile(a, sm, t0);
    __syncthreads();
    // Lanes with pieces of the same pattern add up their matches first: one
    // shared-memory atomic per (round, pattern) instead of one per piece.
    filter_tile<true, false>(a, sm, 0xFFu, t0, nullptr, [&](uint32_t p, uint32_t piece, uint32_t mk) {
        const uint32_t group = __match_any_sync(__activemask(), p);
        const uint32_t sum = __reduce_add_sync(group, __popc(mk));
        if ((threadIdx.x & 31) == __ffs(group) - 1 && sum) atomicAdd(&sm.count[p], sum);
    });
    __syncthreads();
    if (tid < a.np) a.counts[(size_t)tid * a.ld + blockIdx.x] = sm.count[tid];
}

// Pass 3: tiles with matches recompute the match masks of the patterns that
// have some; then, pattern by pattern, thread t takes pieces [4t, 4t+4) (in
// position order), a block scan of the per-thread match counts gives every
// thread its first output slot after the tile's base from pass 2, and each
// thread writes its matches there: the block's stores cover one contiguous
// range. Tiles without matches exit before loading text.
// base(p): the pattern's first output slot of the tile.
template <uint32_t NP, class Base>
__device__ __forceinline__ void write_tile(const SearchArgs &a, SearchSmem &sm, uint16_t (*match)[SR_PIECES],
                                           uint32_t *warp_sum, uint32_t tile, Base base) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t t0 = (uint64_t)tile * kSearchTile;
    // patterns with matches here whose output window is not yet full
    uint32_t want = 0;
    for (uint32_t p = 0; p < NP; p++) {
        size_t at = (size_t)p * a.ld + tile;
        if (a.counts[at] && base(p) < a.max_out[p]) want |= 1u << p;
    }
    if (!want) return;
    load_tile(a, sm, t0);
    for (uint32_t o = tid; o < NP * SR_PIECES / 8; o += SR_THREADS)
        reinterpret_cast<uint4 *>(&match[0][0])[o] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    filter_tile<false, false>(a, sm, want, t0, match,
                       [&](uint32_t p, uint32_t piece, uint32_t mk) { match[p][piece] = (uint16_t)mk; });
    __syncthreads();
    for (uint32_t w = want; w; w &= w - 1) {
        const uint32_t p = __ffs(w) - 1;
        const uint2 m4 = *reinterpret_cast<const uint2 *>(&match[p][4 * tid]);  // my 4 pieces
        const uint32_t n = __popc(m4.x) + __popc(m4.y), inc0 = n;
        uint32_t inc = inc0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t x = 0; x < warp; x++) before += warp_sum[x];
        uint32_t r = base(p) + before + inc - n;
        const uint32_t max_out = a.max_out[p];
        uint32_t *out = a.out[p];
        const uint32_t mm[2] = {m4.x, m4.y};
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            uint32_t bits = mm[h];  // pieces 4t+2h (low 16 bits) and 4t+2h+1 (high 16 bits)
            while (bits && r < max_out) {
                uint32_t b = __ffs(bits) - 1;
                bits &= bits - 1;
                uint32_t piece = 4 * tid + 2 * h + (b >> 4);
                out[r++] = (uint32_t)(t0 + piece * 16 + (b & 15));
            }
        }
        __syncthreads();  // warp_sum is reused by the next pattern
    }
}

// Recomputing form: block b writes tile b. Staged form: a small grid takes
// the tiles the stage pass listed as overflowing their slots (usually none).
template <uint32_t NP>
__global__ void __launch_bounds__(SR_THREADS) search_write_kernel(const __grid_constant__ SearchArgs a) {
    __shared__ SearchSmem sm;
    __shared__ alignas(16) uint16_t match[NP][SR_PIECES];
    __shared__ uint32_t warp_sum[SR_THREADS / 32];
    const uint32_t n = a.stage ? *a.overflow_n : a.n_tiles;
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
        const uint32_t tile = a.stage ? a.overflow_list[i] : i;
        write_tile<NP>(a, sm, match, warp_sum, tile, [&](uint32_t p) { return a.bases[(size_t)p * a.ld + tile]; });
        __syncthreads();  // shared memory is reused by the next tile
    }
}

// ----------------------------------------------------------- staged path --
//
// With a staging buffer the filter and verification run once: pass 1
// (search_stage_kernel) keeps each tile's match masks in shared memory, counts
// every pattern's hits with one block scan for all patterns at once, and writes
// the tile's hits, in (pattern, position) order, as 16-bit tile offsets into the
// tile's staging slot. After the column scan, pass 2 (search_copy_kernel)
// copies them to their final slots. A tile with more hits than its staging slot
// holds is flagged and left to search_write_kernel, which recomputes it.

// Lists the starts at + bit of the set bits, ascending, from both ends at once:
// half the rounds of the lane that has most (256 MiB with 28 M hits of "||||":
// 181 us one at a time, 159 so; run by run 158, all 64 positions of a lane in one
// loop 174).
__device__ __forceinline__ void list_starts(uint16_t *out, uint32_t bits, uint32_t at) {
    uint16_t *end = out + __popc(bits);
    while (bits) {
        const uint32_t lo = __ffs(bits) - 1, hi = 31 - __clz(bits);
        *out++ = (uint16_t)(at + lo);
        *--end = (uint16_t)(at + hi);
        bits &= bits - 1;
        bits &= ~(1u << hi);
    }
}

template <uint32_t NP, bool PLAIN>
__global__ void __launch_bounds__(SR_THREADS, 5) search_stage_kernel(const __grid_constant__ SearchArgs a) {
    constexpr uint32_t NQ = (NP + 1) / 2;  // packed count words, two patterns each
    __shared__ SearchSmem sm;
    __shared__ alignas(16) uint16_t match[NP][SR_PIECES];
    __shared__ uint32_t warp_sum[SR_THREADS / 32][NQ];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tile = blockIdx.x;
    const uint64_t t0 = (uint64_t)tile * kSearchTile;
    if (tid == 0 && tile + kPrefetchTilesAhead < a.n_tiles)
        prefetch_l2(a.text + (uint64_t)(tile + kPrefetchTilesAhead) * kSearchTile, kSearchTile);
    load_tile(a, sm, t0);
    if (tid == 0) sm.active = 0;
    for (uint32_t o = tid; o < NP * SR_PIECES / 8; o += SR_THREADS)
        reinterpret_cast<uint4 *>(&match[0][0])[o] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    // the patterns with hits anywhere in the tile, as the filter finds them
    uint32_t found = 0;
    found |= filter_tile<false, PLAIN>(a, sm, (1u << NP) - 1u, t0, match, [&](uint32_t p, uint32_t piece, uint32_t mk) {
        match[p][piece] = (uint16_t)mk;
        found |= 1u << p;
    });
    found = __reduce_or_sync(0xFFFFFFFFu, found);
    if (lane == 0 && found) atomicOr(&sm.active, found);
    __syncthreads();
    const uint32_t active = sm.active;
    if (active == 0) {  // a tile without hits is done here
        if (tid < NP) a.counts[(size_t)tid * a.ld + tile] = 0;
        if (tid == 0) a.overflow[tile] = 0;
        return;
    }
    uint16_t *stage = reinterpret_cast<uint16_t *>(sm.text);  // the slot, assembled where the text was
    if ((active & (active - 1)) == 0) {  // hits of one pattern only: the usual tile
        const uint32_t p = __ffs(active) - 1;
        const uint2 m = *reinterpret_cast<const uint2 *>(&match[p][4 * tid]);
        const uint32_t mine = __popc(m.x) + __popc(m.y);
        uint32_t inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += t;
        }
        if (lane == 31) warp_sum[warp][0] = inc;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < SR_THREADS / 32; w++) {
            const uint32_t x = warp_sum[w][0];
            before += w < warp ? x : 0u;
            total += x;
        }
        if (tid < NP) a.counts[(size_t)tid * a.ld + tile] = tid == p ? total : 0u;
        const bool over = total > a.stage_cap;
        if (tid == 0) {
            a.overflow[tile] = over ? 1 : 0;
            if (over && a.overflow_list) a.overflow_list[atomicAdd(a.overflow_n, 1u)] = tile;
        }
        if (over) return;  // uniform: recomputed later
        uint32_t r = before + inc - mine;
        const uint32_t mm[2] = {m.x, m.y};
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            list_starts(stage + r, mm[h], 64 * tid + 32 * h);
            r += __popc(mm[h]);
        }
        __syncthreads();
        uint4 *dst = reinterpret_cast<uint4 *>(a.stage + (size_t)tile * a.stage_cap);
        const uint4 *src = reinterpret_cast<const uint4 *>(stage);
        for (uint32_t o = tid; o < (total + 7) / 8; o += SR_THREADS) dst[o] = src[o];
        return;
    }
    // my hits per pattern with hits (4 pieces: at most 64)
    uint2 m4[NP];
#pragma unroll
    for (uint32_t p = 0; p < NP; p++)
        m4[p] = ((active >> p) & 1u) ? *reinterpret_cast<const uint2 *>(&match[p][4 * tid]) : make_uint2(0, 0);
    // counts, two patterns per word; inclusive warp scans of the words that
    // hold a pattern with hits (tile totals stay below 2^16)
    uint32_t packed[NQ], inc[NQ];
#pragma unroll
    for (uint32_t q = 0; q < NQ; q++) packed[q] = 0;
#pragma unroll
    for (uint32_t p = 0; p < NP; p++)
        packed[p >> 1] |= (uint32_t)(__popc(m4[p].x) + __popc(m4[p].y)) << (16 * (p & 1));
#pragma unroll
    for (uint32_t q = 0; q < NQ; q++) {
        inc[q] = packed[q];
        if ((active >> (2 * q)) & 3u) {  // uniform
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc[q], o);
                if ((int)lane >= o) inc[q] += t;
            }
        }
        if (lane == 31) warp_sum[warp][q] = inc[q];
    }
    __syncthreads();
    uint32_t before[NQ], total[NQ];
#pragma unroll
    for (uint32_t q = 0; q < NQ; q++) {
        before[q] = total[q] = 0;
        if ((active >> (2 * q)) & 3u)
            for (uint32_t w = 0; w < SR_THREADS / 32; w++) {
                const uint32_t x = warp_sum[w][q];
                before[q] += w < warp ? x : 0u;
                total[q] += x;
            }
    }
    // tile totals per pattern, and where each pattern's hits start in the slot;
    // the slot is assembled in shared memory (the staged text is no longer
    // read) and stored with 16-byte writes
    static_assert(kSearchStageCap * 2 <= kSearchTile, "the slot fits where the tile text was");
    uint32_t start = 0;
#pragma unroll
    for (uint32_t p = 0; p < NP; p++) {
        const uint32_t sh = 16 * (p & 1);
        const uint32_t tot = (total[p >> 1] >> sh) & 0xFFFFu;
        const uint32_t mine = (packed[p >> 1] >> sh) & 0xFFFFu;
        uint32_t r = start + ((before[p >> 1] >> sh) & 0xFFFFu) + ((inc[p >> 1] >> sh) & 0xFFFFu) - mine;
        if (mine && start + tot <= a.stage_cap) {
            const uint32_t mm[2] = {m4[p].x, m4[p].y};
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                list_starts(stage + r, mm[h], 64 * tid + 32 * h);
                r += __popc(mm[h]);
            }
        }
        if (tid == 0) a.counts[(size_t)p * a.ld + tile] = tot;
        start += tot;
    }
    if (tid == 0) {
        a.overflow[tile] = start > a.stage_cap ? 1 : 0;
        if (start > a.stage_cap && a.overflow_list) a.overflow_list[atomicAdd(a.overflow_n, 1u)] = tile;
    }
    if (start > a.stage_cap) return;  // uniform: recomputed later
    __syncthreads();
    uint4 *dst = reinterpret_cast<uint4 *>(a.stage + (size_t)tile * a.stage_cap);
    const uint4 *src = reinterpret_cast<const uint4 *>(stage);
    for (uint32_t o = tid; o < (start + 7) / 8; o += SR_THREADS) dst[o] = src[o];
}

// Pass 2 of the staged path: two warps per tile. Lane p reads pattern p's
// count and first output slot (all patterns at once: one memory round trip),
// a warp scan places each pattern's hits in the tile's slot, and the warps
// copy them to their final slots, alternate runs of 256 each.
constexpr uint32_t SC_WARPS = 2;                          // warps per tile
constexpr uint32_t SC_TILES = SR_THREADS / 32 / SC_WARPS;  // tiles per block
__global__ void __launch_bounds__(SR_THREADS) search_copy_kernel(SearchArgs a) {
    const uint32_t lane = threadIdx.x & 31, half = (threadIdx.x >> 5) % SC_WARPS;
    const uint32_t tile = blockIdx.x * SC_TILES + (threadIdx.x >> 5) / SC_WARPS;
    if (tile >= a.n_tiles || a.overflow[tile]) return;  // overflowing tiles: search_write_kernel
    uint32_t n = 0, base = 0, max_out = 0;
    if (lane < a.np) {
        const size_t at = (size_t)lane * a.ld + tile;
        n = a.counts[at];
        base = a.bases[at];
        max_out = a.max_out[lane];
    }
    uint32_t inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if ((int)lane >= o) inc += t;
    }
    if (__shfl_sync(0xFFFFFFFFu, inc, 31) == 0) return;
    const uint64_t t0 = (uint64_t)tile * kSearchTile;
    const uint16_t *slot = a.stage + (size_t)tile * a.stage_cap;
    for (uint32_t p = 0; p < a.np; p++) {
        const uint32_t np_ = __shfl_sync(0xFFFFFFFFu, n, p);
        if (np_ == 0) continue;
        const uint32_t b = __shfl_sync(0xFFFFFFFFu, base, p), mx = __shfl_sync(0xFFFFFFFFu, max_out, p);
        const uint32_t start = __shfl_sync(0xFFFFFFFFu, inc - n, p);
        const uint32_t lim = b >= mx ? 0u : min(np_, mx - b);  // the first max_out hits overall
        uint32_t *__restrict__ out = a.out[p] + b;
        const uint16_t *__restrict__ src = slot + start;
        // the tile's warps take alternate runs of 256 hits; eight independent
        // loads in flight per lane before the stores
        for (uint32_t i0 = half * 256; i0 < lim; i0 += 256 * SC_WARPS) {
            uint32_t v[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                const uint32_t i = i0 + j * 32 + lane;
                v[j] = i < lim ? __ldg(src + i) : 0u;
            }
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                const uint32_t i = i0 + j * 32 + lane;
                if (i < lim) out[i] = (uint32_t)(t0 + v[j]);
            }
        }
    }
}

// Pass 2 of a text of at most kSearchFinishTiles tiles, block b for tile b: it
// adds up the counts of the tiles before its own itself (one load a thread and
// pattern, all in flight at once), copies the tile's hits to their final
// slots, or recomputes a tile that overflowed its slot; the last tile's block
// writes the totals. Two launches instead of four and a memset: on the host
// each costs 3.9 us.
template <uint32_t NP>
__global__ void __launch_bounds__(SR_THREADS) search_finish_kernel(const __grid_constant__ SearchArgs a) {
    __shared__ SearchSmem sm;
    __shared__ alignas(16) uint16_t match[NP][SR_PIECES];
    __shared__ uint32_t warp_sum[SR_THREADS / 32], part[NP][SR_THREADS / 32], base[NP];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
    const bool over = a.overflow[tile], last = tile == a.n_tiles - 1;
    uint32_t n[NP], any = 0;
#pragma unroll
    for (uint32_t p = 0; p < NP; p++) any |= n[p] = a.counts[(size_t)p * a.ld + tile];
    if (!any && !last) return;  // uniform
#pragma unroll
    for (uint32_t p = 0; p < NP; p++) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < kSearchFinishTiles / SR_THREADS; i++) {
            const uint32_t t = i * SR_THREADS + tid;
            sum += t < tile ? a.counts[(size_t)p * a.ld + t] : 0u;
        }
        sum = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (lane == 0) part[p][warp] = sum;
    }
    __syncthreads();
    if (tid < NP) {
        uint32_t b = 0;
#pragma unroll
        for (uint32_t w = 0; w < SR_THREADS / 32; w++) b += part[tid][w];
        base[tid] = b;
        if (last) a.totals[tid] = b + a.counts[(size_t)tid * a.ld + tile];
    }
    __syncthreads();
    if (over) {  // uniform
        write_tile<NP>(a, sm, match, warp_sum, tile, [&](uint32_t p) { return base[p]; });
        return;
    }
    const uint32_t t0 = tile * kSearchTile;
    const uint16_t *src = a.stage + (size_t)tile * a.stage_cap;
#pragma unroll
    for (uint32_t p = 0; p < NP; p++) {
        const uint32_t b = base[p], mx = a.max_out[p], lim = b >= mx ? 0u : min(n[p], mx - b);
        for (uint32_t i = tid; i < lim; i += SR_THREADS) a.out[p][b + i] = t0 + __ldg(src + i);
        src += n[p];
    }
}

// How common a byte is in text, 0 (rare) to 4, for the choice of anchor words.
struct ByteWeights {
    uint8_t of[256];
    constexpr ByteWeights() : of{} {
        for (int c = 'a'; c <= 'z'; c++) of[c] = 2;
        for (int c = 0x80; c < 256; c++) of[c] = 1;
        for (char c : {'-', '=', '.', ',', '/', ':', '@', '*', '#', '_', '\t', '\r'}) of[(uint8_t)c] = 2;
        for (char c : {'e', 't', 'a', 'o', 'i', 'n', 's', 'r', 'h', 'l'}) of[(uint8_t)c] = 3;
        for (char c : {' ', '|', '\n'}) of[(uint8_t)c] = 4;
    }
};
constexpr ByteWeights kByteWeights;
static uint32_t byte_weight(uint8_t c) { return kByteWeights.of[c]; }

// How common a four-byte word is: repeated bytes count most.
static uint32_t word_weight(const uint8_t *p) {
    uint32_t w = 0;
    for (uint32_t i = 0; i < 4; i++) w += byte_weight(p[i]) + (i && p[i] == p[i - 1] ? 4 : 0);
    return w;
}

// Where the `words` (1 or 4) consecutive words (at r0 + first + 0, 1, ..) lie whose
// most common one is the rarest, the first among equals; weight: that word's. Each
// word is weighed once: a call with a pattern of 250 bytes waited 19 us for the
// choice when each was weighed four times, by library calls, and now waits 1.
static uint32_t rarest_place(const uint8_t *pat, uint32_t len, uint32_t first, uint32_t words, uint32_t &weight) {
    // (a pattern whose halo is not staged is looked for at its beginning)
    const uint32_t reach = len > kSearchMaxStagedPattern ? 0 : kAnchorReach;
    uint32_t best = 0, recent[4] = {};  // the last four words' weights
    weight = ~0u;
    for (uint32_t i = 0; i + 1 < words && first + i + 4 <= len; i++) recent[i % 4] = word_weight(pat + first + i);
    for (uint32_t r0 = 0; r0 + first + words + 3 <= len && r0 <= reach && weight; r0++) {
        const uint32_t i = r0 + words - 1;
        recent[i % 4] = word_weight(pat + first + i);
        const uint32_t w = words == 1 ? recent[i % 4] : std::max({recent[0], recent[1], recent[2], recent[3]});
        if (w < weight) {
            best = r0;
            weight = w;
        }
    }
    return best;
}

void search_add_pattern(SearchArgs &a, const uint8_t *host, const uint8_t *dev, uint32_t len, uint32_t *out,
                        uint32_t max_out) {
    const uint32_t p = a.np++;
    a.pat[p] = dev;
    a.out[p] = out;
    a.max_out[p] = max_out;
    SearchPatMeta &m = a.meta[p];
    m = SearchPatMeta{};
    m.len = len;
    for (uint32_t j = 0; j < 4 && j < len; j++) m.pre[j] = host[j] * 0x01010101u;
    auto word = [&](uint32_t r) {
        return (uint32_t)host[r] | ((uint32_t)host[r + 1] << 8) | ((uint32_t)host[r + 2] << 16) | ((uint32_t)host[r + 3] << 24);
    };
    if (len >= 4) m.last4 = word(len - 4);
    if (len < kAnchorMin) {  // decided from these constants alone
        a.len_class[len > 4 ? 4 : 0] |= 1u << p;
        return;
    }
    if (!dev) {
        a.pat_at[p] = a.n_pat_bytes;
        memcpy(a.pat_bytes + a.n_pat_bytes, host, len);
        a.n_pat_bytes += (len + 15) & ~15u;
    }
    // A run of one byte, however rare the byte: its four anchor words are the same,
    // and in text that is such a run every word has four candidates (64 MiB of "Z",
    // eight of them looked for: 340 us by anchors, 80 by masks). The word of a
    // rare byte is in the map all the same, to tell where there is nothing to look
    // for: eight such patterns in 64 MiB without them 61 us without it, 49 with.
    if (len <= kSearchMaxStagedPattern && std::all_of(host, host + len, [&](uint8_t c) { return c == host[0]; })) {
        if (word_weight(host) < kPoorAnchor) {
            a.rare_runs |= 1u << p;
            a.anchor_hash[a.n_anchor++] = anchor_hash(word(0));
        }
        a.len_class[3] |= 1u << p;
        a.window_pieces = std::max(a.window_pieces, SR_PIECES);
        return;
    }
    uint32_t weight;
    m.r0 = rarest_place(host, len, 1, 4, weight);
    if (weight >= kPoorAnchor) {
        m.r0 = rarest_place(host, len, 0, 1, weight);
        const uint8_t *w = host + m.r0;
        auto pair_weight = [&](uint32_t j) { return byte_weight(w[j]) + byte_weight(w[j + 1]) + (w[j] == w[j + 1] ? 4 : 0); };
        for (uint32_t j = 1; j < 3; j++)
            if (pair_weight(j) < pair_weight(m.pair)) m.pair = j;
        m.pre[0] = w[m.pair] * 0x01010101u;
        m.pre[1] = w[m.pair + 1] * 0x01010101u;
        m.pre[2] = word(m.r0);
        a.len_class[2] |= 1u << p;
        a.window_pieces = std::max(a.window_pieces, SR_PIECES + (m.r0 + m.pair + 15) / 16);
        return;
    }
    a.len_class[1] |= 1u << p;
    for (uint32_t r = 1; r <= 4; r++) {
        m.anc[r - 1] = word(m.r0 + r);
        a.anchor_hash[a.n_anchor++] = anchor_hash(m.anc[r - 1]);
    }
    a.anchor_words = std::max(a.anchor_words, m.r0 / 4 + 2);  // text words past the tile: up to offset r0 + 4
}

constexpr uint32_t kSearchWriteGrid = 512;  // blocks of the staged form's write pass

// The stage pass, without the code for patterns that need more than the steps and
// the anchors where there are none (filter_tile).
template <uint32_t NP>
static void launch_stage(const SearchArgs &a, cudaStream_t st) {
    if ((a.len_class[2] | a.len_class[3] | a.len_class[4]) == 0) {
        search_stage_kernel<NP, true><<<a.n_tiles, SR_THREADS, 0, st>>>(a); OL_LAUNCHED();
    } else {
        search_stage_kernel<NP, false><<<a.n_tiles, SR_THREADS, 0, st>>>(a); OL_LAUNCHED();
    }
}

template <uint32_t NP>
static cudaError_t launch_search_np(const SearchArgs &a, cudaStream_t st) {
    if (a.stage) {
        if (a.n_tiles <= kSearchFinishTiles) {
            SearchArgs r = a;
            r.overflow_list = nullptr;  // the flags are enough
            launch_stage<NP>(r, st);
            search_finish_kernel<NP><<<a.n_tiles, SR_THREADS, 0, st>>>(r); OL_LAUNCHED();
            return cudaGetLastError();
        }
        cudaError_t e0 = cudaMemsetAsync(a.overflow_n, 0, sizeof(uint32_t), st);
        if (e0 != cudaSuccess) return e0;
        launch_stage<NP>(a, st);
        cudaError_t e = launch_scan_columns(a.counts, a.bases, a.totals, a.n_tiles, a.np, a.ld, st);
        if (e != cudaSuccess) return e;
        search_copy_kernel<<<(a.n_tiles + SC_TILES - 1) / SC_TILES, SR_THREADS, 0, st>>>(a); OL_LAUNCHED();
        search_write_kernel<NP><<<std::min(a.n_tiles, kSearchWriteGrid), SR_THREADS, 0, st>>>(a); OL_LAUNCHED();  // listed tiles
        return cudaGetLastError();
    }
    search_count_kernel<NP><<<a.n_tiles, SR_THREADS, 0, st>>>(a); OL_LAUNCHED();
    cudaError_t e = launch_scan_columns(a.counts, a.bases, a.totals, a.n_tiles, a.np, a.ld, st);
    if (e != cudaSuccess) return e;
    search_write_kernel<NP><<<a.n_tiles, SR_THREADS, 0, st>>>(a); OL_LAUNCHED();
    return cudaGetLastError();
}

// One instantiation per pattern count: the per-pattern loops unroll without
// guards and the shared match arrays hold only the launch's patterns.
cudaError_t launch_search(const SearchArgs &a, cudaStream_t st) {
    if (a.n_tiles == 0 || a.np == 0) return cudaSuccess;
    switch (a.np) {
        case 1: return launch_search_np<1>(a, st);
        case 2: return launch_search_np<2>(a, st);
        case 3: return launch_search_np<3>(a, st);
        case 4: return launch_search_np<4>(a, st);
        case 5: return launch_search_np<5>(a, st);
        case 6: return launch_search_np<6>(a, st);
        case 7: return launch_search_np<7>(a, st);
        case 8: return launch_search_np<8>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ol
