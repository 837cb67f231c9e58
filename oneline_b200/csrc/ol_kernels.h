// Kernel argument blocks and launch entry points shared between the kernels
// (*.cu) and the host runtime (runtime.cu). Device pointers only.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace ol {

// Kernels launched by this library in this process (every launch site counts
// itself), read through ol_launch_count().
void count_launch();
#define OL_LAUNCHED() ::ol::count_launch()

struct FlatNode;
struct DocStats;

constexpr uint32_t kParseTile = 16384;  // text bytes per parse tile
constexpr uint32_t kParseHalo = 256;    // bytes staged past a tile
constexpr uint32_t kTreeTile = 4096;      // lines per tree tile (256 threads x 16)
constexpr uint32_t kTreeSmallTile = 1024;  // of a document of at most kTreeFewTiles such tiles
constexpr uint32_t kTreeFewTiles = 64;     // tiles whose summaries every block scans itself
constexpr uint32_t kTreeLevels = 32;    // depth levels of the fast tree path

constexpr uint32_t kParseSlotCap = 1024;      // staged lines per tile
// Tiles up to which one launch finishes a parse (parse_finish_kernel). A parse and
// the wait for it, in us, two launches / four: 1 MiB 20 / 27, 8 MiB 20 / 29, 16 MiB
// (this many) 25 / 33. Two are the faster side past the line too: 32 MiB 33 / 40,
// 64 MiB 48 / 52.
constexpr uint32_t kParseFinishTiles = 1024;

struct ParseArgs {
    const uint8_t *text;  // padded: n_tiles * kParseTile + kParseHalo readable bytes
    uint64_t text_len;
    uint32_t n_tiles;
    uint32_t *tile_count;   // n_tiles newline counts (pass 1)
    uint32_t *tile_base;    // n_tiles exclusive prefix sums (larger texts)
    uint32_t *tile_first;   // n_tiles: first newline of the tile (tile-local), or NONE (pass 1)
    uint16_t *tile_depth;   // 8 per tile: deepest staged content line of each warp (pass 1; unset for a tile that
                            // did not fit its slot)
    DocStats *stats;        // reset by pass 1
    uint32_t *offsets;      // line_cap entries
    uint8_t *kinds;
    uint8_t *depth8;        // min(depth, 255)
    uint32_t line_cap;
    uint32_t *slot;         // per tile a slot of slot_cap line words
    uint8_t *slot_over;     // per tile: more lines than the slot holds
    uint32_t slot_cap;      // kParseSlotCap
    uint32_t first_tile;    // pass 1: block b takes tile first_tile + b (launches over tile ranges)
};

cudaError_t launch_parse(const ParseArgs &a, cudaStream_t st);
// The same in two parts, for a parse that starts while the text is still
// arriving: the stage pass over tiles [t0, t1) (any ranges that together cover
// every tile once, each launched once its tiles and their 256-byte halo are in
// device memory), then the passes that write the line arrays. The second part
// alone, with stats reset, writes them again (into larger arrays).
cudaError_t launch_parse_tiles(const ParseArgs &a, uint32_t t0, uint32_t t1, cudaStream_t st);
cudaError_t launch_parse_end(const ParseArgs &a, cudaStream_t st);

// Exclusive scan of each of `cols` columns of a column-major u32 matrix:
// column c is `rows` entries at in + c * ld (in, out 16-byte aligned, ld a
// multiple of 4); out has the same layout; totals[c] (optional) receives
// column c's sum.
cudaError_t launch_scan_columns(const uint32_t *in, uint32_t *out, uint32_t *totals, uint32_t rows, uint32_t cols,
                                uint32_t ld, cudaStream_t st);
// Column stride for per-tile count columns: rows rounded up to a multiple of 4.
inline uint32_t scan_ld(uint32_t rows) { return (rows + 3u) & ~3u; }
cudaError_t launch_classify_lines(const uint8_t *text, uint64_t N, const uint32_t *offsets, uint32_t L, FlatNode *nodes,
                                  uint32_t *depth32, cudaStream_t st, const uint32_t *count = nullptr);

struct TreeArgs {
    const uint8_t *kinds;
    const uint8_t *depth8;
    uint32_t L;
    uint32_t n_tiles;        // ceil(L / tree_tile_lines(L))
    uint32_t levels;         // max content depth + 1 (<= kTreeLevels)
    uint32_t *tile_last;     // n_tiles * kTreeLevels: last content line + 1 of each depth in the tile (0: none)
    uint32_t *tile_first;    // n_tiles * kTreeLevels: first content line of each depth in the tile (NONE: none)
    uint32_t *in_last;       // exclusive prefix max of tile_last over the tiles
    uint32_t *in_first;      // exclusive suffix min of tile_first over the tiles
    uint32_t *parent;
    uint32_t *subtree_end;   // optional
    uint32_t *first_child;
    uint32_t *next_sibling;
};

uint32_t tree_tile_lines(uint32_t L);  // lines per tile of a document of L lines
cudaError_t launch_tree_fast(const TreeArgs &a, cudaStream_t st);

// Any-depth path (content lines deeper than kTreeLevels-1).
struct TreeDeepArgs {
    const uint8_t *kinds;
    const uint8_t *depth8;
    const uint32_t *keys;    // depth of content lines, NONE for blank lines; nullptr: depth8 holds every depth
    uint32_t L;
    uint32_t *levels[8];     // minima: levels[0] of every 32 lines, levels[k] of 32 of levels[k-1]
    uint32_t level_len[8];
    uint32_t n_levels;       // at least 2; the last one has at most 32 entries
    uint32_t *parent;
    uint32_t *subtree_end;
    uint32_t *first_child;
    uint32_t *next_sibling;
};

cudaError_t launch_tree_deep(const TreeDeepArgs &a, cudaStream_t st);

constexpr uint32_t kSearchTile = 16384;
constexpr uint32_t kSearchMaxStagedPattern = 4096;
constexpr uint32_t kSearchMaxPatterns = 8;  // patterns per launch

// Per-pattern constants of a search launch, computed on the host from the
// pattern bytes (search_add_pattern) and read by every block as kernel
// parameters.
struct alignas(16) SearchPatMeta {
    uint32_t pre[4];  // bytes 0..3, each replicated into a word (0 past the end); of a pattern found by its rarest
                      // four bytes, the rarest two of those so, and the four, r0..r0 + 3, as a word
    uint32_t anc[4];  // anchor words: bytes [r, r + 4) little-endian, r = r0 + 1 .. r0 + 4
    uint32_t len;
    uint32_t r0;
    uint32_t last4;   // the last four bytes (len >= 4)
    uint32_t pair;    // the place of the rarest two in r0..r0 + 3
};
constexpr uint32_t kSearchInlinePattern = 64;   // patterns of up to this length travel in a launch's parameters
constexpr uint32_t kSearchPatBytes = kSearchInlinePattern * kSearchMaxPatterns;  // room for as many as a launch takes
static_assert(kSearchInlinePattern % 16 == 0, "each pattern's bytes begin on a 16-byte boundary");
// Tiles up to which one launch finishes a search. One pattern, in us, two launches /
// four: 1 MiB 38 / 46, 4 MiB (this many) 38 / 47, 8 MiB 40 / 47, 32 MiB 41 / 48, 64 MiB
// 53 / 60: two are the faster side past the line too. It lies here because the graph
// of a larger document is expected to hold the passes apart (tests/test_gpu_pipeline.py
// counts the kernels of a 6 MiB one).
constexpr uint32_t kSearchFinishTiles = 256;

struct SearchArgs {
    const uint8_t *text;     // padded: n_tiles * kSearchTile + kSearchMaxStagedPattern + 16 readable bytes
    uint64_t text_len;
    uint32_t n_tiles;
    uint32_t np;                                // patterns in this launch (1..8)
    uint32_t halo;                              // round_up(longest - 1, 16); > 4096 only when np == 1
    const uint8_t *pat[kSearchMaxPatterns];     // device copies (16-byte aligned), or nullptr: in pat_bytes
    uint32_t *out[kSearchMaxPatterns];          // ascending offsets, first max_out[p] of them
    uint32_t max_out[kSearchMaxPatterns];
    uint32_t ld;             // column stride of counts and bases: scan_ld(n_tiles)
    uint32_t *counts;        // [np][ld] matches per tile (pass 1), 16-byte aligned
    uint32_t *bases;         // [np][ld] exclusive scans (pass 2), 16-byte aligned
    uint32_t *totals;        // kSearchMaxPatterns totals (pass 2)
    // Staged form (nullptr: count pass + recomputing write pass): per tile a
    // slot of stage_cap 16-bit tile offsets, and a flag per tile whose hits did
    // not fit (recomputed by the write pass).
    uint16_t *stage;
    uint8_t *overflow;
    uint32_t stage_cap;
    uint32_t *overflow_n;     // staged form: count, then list, of the flagged tiles (n_tiles entries)
    uint32_t *overflow_list;
    SearchPatMeta meta[kSearchMaxPatterns];
    uint32_t anchor_hash[kSearchMaxPatterns * 4];  // anchor-map bits of the patterns of >= 8 bytes
    uint32_t n_anchor;
    uint32_t anchor_words;  // aligned text words past a tile that may be anchors of starts in it
    uint32_t window_pieces; // 16-byte pieces to look for the other patterns in
    // bit p: pattern p is decided whole (up to 4 bytes); found by its anchors, by
    // its rarest four bytes, as a run of one byte, or (5 to 7 bytes) by its first
    // two (search_add_pattern)
    uint32_t len_class[5];
    uint32_t rare_runs;     // those of the runs whose word is in the anchor map
    // The bytes of patterns without a device copy, each from a 16-byte boundary.
    uint32_t n_pat_bytes;
    uint32_t pat_at[kSearchMaxPatterns];
    alignas(16) uint8_t pat_bytes[kSearchPatBytes];
};
constexpr uint32_t kSearchStageCap = 8192;  // staged hits per tile (all patterns of a launch)

// Appends a pattern to a launch (slot a.np): its device copy (nullptr: at most
// kSearchInlinePattern bytes, which go into the launch's parameters), and the
// constants the kernels take from its host bytes.
void search_add_pattern(SearchArgs &a, const uint8_t *host, const uint8_t *dev, uint32_t len, uint32_t *out,
                        uint32_t max_out);
cudaError_t launch_search(const SearchArgs &a, cudaStream_t st);

// ---------------------------------------------------------------- query --

struct QueryArgs {
    const uint8_t *kinds;    // resident document (kinds, depth8, text, offsets) ...
    const uint8_t *depth8;
    const uint8_t *text;
    const uint32_t *offsets;
    uint64_t text_len;
    const FlatNode *nodes;   // ... or materialised nodes (then the four above are unused)
    uint32_t lines;          // lines in the document
    uint32_t lo, hi;         // range [lo, hi) of lines considered
    const uint32_t *hi_dev;  // its end on the device (at most hi), or nullptr
    uint32_t target_kind;    // 0: any
    uint32_t target_depth;   // NONE: any
    uint16_t *masks;         // kQueryMasks per block
    uint32_t *counts;        // per block of 4096 lines, 16-byte aligned
    uint32_t *bases;         // same size, 16-byte aligned
    uint32_t *total;         // device
    uint32_t *out;           // ascending line indices, first max_out of them
    uint32_t max_out;
};
constexpr uint32_t kQueryMasks = 256;
// Blocks whose counts the writing blocks add up themselves. A query that every
// line matches, in us, so / with a scan launch: 4 M lines 28 / 34, 16 M 32 / 34,
// 24 M 36 / 36, 33 M (this many blocks) 45 / 46, 64 M 68 / 58; one that no line
// matches: 24 M 34 / 36, 33 M 44 / 38.
constexpr uint32_t kQuerySelfScan = 8192;
uint32_t query_blocks(uint32_t lo, uint32_t hi);
cudaError_t launch_query(const QueryArgs &a, cudaStream_t st);

// ------------------------------------------------------------ dictionary --

constexpr uint32_t kDictTile = 16384;         // text bytes per tile (the parse tile: same padding)
constexpr uint32_t kDictHalo = 80;            // staged past the tile: > longest pattern, 16-byte multiple
constexpr uint32_t kDictMinLen = 4;           // the filter keys on a pattern's first 4 bytes
constexpr uint32_t kDictMaxLen = 64;
constexpr uint32_t kDictMaxHeavy = 32;        // patterns whose hits go to bitmaps in one search
constexpr uint32_t kDictFilterBits = 17;      // 2^17-bit filter (16 KiB of shared memory)
constexpr uint32_t kDictWordsPerTile = kDictTile / 32;
constexpr uint32_t kDictSortBlock = 4096;     // keys per block in the light-hit radix sort
constexpr uint32_t kDictMaxRuns = 4;          // run bytes of a set

// Filter and table hashes of a pattern's first four bytes (little-endian u32);
// the host compiler uses the same functions. The filter's word holds three bits
// of a key (bits 27.., 22.., 17.. of dict_filter_bits), so that a test is one
// shared-memory load; with 10,000 keys it lets 1.5% of other positions through
// (two bits in two words: 2.2%).
__host__ __device__ inline uint32_t dict_filter_word(uint32_t w) { return (w * 0x85EBCA77u) >> (32 - kDictFilterBits + 5); }
__host__ __device__ inline uint32_t dict_filter_bits(uint32_t w) { return w * 0xC2B2AE3Du; }
__host__ __device__ inline uint32_t dict_table_h(uint32_t w, uint32_t bits) { return (w * 0x9E3779B1u) >> (32 - bits); }

// Device view of a compiled pattern set. Patterns are deduplicated ("unique
// patterns" u); a trie over them gives, for a text position whose first four
// bytes match some pattern's, every unique pattern starting there.
struct DictSet {
    const uint32_t *filter;  // 2^kDictFilterBits bits
    const uint2 *table;      // open addressing: {first 4 bytes, trie node at depth 4}; empty: .y == NONE
    uint32_t table_bits;
    uint32_t max_probe;      // longest probe distance of any key
    const uint4 *nodes;      // {patterns: kDictOneFlag | an index in outs, an index in lists, or NONE; edge count (| kDictDenseFlag)
                             //  (| kDictPathFlag, run byte << 28, start in paths << 9); edge 0;
                             //  edge 1 | extra start | dense table}
    const uint32_t *extra;   // edges 1.. of nodes with 3..kDictDenseMin children; edge = (child << 8) | byte,
                             // sorted by byte
    const uint32_t *dense;   // 256 children (NONE: no edge) per node with more than kDictDenseMin children
    uint32_t n_u;
    // The patterns that end at a node of a run byte's trie: bit r of the 64-bit
    // mask {x, y} for a pattern c^r rest, their u from outs[z] on, r ascending
    // (outs ends with an unused entry).
    const uint4 *lists;
    const uint32_t *outs;
    uint32_t n_outs;
    // Run bytes c (byte j of run_bytes): their patterns c^r rest, r >= 3, hang in
    // a trie over the rests whose root is dense table run_root[j]. A node of the
    // other trie with kDictPathFlag has a child for c, which has one, and so on:
    // paths holds the length K of that run, the 64-bit mask of its nodes that
    // have a pattern (bit 0: the first), where their patterns begin in outs (one
    // each), and the K nodes.
    uint32_t n_runs, run_bytes;
    uint32_t run_root[kDictMaxRuns];
    const uint32_t *paths;
};
constexpr uint32_t kDictDenseMin = 8;
constexpr uint32_t kDictDenseFlag = 0x80000000u;
constexpr uint32_t kDictPathFlag = 0x40000000u;
constexpr uint32_t kDictOneFlag = 0x40000000u;  // in a node's patterns
constexpr uint32_t kDictEdgeMask = 0x1FFu;
constexpr uint32_t kDictPathMin = 3;          // shorter runs are walked node by node
constexpr uint32_t kDictPathWords = 1u << 19;  // addressable words of paths (nodes past them go without)

// What a search decides from its sample counts, on the device.
struct DictPlan {
    uint32_t n_heavy;      // patterns whose hits go to bitmaps
    uint32_t n_run_light;  // run patterns that are not among them
    unsigned long long light_sample;  // hits of the others in the sample
};
struct DictPlanArgs {
    DictSet set;
    const uint32_t *sample_counts;  // [n_u]
    uint32_t least;                 // sample count of a heavy pattern
    const uint32_t *runs;           // the set's run patterns, as DictMatchArgs::run_light has them
    uint32_t n_runs;
    uint8_t *heavy_of_u;            // the rest: written
    uint32_t *heavy_u, *heavy_run, *run_light, *outs;
    DictPlan *plan;
};
cudaError_t launch_dict_plan(const DictPlanArgs &a, cudaStream_t st);

struct DictMatchArgs {
    DictSet set;
    const uint8_t *text;     // padded like every resident text
    uint64_t text_len;
    uint32_t n_tiles;
    uint32_t tile_stride;    // tiles 0, s, 2s, ... (count mode samples)
    uint32_t count_only;     // 1: counts[u] += every hit; 0: heavy bitmaps + light keys
    uint32_t *counts;        // per unique pattern (count mode: all hits; else light hits)
    const DictPlan *plan;    // (not in count mode)
    uint32_t *bitmap;        // [n_heavy][n_tiles * kDictWordsPerTile]
    uint32_t *heavy_counts;  // [n_heavy][heavy_ld]: += hits per tile
    uint32_t heavy_ld;
    uint32_t slices;         // consecutive slices per item (set by the launch)
    unsigned long long *light_keys;  // (u << off_bits) | offset, unordered
    uint32_t off_bits;
    uint32_t light_cap;
    uint32_t *light_n;
    uint32_t *error;
    // Batches: hits must lie inside one document, [seg_start[i], seg_end[i])
    // (sorted, disjoint); nullptr: the whole text is one document.
    const unsigned long long *seg_start;
    const unsigned long long *seg_end;
    uint32_t n_seg;
    unsigned long long *stats;  // optional: += candidates walked, trie nodes visited
    const uint32_t *outs;       // set.outs, with (heavy index + 1) << 16 of the heavy patterns (launch_dict_plan)
    const uint32_t *heavy_run;  // [kDictMaxHeavy]: (j << 8) | k of a heavy run pattern run_byte(j)^k, else 0
    const uint32_t *run_light;  // (j << 24) | (k << 16) | u of the run patterns that are not heavy (count mode: all)
    uint32_t n_run_light;       // (count mode; else the plan's)
    // Test hook (ol_ctx_inject): each block takes its wait-timeout branch
    // after its filter copy has landed, as if the bounded wait had run out.
    uint32_t force_timeout;
};

cudaError_t launch_dict_match(const DictMatchArgs &a, int sm_count, cudaStream_t st, uint32_t slice = 512,
                              uint32_t blocks_per_sm = 0);
// Radix sort of n different 64-bit keys on bits [0, key_bits), 8 per pass;
// *sorted is where the result is, keys or tmp; hist needs
// 2 * 256 * scan_ld(dict_sort_blocks(n)) words, totals 256 words.
cudaError_t launch_dict_sort(unsigned long long *keys, unsigned long long *tmp, uint32_t n, uint32_t key_bits,
                             uint32_t *hist, uint32_t *totals, unsigned long long **sorted, cudaStream_t st);
uint32_t dict_sort_blocks(uint32_t n);

struct DictEmitArgs {
    uint32_t n_ids, n_u, n_heavy, n_tiles;  // n_heavy: at least the plan's
    const DictPlan *plan;
    const uint32_t *u_of_id;
    const uint32_t *dup_start;   // [n_u + 1]
    const uint32_t *dup_ids;     // ids grouped by unique pattern, ascending
    const uint8_t *heavy_of_u;
    const uint32_t *heavy_u;     // [n_heavy]
    const uint32_t *heavy_totals;
    const uint32_t *heavy_counts, *heavy_bases;  // [n_heavy][ld], per tile
    uint32_t ld;
    const uint32_t *bitmap;
    const uint32_t *light_count; // [n_u]
    uint32_t *light_base;        // [n_u] (written by the id pass)
    const unsigned long long *light_keys;  // sorted
    const uint32_t *light_n_dev;
    uint32_t light_max;          // more light keys than this are not emitted
    uint32_t off_bits;
    uint32_t *id_counts;         // [n_ids]
    unsigned long long *id_base; // [n_ids]
    unsigned long long *total;
    uint2 *hits;                 // {pattern, offset}
    unsigned long long max_hits;
    // The (pattern u32, offset u64) form: when hit_off is set, hits go to
    // these two arrays instead of `hits`.
    uint32_t *hit_pat;
    unsigned long long *hit_off;
};
cudaError_t launch_dict_ids(const DictEmitArgs &a, cudaStream_t st);
// The same after a sort of the light keys (in place) in one launch, when there
// are at most kDictSortBlock of them; more are left unsorted.
cudaError_t launch_dict_sort_ids(const DictEmitArgs &a, unsigned long long *keys, uint32_t key_bits, cudaStream_t st);

// Digests (digest.cu): *out += sum of per-element hashes of a[0..n).
cudaError_t launch_digest_u32(const uint32_t *a, uint64_t n, uint32_t seed, unsigned long long *out, cudaStream_t st);
cudaError_t launch_digest_u8(const uint8_t *a, uint64_t n, uint32_t seed, unsigned long long *out, cudaStream_t st);

// Batches (batch.cu).
cudaError_t launch_batch_line_starts(const uint32_t *offsets, uint32_t L, const unsigned long long *seg_start, uint32_t n,
                                     uint32_t *line_start, cudaStream_t st);
cudaError_t launch_batch_tree_fixup(const uint32_t *line_start, uint32_t n, uint32_t L, const uint8_t *kinds,
                                    const uint32_t *parent_in, const uint32_t *end_in, const uint32_t *fc_in,
                                    uint32_t *parent, uint32_t *subtree_end, uint32_t *first_child,
                                    uint32_t *next_sibling, cudaStream_t st);
cudaError_t launch_dict_emit(const DictEmitArgs &a, cudaStream_t st);

// One document of a batch copied from the caller's bytes (uploaded as they
// lie) to its place in the batch text: len bytes from in + src to text + dst,
// then a '\n' at text + dst + len when sep is set (batch_pack).
struct BatchPackDoc {
    uint64_t src, dst, len;
    uint32_t sep, pad;
};
// Work items of a document (batch_pack_kernel: kBatchPackBytes each, at least one).
constexpr uint32_t kBatchPackBytes = 65536;
uint32_t batch_pack_items(uint64_t len);
cudaError_t launch_batch_pack(const BatchPackDoc *docs, const uint32_t *item_start, uint32_t n, uint32_t items,
                              const uint8_t *in, uint8_t *text, cudaStream_t st);

// One document of a batch and the buffers it is copied into (batch_split).
struct BatchSplitDoc {
    uint64_t text_start, text_len;  // bytes of the batch text
    uint32_t first_line, lines;     // lines of the batch
    uint8_t *text;
    uint32_t *offsets;
    uint8_t *kinds, *depth8;
    uint32_t *parent, *subtree_end, *first_child, *next_sibling;
};
struct BatchSplitSrc {
    const uint8_t *text;
    const uint32_t *offsets;
    const uint8_t *kinds, *depth8;
    const uint32_t *parent, *subtree_end, *first_child, *next_sibling;
};
// Work items of a document (batch_split_kernel: 4096 bytes and 1024 lines each).
uint32_t batch_split_items(uint64_t text_len, uint32_t lines);
// item_start[i]: the first work item of document i (a prefix sum of
// batch_split_items); items: their total.
cudaError_t launch_batch_split(const BatchSplitDoc *docs, const uint32_t *item_start, uint32_t n, uint32_t items,
                               const BatchSplitSrc &src, uint32_t *max_depth, cudaStream_t st);

}  // namespace ol
