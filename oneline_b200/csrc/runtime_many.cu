// C ABI for dictionary search: GpuParser::compile_patterns / search_many and
// GpuPatternSet::{len, is_empty} (crates/oneline-gpu/src/many.rs:139-176,
// 391-646). Hits are every (pattern, offset), duplicates once per id, ordered
// by (pattern, offset) as ManyPatterns orders them
// (crates/oneline-simd/src/search.rs:259-282).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "runtime.h"

using namespace ol;

struct ol_patset {
    ol_ctx *ctx = nullptr;
    uint32_t n_ids = 0, n_u = 0, n_nodes = 0;
    DevBuf blob;
    DictSet dev{};
    const uint32_t *u_of_id = nullptr, *dup_start = nullptr, *dup_ids = nullptr;
    const uint32_t *d_runs = nullptr;  // device: the run patterns, as DictMatchArgs::run_light has them
    std::vector<uint32_t> runs;        // the same on the host
};

namespace {

struct TrieNode {
    std::vector<std::pair<uint8_t, uint32_t>> kids;
    std::vector<uint32_t> outs;  // patterns that end here: (r << 24) | u
    int in = -1;                 // byte of the edge from the parent (-1: an entry)
    bool rest = false;           // in a run byte's trie
    bool walked = false;         // walks reach it: at depth 4 or more of the other trie
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

uint32_t bits_for(uint32_t v) {  // bits needed to hold values 0..v
    uint32_t b = 0;
    while (b < 32 && (v >> b)) b++;
    return b;
}

// Words a search reads back: one copy, together with the id counts.
struct ManyMeta {
    DictPlan plan;
    uint32_t light_n, error;
    unsigned long long total, walked, nodes;
};

}  // namespace

extern "C" ol_status ol_patset_compile(ol_ctx *ctx, const ol_doc *doc, const uint8_t *const *patterns,
                                       const uint32_t *lens, uint32_t n, ol_patset **out) {
    (void)doc;  // the reference samples the document to size its filter; this filter is fixed
    if (!ctx || !out || (n && (!patterns || !lens))) return OL_ERR_INVALID_ARG;
    *out = nullptr;
    if (n == 0 || n > OL_MAX_DICT_PATTERNS)
        return ctx_fail(ctx, OL_ERR_BAD_PATTERN,
                        "pattern count " + std::to_string(n) + " is outside 1.." + std::to_string(OL_MAX_DICT_PATTERNS));
    for (uint32_t i = 0; i < n; i++)
        if (!patterns[i] || lens[i] < OL_MIN_SET_PATTERN_LEN || lens[i] > OL_MAX_SET_PATTERN_LEN)
            return ctx_fail(ctx, OL_ERR_BAD_PATTERN,
                            "pattern " + std::to_string(i) + " has " + std::to_string(lens[i]) + " bytes; set patterns need " +
                                std::to_string(OL_MIN_SET_PATTERN_LEN) + ".." + std::to_string(OL_MAX_SET_PATTERN_LEN));

    // Unique patterns, in order of first appearance.
    std::unordered_map<std::string, uint32_t> uniq;
    std::vector<uint32_t> u_of_id(n);
    std::vector<const std::string *> u_str;
    uniq.reserve(n * 2);
    for (uint32_t i = 0; i < n; i++) {
        auto r = uniq.emplace(std::string((const char *)patterns[i], lens[i]), (uint32_t)uniq.size());
        if (r.second) u_str.push_back(&r.first->first);
        u_of_id[i] = r.first->second;
    }
    const uint32_t U = (uint32_t)u_str.size();

    // Run bytes: the (at most four) bytes c with the most unique patterns that
    // start with c^4. '\n' is left to the trie: a run of any other byte lies
    // inside one document of a batch.
    std::vector<uint32_t> starts(256, 0);
    auto leading = [](const std::string &p) {  // length of the run that p starts with
        size_t r = 1;
        while (r < p.size() && p[r] == p[0]) r++;
        return (uint32_t)r;
    };
    for (const std::string *p : u_str)
        if ((*p)[0] != '\n' && leading(*p) >= 4) starts[(uint8_t)(*p)[0]]++;
    std::vector<uint32_t> run_bytes;
    for (uint32_t c = 0; c < 256; c++)
        if (starts[c]) run_bytes.push_back(c);
    std::sort(run_bytes.begin(), run_bytes.end(), [&](uint32_t x, uint32_t y) { return starts[x] > starts[y]; });
    if (run_bytes.size() > kDictMaxRuns) run_bytes.resize(kDictMaxRuns);
    const uint32_t n_runs = (uint32_t)run_bytes.size();

    // The run bytes' tries (roots: nodes 1 .. n_runs) over what follows c^r in
    // the patterns that start with c^3, and the trie over all other patterns
    // (root: node 0) with the node after the first four bytes of each.
    std::vector<TrieNode> trie(1 + n_runs);
    std::unordered_map<uint32_t, uint32_t> key_node;
    std::vector<uint32_t> filter_keys, runs;
    for (uint32_t u = 0; u < U; u++) {
        const std::string &p = *u_str[u];
        uint32_t v = 0;
        size_t first = 0;
        const uint32_t r = leading(p);
        for (uint32_t j = 0; r >= 3 && j < n_runs; j++) {
            if (run_bytes[j] != (uint8_t)p[0]) continue;
            v = 1 + j;
            first = r;
        }
        if (v && first == p.size()) {  // c^k (k >= 4)
            runs.push_back(((v - 1) << 24) | (r << 16) | u);
            continue;
        }
        uint32_t key;
        memcpy(&key, p.data() + (v ? first - 3 : 0), 4);  // c c c rest[0], or the first four bytes
        filter_keys.push_back(key);
        for (size_t j = first; j < p.size(); j++) {
            uint8_t b = (uint8_t)p[j];
            uint32_t next = NONE;
            for (auto &k : trie[v].kids)
                if (k.first == b) next = k.second;
            if (next == NONE) {
                next = (uint32_t)trie.size();
                trie[v].kids.emplace_back(b, next);
                trie.emplace_back();
                trie[next].rest = first != 0;
                trie[next].walked = !first && j >= kDictMinLen - 1;
                trie[next].in = j == (first ? first : kDictMinLen - 1) ? -1 : b;
            }
            v = next;
            if (!first && j == kDictMinLen - 1) key_node[key] = v;
        }
        trie[v].outs.push_back(((first ? r : 0u) << 24) | u);
    }
    const uint32_t n_nodes = (uint32_t)trie.size();
    if (n_nodes >= (1u << 24)) return ctx_fail(ctx, OL_ERR_BAD_PATTERN, "pattern set too large for the trie");
    std::vector<uint4> nodes(n_nodes);
    std::vector<uint32_t> extra, dense, outs, paths, path_of(n_nodes, NONE);
    std::vector<uint4> lists;
    // The runs of run bytes in the trie (kDictPathFlag), and their nodes' patterns.
    for (uint32_t v = n_runs + 1; v < n_nodes; v++) nodes[v].x = NONE;
    for (uint32_t v = n_runs + 1; v < n_nodes; v++) {
        for (uint32_t j = 0; j < n_runs && path_of[v] == NONE && trie[v].walked; j++) {
            if (trie[v].in == (int)run_bytes[j]) continue;  // the run begins before v
            std::vector<uint32_t> run;
            for (uint32_t x = v; x != NONE;) {
                uint32_t next = NONE;
                for (auto &e : trie[x].kids)
                    if (e.first == run_bytes[j]) next = e.second;
                if (next != NONE) run.push_back(next);
                x = next;
            }
            if (run.size() < kDictPathMin || paths.size() + 4 + run.size() > kDictPathWords) continue;
            path_of[v] = (j << 28) | ((uint32_t)paths.size() << 9);
            uint64_t mask = 0;
            const uint32_t first = (uint32_t)outs.size();
            for (uint32_t i = 0; i < run.size(); i++) {  // at most 60
                const TrieNode &x = trie[run[i]];
                if (x.outs.empty()) continue;
                mask |= 1ull << i;
                nodes[run[i]].x = kDictOneFlag | (uint32_t)outs.size();
                outs.push_back(x.outs[0]);
            }
            paths.insert(paths.end(), {(uint32_t)run.size(), (uint32_t)mask, (uint32_t)(mask >> 32), first});
            paths.insert(paths.end(), run.begin(), run.end());
        }
    }
    for (uint32_t v = 0; v < n_nodes; v++) {
        auto &o = trie[v].outs;
        if (v <= n_runs) nodes[v].x = NONE;
        if (o.empty() || nodes[v].x != NONE) continue;
        if (!trie[v].rest) {  // one pattern: they are unique
            nodes[v].x = kDictOneFlag | (uint32_t)outs.size();
            outs.push_back(o[0]);
            continue;
        }
        std::sort(o.begin(), o.end());  // r ascending, 3..63
        nodes[v].x = (uint32_t)lists.size();
        uint4 l{0, 0, (uint32_t)outs.size(), 0};
        for (uint32_t x : o) {
            (x >> 24 < 32 ? l.x : l.y) |= 1u << ((x >> 24) & 31);
            outs.push_back(x & 0xFFFFFFu);
        }
        lists.push_back(l);
    }
    outs.push_back(0);
    for (uint32_t v = 0; v < n_nodes; v++) {
        auto &k = trie[v].kids;
        std::sort(k.begin(), k.end());
        uint4 r{nodes[v].x, (uint32_t)k.size(), 0, 0};
        if (path_of[v] != NONE) r.y |= kDictPathFlag | path_of[v];
        auto pack = [](const std::pair<uint8_t, uint32_t> &e) { return (e.second << 8) | e.first; };
        if (k.size() > kDictDenseMin || (v >= 1 && v <= n_runs)) {
            // many children: a 256-entry table, one load per step
            r.y |= kDictDenseFlag;
            r.w = (uint32_t)(dense.size() / 256);
            dense.resize(dense.size() + 256, NONE);
            for (auto &e : k) dense[(size_t)r.w * 256 + e.first] = e.second;
        } else {
            if (!k.empty()) r.z = pack(k[0]);
            if (k.size() == 2) r.w = pack(k[1]);
            if (k.size() > 2) {
                r.w = (uint32_t)extra.size();
                for (size_t i = 1; i < k.size(); i++) extra.push_back(pack(k[i]));
            }
        }
        nodes[v] = r;
    }
    if (extra.empty()) extra.push_back(0);
    if (dense.empty()) dense.push_back(NONE);
    if (paths.empty()) paths.push_back(0);

    // The filter, and the hash table over the distinct first-four-byte keys.
    std::vector<uint32_t> filter(1u << (kDictFilterBits - 5), 0);
    uint32_t table_bits = 10;
    while ((1u << table_bits) < 2 * key_node.size()) table_bits++;
    std::vector<uint2> table(1u << table_bits, make_uint2(0, NONE));
    uint32_t max_probe = 0;
    for (uint32_t key : filter_keys) {
        const uint32_t g = dict_filter_bits(key);
        filter[dict_filter_word(key)] |= (1u << (g >> 27)) | (1u << ((g >> 22) & 31)) | (1u << ((g >> 17) & 31));
    }
    for (auto &kv : key_node) {
        uint32_t key = kv.first;
        uint32_t slot = dict_table_h(key, table_bits), dist = 0;
        while (table[slot].y != NONE) {
            slot = (slot + 1) & ((1u << table_bits) - 1);
            dist++;
        }
        table[slot] = make_uint2(key, kv.second);
        max_probe = std::max(max_probe, dist);
    }

    // Ids grouped by unique pattern.
    std::vector<uint32_t> dup_start(U + 1, 0), dup_ids(n);
    for (uint32_t i = 0; i < n; i++) dup_start[u_of_id[i] + 1]++;
    for (uint32_t u = 0; u < U; u++) dup_start[u + 1] += dup_start[u];
    {
        std::vector<uint32_t> fill(dup_start.begin(), dup_start.end() - 1);
        for (uint32_t i = 0; i < n; i++) dup_ids[fill[u_of_id[i]]++] = i;
    }

    // One device blob.
    size_t off_filter = 0, sz_filter = filter.size() * 4;
    size_t off_table = align256(off_filter + sz_filter), sz_table = table.size() * 8;
    size_t off_nodes = align256(off_table + sz_table), sz_nodes = nodes.size() * 16;
    size_t off_extra = align256(off_nodes + sz_nodes), sz_extra = extra.size() * 4;
    size_t off_dense = align256(off_extra + sz_extra), sz_dense = dense.size() * 4;
    size_t off_uid = align256(off_dense + sz_dense), sz_uid = (size_t)n * 4;
    size_t off_ds = align256(off_uid + sz_uid), sz_ds = dup_start.size() * 4;
    size_t off_di = align256(off_ds + sz_ds), sz_di = dup_ids.size() * 4;
    size_t off_outs = align256(off_di + sz_di), sz_outs = outs.size() * 4;
    size_t off_runs = align256(off_outs + sz_outs), sz_runs = runs.size() * 4;
    size_t off_paths = align256(off_runs + std::max<size_t>(sz_runs, 4)), sz_paths = paths.size() * 4;
    size_t off_lists = align256(off_paths + sz_paths), sz_lists = lists.size() * sizeof(uint4);
    size_t total = align256(off_lists + sz_lists);
    std::vector<uint8_t> host(total, 0);
    memcpy(host.data() + off_filter, filter.data(), sz_filter);
    memcpy(host.data() + off_table, table.data(), sz_table);
    memcpy(host.data() + off_nodes, nodes.data(), sz_nodes);
    memcpy(host.data() + off_extra, extra.data(), sz_extra);
    memcpy(host.data() + off_dense, dense.data(), sz_dense);
    memcpy(host.data() + off_uid, u_of_id.data(), sz_uid);
    memcpy(host.data() + off_ds, dup_start.data(), sz_ds);
    memcpy(host.data() + off_di, dup_ids.data(), sz_di);
    memcpy(host.data() + off_outs, outs.data(), sz_outs);
    if (sz_runs) memcpy(host.data() + off_runs, runs.data(), sz_runs);
    memcpy(host.data() + off_paths, paths.data(), sz_paths);
    if (sz_lists) memcpy(host.data() + off_lists, lists.data(), sz_lists);

    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    ol_patset *s = new ol_patset();
    s->ctx = ctx;
    s->n_ids = n;
    s->n_u = U;
    s->n_nodes = n_nodes;
    cudaError_t e = s->blob.reserve(total, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(s->blob.ptr, host.data(), total, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        s->blob.release(ctx->stream);
        delete s;
        return ctx_cuda(ctx, e, "compile_patterns");
    }
    uint8_t *b = (uint8_t *)s->blob.ptr;
    s->dev.filter = (const uint32_t *)(b + off_filter);
    s->dev.table = (const uint2 *)(b + off_table);
    s->dev.table_bits = table_bits;
    s->dev.max_probe = max_probe;
    s->dev.nodes = (const uint4 *)(b + off_nodes);
    s->dev.extra = (const uint32_t *)(b + off_extra);
    s->dev.dense = (const uint32_t *)(b + off_dense);
    s->dev.n_u = U;
    s->u_of_id = (const uint32_t *)(b + off_uid);
    s->dup_start = (const uint32_t *)(b + off_ds);
    s->dup_ids = (const uint32_t *)(b + off_di);
    s->dev.lists = (const uint4 *)(b + off_lists);
    s->dev.outs = (const uint32_t *)(b + off_outs);
    s->dev.n_outs = (uint32_t)outs.size();
    s->dev.paths = (const uint32_t *)(b + off_paths);
    s->dev.n_runs = n_runs;
    for (uint32_t j = 0; j < n_runs; j++) {
        s->dev.run_bytes |= run_bytes[j] << (8 * j);
        s->dev.run_root[j] = nodes[1 + j].w;
    }
    s->d_runs = (const uint32_t *)(b + off_runs);
    s->runs = std::move(runs);
    *out = s;
    return OL_OK;
}

extern "C" void ol_patset_free(ol_patset *s) {
    if (!s) return;
    if (s->ctx) {
        std::lock_guard<std::recursive_mutex> g(s->ctx->mu);
        cudaSetDevice(s->ctx->device);
        s->blob.release(s->ctx->stream);
    }
    delete s;
}

extern "C" uint32_t ol_patset_len(const ol_patset *s) { return s ? s->n_ids : 0; }
extern "C" uint32_t ol_patset_unique(const ol_patset *s) { return s ? s->n_u : 0; }


// The whole search; hits go to d_hits (capacity max_hits) when given, else to
// host_hits through ctx->dict_hits. counts (n_ids) and *total are host outputs.
// seg_start/seg_end (device, n_seg): batches, whose hits stay inside a document.
//
// The host waits as seldom as the sizes allow. Texts of up to kPlanTiles tiles
// go from the sample to the match pass on the device's own plan, with scratch
// for as many heavy patterns as there can be; larger ones read the plan first.
// With up to kFewTiles tiles the light keys are taken to be few enough for one
// block to sort; if they were not, the host learns it with the counts, sorts
// them and places the ids (and writes device hits) once more.
// Device hits, in us. The device's plan / a plan that is read: 1 MiB and 100 patterns
// 100 / 114, 4 MiB 126 / 148, 16 MiB 182 / 196, 32 MiB 226 / 245; past 64 MiB these
// 15 to 20 us are 1 to 5 % of the search, and bitmaps for 32 patterns, 4 bytes a text
// byte, are not worth them. One block's sort tried / the count read first: 100 patterns 1 MiB 100 / 114,
// 2 MiB 107 / 121, 4 MiB (256 tiles) 126 / 127, and tried past that 10,000 patterns in
// 8 MiB 593 / 475; with so many patterns the try is lost below 4 MiB too (1 MiB 440 / 365).
// Sample tiles, 64 MiB and 10,000 patterns: 40 1398, 160 1424, 640 1485 (fewer tell
// frequent patterns less surely).
constexpr uint32_t kPlanTiles = 4096, kFewTiles = 256, kSampleTiles = 160;

ol_status ol::many_run(ol_ctx *ctx, const ol_doc *d, const ol_patset *set, uint64_t max_hits, uint32_t heavy_min_hits,
                       uint32_t *counts, uint64_t *total, const HitDest &dest,
                       const unsigned long long *seg_start, const unsigned long long *seg_end, uint32_t n_seg) {
    cudaStream_t st = ctx->stream;
    const uint32_t n = set->n_ids, U = set->n_u;
    const uint64_t N = d->text_len;
    *total = 0;
    memset(counts, 0, (size_t)n * 4);
    if (N < kDictMinLen) return OL_OK;
    const uint32_t n_tiles = (uint32_t)((N + kDictTile - 1) / kDictTile);
    const uint32_t n_words = n_tiles * kDictWordsPerTile, hld = scan_ld(n_tiles);
    const uint32_t off_bits = std::max<uint32_t>(bits_for((uint32_t)(N - 1)), 1), key_bits = off_bits + bits_for(U - 1);

    // Scratch, carved from ctx->dict_small. Id counts and meta are read back
    // together; meta's counters up to the sample counts start from zero.
    size_t at = 0;
    auto carve = [&](size_t bytes, size_t align = 16) {
        at = (at + align - 1) & ~(align - 1);
        const size_t o = at;
        at += bytes;
        return o;
    };
    const size_t o_idc = carve((size_t)n * 4), o_meta = carve(sizeof(ManyMeta));
    const size_t o_lcount = carve((size_t)U * 4), o_hcounts = carve((size_t)kDictMaxHeavy * hld * 4), rezero_end = at;
    const size_t o_sample = carve((size_t)U * 4), zero_end = at;
    const size_t o_lbase = carve((size_t)U * 4), o_heavy_of = carve(U), o_heavy_u = carve(kDictMaxHeavy * 4);
    const size_t o_htot = carve(kDictMaxHeavy * 4), o_hbases = carve((size_t)kDictMaxHeavy * hld * 4);
    const size_t o_hrun = carve(kDictMaxHeavy * 4), o_rlight = carve(std::max<size_t>(set->runs.size(), 1) * 4);
    const size_t o_outs = carve((size_t)set->dev.n_outs * 4), o_idb = carve((size_t)n * 8), o_stot = carve(256 * 4);
    cudaError_t e = ctx->dict_small.reserve(at, st);
    const size_t back = o_meta + sizeof(ManyMeta);  // bytes read back
    if (e == cudaSuccess) e = ctx->host_words.reserve(back);
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many");
    uint8_t *b = (uint8_t *)ctx->dict_small.ptr;
    ManyMeta *meta = (ManyMeta *)(b + o_meta);
    const ManyMeta *hm = (const ManyMeta *)(ctx->host_words.ptr + o_meta);
    uint32_t *light_count = (uint32_t *)(b + o_lcount), *heavy_counts = (uint32_t *)(b + o_hcounts);
    uint32_t *heavy_bases = (uint32_t *)(b + o_hbases), *heavy_totals = (uint32_t *)(b + o_htot);
    const size_t o_zero = o_meta + offsetof(ManyMeta, light_n);
    auto read_meta = [&]() -> cudaError_t {  // id counts and meta, as the stream has them now
        cudaError_t r = cudaMemcpyAsync(ctx->host_words.ptr, b, back, cudaMemcpyDeviceToHost, st);
        return r == cudaSuccess ? cudaStreamSynchronize(st) : r;
    };

    // 1. Counts on a sample of tiles (every tile when the text is small) pick
    //    the heavy patterns: those expected to have at least `threshold` hits.
    const uint32_t sample = std::min(std::max(n_tiles / 8, 4u), kSampleTiles), stride = std::max<uint32_t>(1, n_tiles / sample);
    const uint32_t n_work = (n_tiles + stride - 1) / stride;
    const double scale = (double)n_tiles / (double)n_work;
    const double threshold = heavy_min_hits ? (double)heavy_min_hits
                                            : std::max(4096.0, (double)N / (double)std::max<uint32_t>(ctx->tune.dict_heavy_divisor, 1));
    DictMatchArgs ma{};
    ma.set = set->dev;
    ma.text = d->text;
    ma.text_len = N;
    ma.n_tiles = n_tiles;
    ma.tile_stride = stride;
    ma.count_only = 1;
    ma.counts = (uint32_t *)(b + o_sample);
    ma.error = &meta->error;
    ma.outs = set->dev.outs;
    ma.run_light = set->d_runs;
    ma.n_run_light = (uint32_t)set->runs.size();
    ma.seg_start = seg_start;
    ma.seg_end = seg_end;
    ma.n_seg = n_seg;
    // an armed injected timeout is taken by this search's first match pass
    ma.force_timeout = (ctx->inject & OL_INJECT_DICT_WAIT_TIMEOUT) ? 1u : 0u;
    ctx->inject &= ~OL_INJECT_DICT_WAIT_TIMEOUT;
    e = cudaMemsetAsync(b + o_zero, 0, zero_end - o_zero, st);
    if (e == cudaSuccess) {
        GpuPass pass(ctx, "dictionary: sample counts");
        e = launch_dict_match(ma, ctx->sm_count, st, ctx->tune.dict_slice, ctx->tune.dict_blocks_per_sm);
    }
    DictPlanArgs pa{};
    pa.set = set->dev;
    pa.sample_counts = ma.counts;
    pa.least = (uint32_t)std::min(std::max(std::ceil(threshold / scale), 1.0), 4294967295.0);
    pa.runs = set->d_runs;
    pa.n_runs = (uint32_t)set->runs.size();
    pa.heavy_of_u = b + o_heavy_of;
    pa.heavy_u = (uint32_t *)(b + o_heavy_u);
    pa.heavy_run = (uint32_t *)(b + o_hrun);
    pa.run_light = (uint32_t *)(b + o_rlight);
    pa.outs = (uint32_t *)(b + o_outs);
    pa.plan = &meta->plan;
    if (e == cudaSuccess) e = launch_dict_plan(pa, st);
    uint32_t H = std::min(kDictMaxHeavy, U);  // as many as there can be
    uint64_t cap = std::max<uint64_t>(N / 16, 65536);
    auto read_plan = [&]() -> ol_status {  // as many heavy patterns and light hits as the sample promises
        cudaError_t r = read_meta();
        prof_mark(ctx, "dictionary: wait for the sample");
        if (r != cudaSuccess) return ctx_cuda(ctx, r, "search_many sample");
        if (hm->error & OL_DEVERR_TIMEOUT) return ctx_fail(ctx, OL_ERR_TIMEOUT, "search_many: a bounded wait ran out");
        H = hm->plan.n_heavy;
        cap = std::min<uint64_t>(0xFFFFFFF0ull, (uint64_t)((double)hm->plan.light_sample * scale * 1.25) + 65536);
        return OL_OK;
    };
    auto reserve_hits = [&]() -> cudaError_t {  // the bitmaps and the first attempt's keys
        cudaError_t r = H ? ctx->dict_bitmap.reserve((size_t)H * n_words * 4, st) : cudaSuccess;
        return r == cudaSuccess ? ctx->dict_keys.reserve((size_t)cap * 16, st) : r;
    };
    ol_status ps = OL_OK;
    if (e == cudaSuccess && n_tiles > kPlanTiles) ps = read_plan();
    if (ps != OL_OK) return ps;
    if (e == cudaSuccess) e = reserve_hits();
    if (e == cudaErrorMemoryAllocation && n_tiles <= kPlanTiles) {
        // no memory for all there can be (at most 5 bytes a text byte): what the sample promises may fit
        cudaGetLastError();
        ctx->dict_bitmap.release(st);
        ctx->dict_keys.release(st);
        if ((ps = read_plan()) != OL_OK) return ps;
        e = reserve_hits();
    }
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many");

    // 2. The match pass; 3. heavy ranks, light order, per-id slots; 4. hits.
    //    The light keys' buffer is grown and the match pass run again if they
    //    overflow it.
    DictEmitArgs ea{};
    auto timed_out = [&]() { return (hm->error & OL_DEVERR_TIMEOUT) != 0; };
    auto hits_dest = [&](uint64_t k) -> cudaError_t {  // where hits go on the device: k of them
        if (dest.off && !dest.pair_on_host) {
            ea.hit_pat = dest.pat;
            ea.hit_off = reinterpret_cast<unsigned long long *>(dest.off);
        } else if (dest.dev) {
            ea.hits = reinterpret_cast<uint2 *>(dest.dev);
        } else {
            const size_t off_at = (k * 4 + 255) & ~(size_t)255;  // pair form in scratch: patterns, then offsets
            cudaError_t r = ctx->dict_hits.reserve(dest.off ? off_at + k * 8 : k * 8, st);
            if (r != cudaSuccess) return r;
            if (dest.off) {
                ea.hit_pat = (uint32_t *)ctx->dict_hits.ptr;
                ea.hit_off = (unsigned long long *)((uint8_t *)ctx->dict_hits.ptr + off_at);
            } else {
                ea.hits = (uint2 *)ctx->dict_hits.ptr;
            }
        }
        ea.max_hits = k;
        return cudaSuccess;
    };
    const bool on_device = max_hits && (dest.dev || (dest.off && !dest.pair_on_host));
    bool emitted = false;
    for (int attempt = 0;; attempt++) {
        e = ctx->dict_keys.reserve((size_t)cap * 16, st);
        cap = std::min<uint64_t>(ctx->dict_keys.bytes / 16, 0xFFFFFFF0ull);
        if (e == cudaSuccess && attempt) e = cudaMemsetAsync(b + o_zero, 0, rezero_end - o_zero, st);
        unsigned long long *keys = (unsigned long long *)ctx->dict_keys.ptr;
        ma.stats = &meta->walked;
        ma.force_timeout = 0;
        ma.tile_stride = 1;
        ma.count_only = 0;
        ma.counts = light_count;
        ma.plan = pa.plan;
        ma.bitmap = (uint32_t *)ctx->dict_bitmap.ptr;
        ma.heavy_counts = heavy_counts;
        ma.heavy_ld = hld;
        ma.light_keys = keys;
        ma.off_bits = off_bits;
        ma.light_cap = (uint32_t)cap;
        ma.light_n = &meta->light_n;
        ma.outs = pa.outs;
        ma.heavy_run = pa.heavy_run;
        ma.run_light = pa.run_light;
        if (e == cudaSuccess) {
            GpuPass pass(ctx, "dictionary: match");
            e = launch_dict_match(ma, ctx->sm_count, st, ctx->tune.dict_slice, ctx->tune.dict_blocks_per_sm);
        }
        bool known = n_tiles > kFewTiles;  // the light key count, on the host
        if (e == cudaSuccess && known) e = read_meta();
        if (known) prof_mark(ctx, "dictionary: wait for the match pass");
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many match");
        if (known && timed_out()) return ctx_fail(ctx, OL_ERR_TIMEOUT, "search_many: a bounded wait ran out");
        if (known && hm->light_n > cap) {
            if (attempt == 2) return ctx_fail(ctx, OL_ERR_CUDA, "search_many: light hit count kept growing");
            cap = (uint64_t)hm->light_n + 1024;
            continue;
        }
        ea.n_ids = n;
        ea.n_u = U;
        ea.n_heavy = H;
        ea.n_tiles = n_tiles;
        ea.plan = pa.plan;
        ea.u_of_id = set->u_of_id;
        ea.dup_start = set->dup_start;
        ea.dup_ids = set->dup_ids;
        ea.heavy_of_u = pa.heavy_of_u;
        ea.heavy_u = pa.heavy_u;
        ea.heavy_totals = heavy_totals;
        ea.heavy_counts = heavy_counts;
        ea.heavy_bases = heavy_bases;
        ea.ld = hld;
        ea.bitmap = (const uint32_t *)ctx->dict_bitmap.ptr;
        ea.light_count = light_count;
        ea.light_base = (uint32_t *)(b + o_lbase);
        ea.light_keys = keys;
        ea.light_n_dev = &meta->light_n;
        ea.light_max = known ? hm->light_n : kDictSortBlock;
        ea.off_bits = off_bits;
        ea.id_counts = (uint32_t *)(b + o_idc);
        ea.id_base = (unsigned long long *)(b + o_idb);
        ea.total = &meta->total;
        auto order = [&]() -> cudaError_t {  // light order and per-id slots
            cudaError_t r;
            if (!known || hm->light_n <= kDictSortBlock) return launch_dict_sort_ids(ea, keys, key_bits, st);
            const uint32_t light_n = hm->light_n;
            r = ctx->dict_sort.reserve((size_t)2 * 256 * scan_ld(dict_sort_blocks(light_n)) * 4, st);
            unsigned long long *sorted = keys;
            if (r == cudaSuccess)
                r = launch_dict_sort(keys, keys + cap, light_n, key_bits, (uint32_t *)ctx->dict_sort.ptr, (uint32_t *)(b + o_stot),
                                     &sorted, st);
            ea.light_keys = sorted;
            ea.light_max = light_n;
            return r == cudaSuccess ? launch_dict_ids(ea, st) : r;
        };
        auto emit = [&]() {
            GpuPass pass(ctx, "dictionary: emit");
            return launch_dict_emit(ea, st);
        };
        {
            GpuPass order_pass(ctx, "dictionary: rank and sort");
            if (H) e = launch_scan_columns(heavy_counts, heavy_bases, heavy_totals, n_tiles, H, hld, st);
            if (e == cudaSuccess) e = order();
        }
        if (e == cudaSuccess && on_device) {
            e = hits_dest(max_hits);
            if (e == cudaSuccess) e = emit();
            emitted = true;
        }
        if (e == cudaSuccess) e = read_meta();
        prof_mark(ctx, "dictionary: wait for the slots");
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many");
        if (timed_out()) return ctx_fail(ctx, OL_ERR_TIMEOUT, "search_many: a bounded wait ran out");
        if (!known && hm->light_n > kDictSortBlock) {  // more light keys than one block sorts
            if (hm->light_n > cap) {
                if (attempt == 2) return ctx_fail(ctx, OL_ERR_CUDA, "search_many: light hit count kept growing");
                cap = (uint64_t)hm->light_n + 1024;
                continue;
            }
            known = true;
            GpuPass order_pass(ctx, "dictionary: rank and sort");
            e = order();
            order_pass.done();
            if (e == cudaSuccess && emitted) e = emit();
            if (e == cudaSuccess) e = read_meta();
            if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many");
        }
        break;
    }
    memcpy(counts, ctx->host_words.ptr + o_idc, (size_t)n * 4);
    *total = hm->total;
    ctx->dict_stats[0] = N;
    ctx->dict_stats[1] = hm->walked;
    ctx->dict_stats[2] = hm->nodes;
    ctx->dict_stats[3] = hm->plan.n_heavy;
    ctx->dict_stats[4] = hm->light_n;
    ctx->dict_stats[5] = hm->total;
    const uint64_t k = std::min<uint64_t>(hm->total, max_hits);
    if (k == 0 || emitted) return OL_OK;

    // Hits for the host: through scratch of their number.
    ea.n_heavy = hm->plan.n_heavy;
    ea.light_max = hm->light_n;
    e = hits_dest(k);
    if (e == cudaSuccess) {
        GpuPass pass(ctx, "dictionary: emit");
        e = launch_dict_emit(ea, st);
    }
    if (e == cudaSuccess && (dest.host || dest.pair_on_host)) {
        GpuPass pass(ctx, "download");
        if (dest.pair_on_host) {
            e = cudaMemcpyAsync(dest.pat, ea.hit_pat, k * 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(dest.off, ea.hit_off, k * 8, cudaMemcpyDeviceToHost, st);
        } else {
            e = cudaMemcpyAsync(dest.host, ea.hits, k * 8, cudaMemcpyDeviceToHost, st);
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    prof_mark(ctx, "dictionary: emit hits");
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "search_many emit");
    return OL_OK;
}

extern "C" ol_status ol_search_many(ol_ctx *ctx, const ol_doc *d, const ol_patset *set, uint64_t max_hits,
                                    uint32_t *counts, uint64_t *total_hits, ol_hit *hits) {
    if (!ctx || !d || !set || !counts || !total_hits || (max_hits && !hits)) return OL_ERR_INVALID_ARG;
    if (set->ctx != ctx) return ctx_fail(ctx, OL_ERR_INVALID_ARG, "pattern set belongs to another context");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    HitDest dest;
    dest.host = hits;
    return many_run(ctx, d, set, max_hits, 0, counts, total_hits, dest, nullptr, nullptr, 0);
}

extern "C" ol_status ol_search_many_device(ol_ctx *ctx, const ol_doc *d, const ol_patset *set, uint64_t max_hits,
                                           uint32_t heavy_min_hits, uint32_t *counts, uint64_t *total_hits,
                                           ol_hit *d_hits) {
    if (!ctx || !d || !set || !counts || !total_hits || (max_hits && !d_hits)) return OL_ERR_INVALID_ARG;
    if (set->ctx != ctx) return ctx_fail(ctx, OL_ERR_INVALID_ARG, "pattern set belongs to another context");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    HitDest dest;
    dest.dev = d_hits;
    return many_run(ctx, d, set, max_hits, heavy_min_hits, counts, total_hits, dest, nullptr, nullptr, 0);
}

extern "C" ol_status ol_search_many_u64(ol_ctx *ctx, const ol_doc *d, const ol_patset *set, uint64_t max_hits,
                                        uint32_t *counts, uint64_t *total_hits, uint32_t *patterns, uint64_t *offsets) {
    if (!ctx || !d || !set || !counts || !total_hits || (max_hits && (!patterns || !offsets))) return OL_ERR_INVALID_ARG;
    if (set->ctx != ctx) return ctx_fail(ctx, OL_ERR_INVALID_ARG, "pattern set belongs to another context");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    HitDest dest;
    dest.pat = patterns;
    dest.off = offsets;
    dest.pair_on_host = true;
    return many_run(ctx, d, set, max_hits, 0, counts, total_hits, dest, nullptr, nullptr, 0);
}

extern "C" ol_status ol_search_many_device_u64(ol_ctx *ctx, const ol_doc *d, const ol_patset *set, uint64_t max_hits,
                                               uint32_t heavy_min_hits, uint32_t *counts, uint64_t *total_hits,
                                               uint32_t *d_patterns, uint64_t *d_offsets) {
    if (!ctx || !d || !set || !counts || !total_hits || (max_hits && (!d_patterns || !d_offsets)))
        return OL_ERR_INVALID_ARG;
    if (((uintptr_t)d_offsets & 7) || ((uintptr_t)d_patterns & 3))
        return ctx_fail(ctx, OL_ERR_INVALID_ARG, "d_offsets must be 8-byte and d_patterns 4-byte aligned");
    if (set->ctx != ctx) return ctx_fail(ctx, OL_ERR_INVALID_ARG, "pattern set belongs to another context");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    HitDest dest;
    dest.pat = d_patterns;
    dest.off = d_offsets;
    return many_run(ctx, d, set, max_hits, heavy_min_hits, counts, total_hits, dest, nullptr, nullptr, 0);
}

extern "C" ol_status ol_dict_stats(ol_ctx *ctx, uint64_t *out) {
    if (!ctx || !out) return OL_ERR_INVALID_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    for (int i = 0; i < 6; i++) out[i] = ctx->dict_stats[i];
    return OL_OK;
}
