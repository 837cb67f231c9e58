// C ABI for the node query filter: GpuParser::query_document, query_subtree,
// query_raw and query (crates/oneline-gpu/src/document.rs:94-127, 165-190,
// tree.rs:292-313, query.rs:228-329). Results are QueryResult
// (query.rs:10-19): the true total and the first min(total, max_matches)
// matching line indices, ascending.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "runtime.h"

using namespace ol;

namespace {

// Matches that come back together with their number; more take a second copy.
constexpr uint32_t kQueryFirst = 16384;

// Blocks (of 4096 lines, from the root to the document's end) past which a
// subtree query reads the subtree's end first. One line's subtree, in us, end on
// the device / read first: 8 M lines 30 / 37, 16 M 33 / 34, 24 M 33 / 32, 64 M
// 47 / 32, and of 128 M 68 on the device.
constexpr uint32_t kSubtreeEndBlocks = 4096;

// Runs the filter over lines [lo, hi) of a resident document (or over `nodes`
// when given; hi_dev: the range's end on the device, at most hi) and downloads
// the result.
ol_status run_query(ol_ctx *ctx, const ol_doc *d, const FlatNode *nodes, uint32_t lines, uint32_t lo, uint32_t hi,
                    const uint32_t *hi_dev, uint32_t kind, uint32_t depth, uint32_t max_matches, uint32_t *total,
                    uint32_t *out) {
    cudaStream_t st = ctx->stream;
    *total = 0;
    if (hi <= lo) return OL_OK;
    const uint32_t blocks = query_blocks(lo, hi), ld = scan_ld(blocks), first = std::min(max_matches, kQueryFirst);
    const size_t small = ((size_t)2 * ld + 4) * 4, masks = (size_t)blocks * kQueryMasks * 2;
    cudaError_t e = ctx->search_out.reserve(small + masks + (size_t)std::max<uint32_t>(max_matches, 1) * 4, st);
    if (e == cudaSuccess) e = ctx->host_words.reserve((4 + (size_t)first) * 4);
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "query");
    uint32_t *w = (uint32_t *)ctx->search_out.ptr;
    QueryArgs a{};
    if (!nodes) {
        a.kinds = d->kinds;
        a.depth8 = d->depth8;
        a.text = d->text;
        a.offsets = d->offsets;
        a.text_len = d->text_len;
    }
    a.nodes = nodes;
    a.lines = lines;
    a.lo = lo;
    a.hi = hi;
    a.hi_dev = hi_dev;
    a.target_kind = kind;
    a.target_depth = depth;
    a.masks = (uint16_t *)w;
    w += masks / 4;
    a.counts = w;
    a.bases = w + ld;
    a.total = w + 2 * ld;  // the total, then (16 bytes on) the matches: one copy brings both
    a.out = w + 2 * ld + 4;
    a.max_out = max_matches;
    {
        GpuPass pass(ctx, "query");
        e = launch_query(a, st);
    }
    const uint32_t *back = (const uint32_t *)ctx->host_words.ptr;
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ctx->host_words.ptr, a.total, (4 + (size_t)first) * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    prof_mark(ctx, "query: wait for the count");
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "query");
    *total = back[0];
    const uint32_t k = std::min(*total, max_matches), k0 = std::min(k, first);
    if (k0) memcpy(out, back + 4, (size_t)k0 * 4);
    if (k > k0) {
        GpuPass pass(ctx, "download");
        e = cudaMemcpyAsync(out + k0, a.out + k0, (size_t)(k - k0) * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    prof_mark(ctx, "query: download matches");
    return ctx_cuda(ctx, e, "query");
}

}  // namespace

extern "C" ol_status ol_query_document(ol_ctx *ctx, const ol_doc *d, uint32_t kind, uint32_t depth, uint32_t max_matches,
                                       uint32_t *total, uint32_t *out) {
    if (!ctx || !d || !total || (max_matches && !out)) return OL_ERR_INVALID_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    return run_query(ctx, d, nullptr, d->line_count, 0, d->line_count, nullptr, kind, depth, max_matches, total,
                     out);
}

extern "C" ol_status ol_query_subtree(ol_ctx *ctx, const ol_doc *d, const ol_tree *t, uint64_t root, uint32_t kind,
                                      uint32_t depth, uint32_t max_matches, uint32_t *total, uint32_t *out) {
    if (!ctx || !d || !t || !total || (max_matches && !out)) return OL_ERR_INVALID_ARG;
    if (root >= t->line_count || t->line_count != d->line_count)
        return ctx_fail(ctx, OL_ERR_INVALID_ARG,
                        "line " + std::to_string(root) + " is out of range (document has " +
                            std::to_string(d->line_count) + " lines, tree has " + std::to_string(t->line_count) + ")");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    // The subtree's end stays on the device while the blocks past it, which have
    // nothing to do, cost less than the wait for it.
    const uint32_t *end = (const uint32_t *)t->end_buf.ptr + root;
    uint32_t hi = d->line_count;
    if (query_blocks((uint32_t)root, hi) > kSubtreeEndBlocks) {
        cudaError_t e = ctx->host_words.reserve(4);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->host_words.ptr, end, 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "query_subtree");
        memcpy(&hi, ctx->host_words.ptr, 4);
        end = nullptr;
    }
    return run_query(ctx, d, nullptr, d->line_count, (uint32_t)root, hi, end, kind, depth, max_matches, total, out);
}

extern "C" ol_status ol_query_raw(ol_ctx *ctx, const uint8_t *text, uint64_t len, uint32_t kind, uint32_t depth,
                                  uint32_t max_matches, uint32_t *total, uint32_t *out) {
    if (!ctx || !total || (max_matches && !out) || (len && !text)) return OL_ERR_INVALID_ARG;
    *total = 0;
    if (len > OL_MAX_GPU_INPUT_LEN) return ctx_fail(ctx, OL_ERR_INPUT_TOO_LARGE, "input too large");
    if (len == 0) return OL_OK;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    ol_doc *d = nullptr;
    ol_status s = ol_doc_upload(ctx, text, len, &d);
    if (s == OL_OK) s = ol_query_document(ctx, d, kind, depth, max_matches, total, out);
    ol_doc_free(d);
    return s;
}

extern "C" ol_status ol_query(ol_ctx *ctx, const uint8_t *text, uint64_t len, const uint32_t *offsets, uint64_t n_lines,
                              uint32_t kind, uint32_t depth, uint32_t max_matches, uint32_t *total, uint32_t *out) {
    if (!ctx || !total || (max_matches && !out) || (n_lines && (!offsets || !text))) return OL_ERR_INVALID_ARG;
    *total = 0;
    if (len > OL_MAX_GPU_INPUT_LEN) return ctx_fail(ctx, OL_ERR_INPUT_TOO_LARGE, "input too large");
    if (n_lines == 0) return OL_OK;
    if (len == 0) return ctx_fail(ctx, OL_ERR_INVALID_ARG, "line offsets given for an empty text");
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaSetDevice(ctx->device);
    cudaStream_t st = ctx->stream;
    ol_doc *d = nullptr;
    ol_status s = new_text_doc(ctx, text, len, &d);
    if (s != OL_OK) return s;
    cudaError_t e = ctx->scratch_b.reserve((size_t)n_lines * 4, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->scratch_b.ptr, offsets, (size_t)n_lines * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = ctx->scratch_c.reserve((size_t)n_lines * sizeof(FlatNode), st);
    if (e == cudaSuccess)
        e = launch_classify_lines(d->text, len, (const uint32_t *)ctx->scratch_b.ptr, (uint32_t)n_lines,
                                  (FlatNode *)ctx->scratch_c.ptr, nullptr, st);
    s = ctx_cuda(ctx, e, "query");
    if (s == OL_OK)
        s = run_query(ctx, d, (const FlatNode *)ctx->scratch_c.ptr, (uint32_t)n_lines, 0, (uint32_t)n_lines, nullptr, kind,
                      depth, max_matches, total, out);
    ol_doc_free(d);
    return s;
}
