"""The calls this framework is used for, as cases that can be timed.

Each case is a plain dict; ``case["kind"]`` names the call:

* ``parse_raw``   one-shot parse of host text into offsets and nodes
* ``document``    a text in device memory made a resident document, with its tree
* ``tree``        tree links of a resident document, buffers reused
* ``search``      one pattern in a resident document
* ``multi``       several patterns in a resident document
* ``pipeline``    re-parse, tree and multi-pattern search replayed as one graph
* ``dictionary``  a compiled dictionary over a resident document
* ``batch``       many uneven documents: upload, parse, trees, dictionary
* ``query``       lines of one kind and depth, in the document and in a subtree

``prepare`` makes the inputs and the handles a program keeps, ``run`` is one
pass, ``work`` the bytes that the call cannot do without. All results are whole
numbers. Texts come from ``oneline_b200.datagen``.
"""
from __future__ import annotations

import ctypes
import math
from concurrent.futures import ThreadPoolExecutor
from functools import lru_cache

import numpy as np
import torch

from oneline_b200 import GpuParser, _lib, datagen

KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30
CHUNK = 4 * MIB  # text is generated in chunks of this size, in parallel

# What a text of each sort holds, for the byte counts of work(): bytes per line
# and occurrences of "||||" per byte.
LINE_BYTES = {"corpus": 48.8, "repeat": 17.6, "short-lines": 22.6, "mixed": 83.3, "long-lines": 676.0,
              "prose": 84.2, "nested": 83.9, "deep": 41.5}
PIPES4 = {"corpus": 0.104, "repeat": 0.0, "short-lines": 0.05, "mixed": 0.013, "long-lines": 0.0017,
          "prose": 0.013, "nested": 0.015, "deep": 0.62}
PROFILES = ("repeat", "short-lines", "mixed", "long-lines", "prose", "nested")


# ------------------------------------------------------------------- cases --

def listed() -> list[dict]:
    return [
        # one small note parsed from host memory: the latency of a whole call
        {"name": "parse_raw_4k", "kind": "parse_raw", "text": "mixed", "bytes": 4 * KIB + 3},
        # a text that is already on the GPU becomes a document with its tree:
        # a common file size, and a large file of many short lines
        {"name": "document_1m", "kind": "document", "text": "corpus", "bytes": 1 * MIB},
        {"name": "document_64m", "kind": "document", "text": "short-lines", "bytes": 64 * MIB + 4099},
        # nesting deeper than 32 levels, which the strict build refuses
        {"name": "tree_deep_16m", "kind": "tree", "text": "deep", "bytes": 16 * MIB + 1, "strict": False},
        # one look-up in an open document: the latency of an interactive search
        {"name": "search_1m", "kind": "search", "text": "corpus", "bytes": 1 * MIB, "length": 12,
         "max_matches": 4096},
        # several patterns at once, results to the host, over a middle-sized document
        {"name": "multi_100m", "kind": "multi", "text": "prose", "bytes": 100_000_007, "patterns": 5, "shortest": 3,
         "longest": 64, "max_matches": 65536},
        # a document that is re-read again and again: one graph launch a pass, at
        # a size where launches count and at the benchmark's 1 GiB
        {"name": "pipeline_2m", "kind": "pipeline", "text": "mixed", "bytes": 2 * MIB + 777, "patterns": 3},
        {"name": "pipeline_1g", "kind": "pipeline", "text": "corpus", "bytes": 1 * GIB, "patterns": 8},
        # a few watched terms over one served document, hits to the host
        {"name": "dictionary_256k", "kind": "dictionary", "text": "corpus", "bytes": 256 * KIB + 13, "patterns": 40,
         "device": False, "max_hits": 1 << 18},
        # the benchmark's 10,000-pattern dictionary, hits left on the device
        {"name": "dictionary_256m", "kind": "dictionary", "text": "corpus", "bytes": 256 * MIB, "patterns": 10_000,
         "device": True, "max_hits": 1_200_000_000},
        # a corpus of many uneven documents from page-locked memory, end to end
        {"name": "batch_2500", "kind": "batch", "docs": 2500, "median": 16 * KIB, "patterns": 1000,
         "max_hits": 100_000_000},
        # outline filters over a large document
        {"name": "query_256m", "kind": "query", "text": "corpus", "bytes": 256 * MIB, "line_kind": 4, "depth": 5,
         "max_matches": 1 << 18},
    ]


def _log(rng, lo: int, hi: int) -> int:
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(("parse_raw", "document", "tree", "search", "multi", "pipeline", "dictionary", "batch", "query"))
    text = rng.choice(("corpus", "corpus") + PROFILES)
    if kind == "parse_raw":
        return {"kind": kind, "text": text, "bytes": _log(rng, 256, 16 * MIB)}
    if kind == "document":
        return {"kind": kind, "text": text, "bytes": _log(rng, 4 * KIB, 512 * MIB)}
    if kind == "tree":
        strict = rng.random() < 0.7
        return {"kind": kind, "text": text if strict else "deep", "strict": strict,
                "bytes": _log(rng, 64 * KIB, 512 * MIB if strict else 16 * MIB)}
    if kind == "search":
        return {"kind": kind, "text": text, "bytes": _log(rng, 16 * KIB, 512 * MIB), "length": rng.randint(1, 64),
                "max_matches": _log(rng, 64, 65536)}
    if kind == "multi":
        return {"kind": kind, "text": text, "bytes": _log(rng, 256 * KIB, 512 * MIB), "patterns": rng.randint(2, 12),
                "shortest": rng.randint(1, 8), "longest": _log(rng, 16, 1024), "max_matches": _log(rng, 64, 1 << 18)}
    if kind == "pipeline":
        return {"kind": kind, "text": text, "bytes": _log(rng, 64 * KIB, 1 * GIB), "patterns": rng.randint(1, 8)}
    if kind == "dictionary":
        device = rng.random() < 0.6
        if text == "repeat":  # every sampled pattern would occur once a period, thousands a line
            text = "nested"
        n = _log(rng, 16 * KIB, 64 * MIB if device else 4 * MIB)
        return {"kind": kind, "text": text, "bytes": n, "patterns": _log(rng, 8, 10_000), "device": device,
                "max_hits": 4 * n if device else _log(rng, 1024, 1 << 18)}
    if kind == "batch":
        return {"kind": kind, "docs": _log(rng, 8, 2500), "median": _log(rng, 2 * KIB, 16 * KIB),
                "patterns": _log(rng, 8, 1000), "max_hits": 100_000_000}
    return {"kind": kind, "text": text, "bytes": _log(rng, 64 * KIB, 512 * MIB), "line_kind": rng.randint(0, 7),
            "depth": rng.choice((-1, 0, 1, 2, 3, 5, 8)), "max_matches": _log(rng, 1024, 1 << 18)}


# ------------------------------------------------------------------ inputs --

@lru_cache(maxsize=None)
def _parser() -> GpuParser:
    """The one parser that a program keeps."""
    return GpuParser(0)


def _deep_lines(n: int, seed: int) -> bytes:
    """At least n bytes of lines whose depth walks between 0 and 60 in steps of up to 3."""
    rng = np.random.RandomState(seed)
    count = n // 20 + 16
    walk = np.abs((np.cumsum(rng.randint(-3, 4, count)) + 20) % 120 - 60)
    words = [b"item", b"- entry of a list", b"=[ Section ]", b"@card(title)", b"some plain text here", b""]
    picks = rng.randint(0, len(words), count)
    out, size = [], 0
    for d, w in zip(walk.tolist(), picks.tolist()):
        line = b"|" * d + b" " + words[w] + b"\n"
        out.append(line)
        size += len(line)
        if size >= n:
            break
    return b"".join(out)


def _text(sort: str, n: int, seed: int) -> np.ndarray:
    """n bytes of a sort of text (a pinned buffer, so that uploads of it are direct)."""
    buf = torch.empty(n, dtype=torch.uint8, pin_memory=n >= CHUNK).numpy()

    def fill(at: int) -> None:
        part = buf[at: at + CHUNK]
        s = (seed * 1_000_003 + at // CHUNK) % (1 << 62) + 1
        if sort == "corpus":
            datagen.corpus_into(part, s)
        elif sort == "deep":
            part[:] = np.frombuffer(_deep_lines(part.size, s % (1 << 32)), np.uint8)[: part.size]
        else:
            whole = datagen.generate(datagen.PROFILES[sort], part.size + 1024, s)
            part[:] = np.frombuffer(whole, np.uint8)[: part.size]

    with ThreadPoolExecutor(8) as pool:
        list(pool.map(fill, range(0, n, CHUNK)))
    return buf


def _patterns(text: np.ndarray, seed: int, lengths) -> list[bytes]:
    """One pattern per length: every other one is not in the text."""
    rng = np.random.RandomState(seed % (1 << 32))
    out = []
    for i, m in enumerate(lengths):
        m = min(int(m), text.size)
        if i % 2 == 0:
            at = int(rng.randint(0, text.size - m + 1))
            out.append(text[at: at + m].tobytes())
        else:
            out.append(rng.randint(33, 127, m).astype(np.uint8).tobytes())
    return out


def _batch_offsets(case: dict) -> np.ndarray:
    """Where the documents of a batch begin: log-normal sizes."""
    sizes = datagen.lognormal_sizes(case["docs"], case["docs"], float(case["median"]), 1.5, 256, 64 * MIB)
    offs = np.zeros(case["docs"] + 1, np.uint64)
    offs[1:] = np.cumsum(sizes)
    return offs


def _spread(lo: int, hi: int, n: int) -> list[int]:
    """n lengths from lo to hi, spread over their logarithm."""
    return [int(round(math.exp(math.log(lo) + (math.log(hi) - math.log(lo)) * i / max(n - 1, 1)))) for i in range(n)]


def prepare(case: dict, seed: int) -> dict:
    p, kind = _parser(), case["kind"]
    s = {"case": case, "parser": p}
    if kind == "batch":
        offs = _batch_offsets(case)
        data = torch.empty(int(offs[-1]), dtype=torch.uint8, pin_memory=True).numpy()

        def fill(i: int) -> None:
            datagen.corpus_into(data[int(offs[i]): int(offs[i + 1])], seed * 1_000_003 % (1 << 62) + i + 1)

        with ThreadPoolExecutor(8) as pool:
            list(pool.map(fill, range(case["docs"])))
        s["data"], s["offs"] = data, offs
        s["set"] = p.compile_patterns(None, datagen.patterns_dictionary(data, seed + 2, case["patterns"]))
        s["hits"] = torch.zeros((case["max_hits"], 2), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return s

    text = _text(case["text"], case["bytes"], seed)
    if kind == "parse_raw":
        s["text"] = text.tobytes()
        return s
    if kind == "document":
        s["text"] = torch.from_numpy(text).cuda()
        s["tree"] = None
        torch.cuda.synchronize()
        return s
    s["doc"] = doc = p.upload(text)
    if kind == "tree":
        s["tree"] = p.build_tree(doc, strict_depth=case["strict"])
    elif kind == "search":
        s["pattern"] = _patterns(text, seed, [case["length"]])[0]
    elif kind == "multi":
        s["patterns"] = _patterns(text, seed, _spread(case["shortest"], case["longest"], case["patterns"]))
    elif kind == "pipeline":
        pats = datagen.patterns_eight(text, seed + 1)[: case["patterns"]]
        s["tree"] = p.build_tree(doc)
        # even ones come from the text, and a short one may be a run of "|"; odd ones are random bytes
        rooms = [4096 if i % 2 else case["bytes"] // (6 if i == 0 else 12) for i in range(len(pats))]
        s["outs"] = [torch.zeros(r, dtype=torch.int32, device="cuda") for r in rooms]
        s["totals"] = torch.zeros(len(pats), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        s["pipeline"] = p.capture_pipeline(doc, s["tree"], pats, rooms, s["totals"].data_ptr(),
                                           [o.data_ptr() for o in s["outs"]])
    elif kind == "dictionary":
        s["set"] = p.compile_patterns(doc, datagen.patterns_dictionary(text, seed + 2, case["patterns"]),
                                      max_patterns=None)
        if case["device"]:
            s["hits"] = torch.zeros((case["max_hits"], 2), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
    elif kind == "query":
        s["tree"] = p.build_tree(doc)
        # the root with the largest subtree among the first lines
        ends = p.download_links(s["tree"]).subtree_end[:4096].astype(np.int64)
        s["root"] = int(np.argmax(ends - np.arange(ends.size)))
    return s


# --------------------------------------------------------------------- run --

class Results(dict):
    """The results of a pass where a program has them: in the arrays that the
    call returned, or in device memory, where it goes on working with them. Each
    is read out when it is looked at, into an array of the case's fixed room
    (zeros after the values)."""

    def __getitem__(self, name):
        return super().__getitem__(name)()


def _line_room(case: dict) -> int:
    n = int(_batch_offsets(case)[-1]) if case["kind"] == "batch" else case["bytes"]
    return int(1.5 * n / LINE_BYTES[case.get("text", "corpus")]) + 1024 + case.get("docs", 0)


def _padded(values: np.ndarray, room: int) -> np.ndarray:
    if values.shape[0] > room:
        raise ValueError(f"{values.shape[0]} values for a room of {room}")
    out = np.zeros((room,) + values.shape[1:], values.dtype)
    out[: values.shape[0]] = values
    return out


def _depths(doc) -> np.ndarray:
    """The depth of every line (clamped to 255), from the document's device array."""
    view, n = ctypes.c_void_p(), doc.line_count()
    _lib.check(_lib.load().ol_doc_device_views(doc.handle, None, None, None, ctypes.byref(view)))

    class Array:
        __cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (view.value, False), "version": 3}

    return torch.as_tensor(Array(), device="cuda").cpu().numpy()


def _document_results(case: dict, doc) -> dict:
    room = _line_room(case)
    return {"offsets": lambda: _padded(doc.read_offsets(), room), "kinds": lambda: _padded(doc.read_kinds(), room),
            "depths": lambda: _padded(_depths(doc), room), "lines": doc.line_count}


def _tree_results(case: dict, parser, tree) -> dict:
    room = _line_room(case)
    return {k: (lambda k=k: _padded(parser.download_tree(tree)[k], room))
            for k in ("parent", "subtree_end", "first_child", "next_sibling")}


def _batch_results(case: dict, parser, batch) -> dict:
    room = _line_room(case)

    def whole(name):
        return _padded(np.concatenate([parser.read_batch_doc(batch, i)[name] for i in range(len(batch))]), room)

    return {k: (lambda k=k: whole(k))
            for k in ("offsets", "kinds", "parent", "subtree_end", "first_child", "next_sibling")}


def run(state: dict):
    p, case = state["parser"], state["case"]
    kind, doc = case["kind"], state.get("doc")
    if kind == "parse_raw":
        tree = p.parse_raw(state["text"])
        return Results(offsets=lambda: _padded(tree.line_offsets, _line_room(case)), lines=lambda: len(tree.nodes),
                       nodes=lambda: _padded(tree.nodes.view(np.uint32).reshape(-1, 4), _line_room(case)))
    if kind == "document":
        text = state["text"]
        old = state.pop("doc", None)
        if old is not None:
            old.free()
        state["doc"] = doc = p.upload_device(text.data_ptr(), text.numel())
        state["tree"] = tree = p.build_tree_reusing(doc, state["tree"])
        return Results(_document_results(case, doc) | _tree_results(case, p, tree))
    if kind == "tree":
        state["tree"] = tree = p.build_tree_reusing(doc, state["tree"], strict_depth=case["strict"])
        return Results(_tree_results(case, p, tree))
    if kind == "search":
        r = p.search_document(doc, state["pattern"], case["max_matches"])
        return Results(total=lambda: r.total_matches, offsets=lambda: _padded(r.offsets, case["max_matches"]))
    if kind == "multi":
        rs = p.search_document_multi(doc, state["patterns"], case["max_matches"])
        return Results(totals=lambda: [r.total_matches for r in rs],
                       offsets=lambda: [_padded(r.offsets, case["max_matches"]) for r in rs])
    if kind == "pipeline":
        state["pipeline"].launch()
        return Results(_document_results(case, doc) | _tree_results(case, p, state["tree"]),
                       totals=lambda: state["totals"], hits=lambda: state["outs"])
    if kind == "dictionary" and case["device"]:
        counts, total = p.search_many_device(doc, state["set"], state["hits"].data_ptr(), case["max_hits"])
        return {"counts": counts, "total": total, "hits": state["hits"]}
    if kind == "dictionary":
        r = p.search_many(doc, state["set"], case["max_hits"])
        return Results(counts=lambda: r.counts, total=lambda: r.total_hits,
                       hits=lambda: _padded(r.hits.view(np.uint32).reshape(-1, 2), case["max_hits"]))
    if kind == "batch":
        old = state.pop("batch", None)
        if old is not None:
            old.free()
        state["batch"] = batch = p.upload_batch((state["data"], state["offs"]))
        p.build_batch_trees(batch)
        counts, total = p.batch_search_many(batch, state["set"], state["hits"].data_ptr(), case["max_hits"])
        return Results(_batch_results(case, p, batch), counts=lambda: counts, total=lambda: total,
                       hits=lambda: state["hits"])
    room, depth = case["max_matches"], None if case["depth"] < 0 else case["depth"]
    whole = p.query_document(doc, case["line_kind"], depth, room)
    part = p.query_subtree(doc, state["tree"], state["root"], case["line_kind"], None, room)
    return Results(total=lambda: whole.total_matches, lines=lambda: _padded(whole.indices, room),
                   subtree_total=lambda: part.total_matches, subtree_lines=lambda: _padded(part.indices, room))


# -------------------------------------------------------------------- work --

def work(case: dict) -> dict:
    """Bytes of one pass: each input read once, each output written once (line
    and hit counts from what such texts hold)."""
    kind = case["kind"]
    if kind == "batch":
        n = int(_batch_offsets(case)[-1])
        hits = min(0.00036 * case["patterns"] * n, case["max_hits"])
        return {"bytes": 2 * n + 22 * n / LINE_BYTES["corpus"] + 8 * hits, "flops": 0}
    n, lines = case["bytes"], case["bytes"] / LINE_BYTES[case["text"]]
    if kind == "parse_raw":
        return {"bytes": n + 20 * lines, "flops": 0}
    if kind == "document":  # the text copied, then offsets, kinds, depths and four links a line
        return {"bytes": 2 * n + 22 * lines, "flops": 0}
    if kind == "tree":
        return {"bytes": 18 * lines, "flops": 0}
    if kind == "search":
        return {"bytes": n, "flops": 0}
    if kind == "multi":
        return {"bytes": n * -(-case["patterns"] // 8), "flops": 0}
    if kind == "pipeline":
        return {"bytes": n + 22 * lines + 4 * PIPES4[case["text"]] * n, "flops": 0}
    if kind == "dictionary":
        hits = 0.00036 * case["patterns"] * PIPES4[case["text"]] / PIPES4["corpus"] * n
        return {"bytes": n + 8 * min(hits, case["max_hits"]), "flops": 0}
    return {"bytes": 3 * lines, "flops": 0}  # kinds and depths of the document, kinds of the subtree
