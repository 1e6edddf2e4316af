"""Performance cases: the calls a user of the engine makes, over the range of
sizes they are made with.

A case is one pass through a public entry point of the Python package (the
thin mirror of the C ABI): an index build into the caller's buffers, a query
over a resident index, a build with its queries, the compaction of a result
array, a replay of a captured batch, a host-to-host query, a burst of server
requests.  Inputs are the two seeded record families of the package's data
generator (NDJSON posts, one top-level array of products); inputs above 32
MiB repeat whole lines of a 32 MiB base on the device.
"""
from __future__ import annotations

import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
KIB, MIB = 1 << 10, 1 << 20
BASE_BYTES = 32 * MIB
RECORD_BYTES = 2400  # per record (line) of the inputs, a little above what the generator makes


def _load(name: str, path: Path):
    if name in sys.modules:
        return sys.modules[name]
    spec = importlib.util.spec_from_file_location(
        name, path / "__init__.py", submodule_search_locations=[str(path)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


# the package directory name is not an identifier
pkg = _load("gpjson_b200", ROOT / "15418-project_b200")
datagen = _load("gpjson_b200.datagen", ROOT / "15418-project_b200" / "datagen")

# (query, wildcard limit, bitmap level of the records): the benchmark's
# queries and the language extensions.
LANG = ("$.user.lang", 0, 0)
TAGS = ("$.entities.hashtags[*].text", 8, 0)
COUNTRY = ("$.place.country_code", 0, 0)
RETWEET = ("$.retweeted_status.user.id", 0, 0)
CATEGORY = ("$.categoryPath[1:3].id", 0, 1)  # "$[*].categoryPath[1:3].id"
LAST_TAGS = ("$.entities.hashtags[-2:].text", 0, 0)
FOLLOWED = ("$.user[?(@.followers_count >= 10000)].screen_name", 0, 0)
ANY_ID = ("$..id", 8, 0)
QUERIES = {
    "lang": [LANG],
    "tags": [TAGS],
    "country": [COUNTRY],
    "retweet": [RETWEET],
    "category": [CATEGORY],
    "last_tags": [LAST_TAGS],
    "followed": [FOLLOWED],
    "any_id": [ANY_ID],
    "posts": [LANG, TAGS, COUNTRY, RETWEET],
    "filters": [FOLLOWED, LAST_TAGS],
    "descend": [ANY_ID, FOLLOWED],
}

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        torch.cuda.init()
        _ctx = pkg.Context(torch.cuda.current_device())
    return _ctx


_servers = {}


def _server(budget: int):
    if budget not in _servers:
        _servers[budget] = pkg.Server(torch.cuda.current_device(), num_slots=32,
                                      hbm_budget_bytes=budget, host_result_bytes=64 * MIB,
                                      cache_levels=4)
    return _servers[budget]


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _compiled(name: str):
    return [(pkg.compile(q, wildcard_limit=k), base) for q, k, base in QUERIES[name]]


def _levels(name: str) -> int:
    return max(c.max_depth + base for c, base in _compiled(name))


# ---- inputs ------------------------------------------------------------------


FIRST_STRING = {"posts": b'"created_at":"', "posts_deep": b'"created_at":"', "products": b'"name":"'}


def _base(source: str, seed: int, size: int):
    """Host lines of a source and where each ends: posts end every line with a
    newline; products are the array's elements, each followed by ",\n"."""
    if source == "products":
        data = datagen.products(seed, size)
        host = np.empty(data.size - 3, np.uint8)  # "[\n" body "\n]\n" -> body ",\n"
        host[:-2] = data[2:-3]
        host[-2:] = (ord(","), ord("\n"))
    else:
        host = datagen.tweets(seed, size, deep=source == "posts_deep")
    return host, np.flatnonzero(host == 10) + 1


def _piece(source: str, base, first: int, size: int) -> np.ndarray:
    """Exactly `size` bytes of whole lines of a base, from about line `first`
    on.  The number of lines follows from `size` alone; what they lack to it
    lengthens the first string of each of them alike."""
    host, lines = base
    count = int((size - 2.0 * 1200.0 * math.sqrt(size / RECORD_BYTES)) / RECORD_BYTES)
    count = min(max(count, 1), lines.size)
    starts = np.concatenate([[0], lines[:-1]])
    spans = lines[count - 1:] - starts[: lines.size - count + 1]
    fits = np.flatnonzero(spans <= size)
    if not fits.size:
        raise ValueError("no %d lines of the base fit in %d bytes" % (count, size))
    k = int(fits[np.searchsorted(fits, first % spans.size) % fits.size])
    start = int(starts[k])
    part = host[start:start + int(spans[k])]
    text, at, pos = part.tobytes(), np.empty(count, np.int64), 0
    for i in range(count):
        at[i] = text.index(FIRST_STRING[source], pos) + len(FIRST_STRING[source])
        pos = int(lines[k + i]) - start
    missing = size - part.size
    extra = np.full(count, missing // count)
    extra[: missing % count] += 1
    return np.insert(part, np.repeat(at, extra), np.uint8(ord("a")))


def _records(source: str, seed: int, size: int) -> torch.Tensor:
    """Exactly `size` device bytes of whole lines."""
    base = _base(source, seed, min(size + 128 * KIB, BASE_BYTES))
    if size <= BASE_BYTES:
        return torch.from_numpy(_piece(source, base, 0, size)).cuda()
    full = torch.from_numpy(_piece(source, base, 0, BASE_BYTES)).cuda()
    half = torch.from_numpy(_piece(source, base, 9, BASE_BYTES // 2)).cuda()
    whole, rest = divmod(size - half.numel(), BASE_BYTES)
    parts = [half, full.repeat(whole)]
    if rest < 16 * KIB:  # too short for a piece of its own
        parts, rest = parts[1:], rest + half.numel()
    return torch.cat([*parts, torch.from_numpy(_piece(source, base, 5, rest)).cuda()])


def _file_into(dst: torch.Tensor, source: str, parts) -> None:
    """Fills `dst` with one file of the parts' records; a file of products is
    three bytes longer than its records (the array's brackets)."""
    pos = 2 if source == "products" else 0
    for part in parts:
        dst[pos:pos + part.numel()] = part
        pos += part.numel()
    if source == "products":  # the last element's ",\n" becomes "\n]\n"
        dst[:2] = torch.tensor(list(b"[\n"), dtype=torch.uint8, device=dst.device)
        dst[-3:] = torch.tensor(list(b"\n]\n"), dtype=torch.uint8, device=dst.device)


def _brackets(source: str) -> int:
    return 3 if source == "products" else 0


def _partition(source: str, seed: int, size: int, skew: int = 0) -> torch.Tensor:
    """One partition of `size` bytes on the device, `skew` bytes into its
    allocation."""
    data = torch.empty(size + skew, dtype=torch.uint8, device="cuda")[skew:]
    _file_into(data, source, [_records(source, seed, size - _brackets(source))])
    return data


def _index_buffers(data: torch.Tensor, levels: int, verify: bool):
    n = data.numel()
    words = (n + 63) // 64
    lines = 1 + sum(int((part == 10).sum()) for part in data.split(1 << 30))
    new = lambda count: torch.empty(count, dtype=torch.int64, device="cuda")  # noqa: E731
    out = {"string": new(words), "leveled": new(words * levels), "newline": new(lines),
           "summary": new(4)}
    if verify:
        out["escape"], out["quote"] = new(words), new(words)
    ix = pkg.Index()
    ix.d_string = out["string"].data_ptr()
    ix.d_leveled = out["leveled"].data_ptr()
    ix.d_newline = out["newline"].data_ptr()
    ix.newline_capacity = lines
    if verify:
        ix.d_escape, ix.d_quote = out["escape"].data_ptr(), out["quote"].data_ptr()
    return ix, out, lines


def _build(data: torch.Tensor, levels: int, ix, out, verify: bool) -> None:
    _context().build_index_async(data.data_ptr(), data.numel(), levels, ix,
                                 out["summary"].data_ptr(),
                                 flags=pkg.GPJ_INDEX_EMIT_ESCAPE_QUOTE if verify else 0,
                                 stream=_stream())


# ---- one kind of case each: prepare(case, seed) -> state, run(state) -> outputs ----


def _prepare_index(case, seed):
    data = _partition(case["source"], seed, case["bytes"], case.get("skew", 0))
    ix, out, _ = _index_buffers(data, case["levels"], case.get("verify", False))
    return {"data": data, "ix": ix, "out": out, "levels": case["levels"],
            "verify": case.get("verify", False)}


def _run_index(s):
    _build(s["data"], s["levels"], s["ix"], s["out"], s["verify"])
    return s["out"]


def _prepare_query(case, seed):
    """A resident index, as a program keeps it between queries."""
    (compiled, base), = _compiled(case["queries"])
    levels = compiled.max_depth + base
    data = _partition(case["source"], seed, case["bytes"])
    ix, out, lines = _index_buffers(data, levels, False)
    _build(data, levels, ix, out, False)
    ix.num_lines = lines
    res = torch.empty((lines, compiled.num_result_slots, 2), device="cuda",
                      dtype=torch.int64 if case.get("wide") else torch.int32)
    return {"data": data, "ix": ix, "out": out, "compiled": compiled, "base": base, "res": res,
            "wide": bool(case.get("wide"))}


def _run_query(s):
    _context().query(s["ix"], s["compiled"], s["res"].data_ptr(), stream=_stream(),
                     wide=s["wide"], base_level=s["base"])
    return s["res"]


def _prepare_engine(case, seed):
    return {"data": _partition(case["source"], seed, case["bytes"]),
            "levels": _levels(case["queries"]), "compiled": _compiled(case["queries"])}


def _run_engine(s):
    """Library-owned index, every query over it, the status, the release."""
    ctx, stream = _context(), _stream()
    ix = ctx.build_index(s["data"].data_ptr(), s["data"].numel(), s["levels"], stream=stream)
    outs = []
    for compiled, base in s["compiled"]:
        res = torch.empty((ix.num_lines, compiled.num_result_slots, 2), dtype=torch.int32,
                          device="cuda")
        ctx.query(ix, compiled, res.data_ptr(), stream=stream, base_level=base)
        outs.append(res)
    status = ctx.query_status(stream)
    lines = int(ix.num_lines)
    ctx.free_index(ix)
    return {"results": outs, "lines": lines, "status": status}


def _prepare_compact(case, seed):
    """A result array in device memory and buffers for every pair of it."""
    s = _prepare_query({**case, "wide": False}, seed)
    s["res"] = _run_query(s)
    pairs = s["res"].numel() // 2
    s["counts"] = torch.zeros(3, dtype=torch.int64, device="cuda")
    s["matches"] = torch.zeros((pairs, 5), dtype=torch.int64, device="cuda")  # gpj_match rows
    s["arena"] = torch.zeros(pairs * 32, dtype=torch.uint8, device="cuda")
    return s


def _run_compact(s):
    _context().compact(s["res"].data_ptr(), s["res"].shape[0], s["compiled"].num_result_slots,
                       s["data"].data_ptr(), s["data"].numel(), 0, s["matches"].data_ptr(),
                       s["matches"].shape[0], s["arena"].data_ptr(), s["arena"].numel(),
                       s["counts"].data_ptr(), stream=_stream())
    return {"matches": s["matches"], "arena": s["arena"], "counts": s["counts"]}


class _DeviceArray:
    """Library-owned device memory as a tensor source that keeps its owner."""

    def __init__(self, owner, ptr: int, count: int, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr,
                                         "data": (ptr, False), "version": 3}


def _file_sizes(case) -> np.ndarray:
    """Log-normal file sizes from 4 KiB to 64 MiB that sum to about the case's
    bytes."""
    x = np.random.default_rng(case["files"]).lognormal(0.0, 2.0, size=case["files"])
    for _ in range(8):
        x = np.clip(x * (case["bytes"] / x.sum()), 4 * KIB, 64 * MIB)
    return x.astype(np.int64)


def _prepare_batch(case, seed):
    """Half NDJSON posts, half product arrays, packed at 128-byte offsets; the
    plan is captured once and replayed."""
    rng = np.random.default_rng(seed)
    page = 256 * KIB
    sources, bases, pages = ("posts", "products"), [], []
    for i, source in enumerate(sources):
        base = _base(source, seed + i, 8 * MIB)
        bases.append(base)
        pages.append([torch.from_numpy(_piece(source, base, 111 * j, page)).cuda()
                      for j in range(24)])
    table, pos = [], 0
    for f, size in enumerate(int(s) for s in _file_sizes(case)):
        table.append((pos, size, f % 2))
        pos += (size + 127) // 128 * 128
    buf = torch.zeros(pos, dtype=torch.uint8, device="cuda")
    for offset, size, kind in table:
        source = sources[kind]
        whole, rest = divmod(size - _brackets(source), page)
        if whole and rest < 16 * KIB:
            whole, rest = whole - 1, rest + page
        parts = [pages[kind][int(j)] for j in rng.integers(24, size=whole)]
        first = int(rng.integers(bases[kind][1].size))
        parts.append(torch.from_numpy(_piece(source, bases[kind], first, rest)).cuda())
        _file_into(buf[offset:offset + size], source, parts)
    queries = [(c, b, c.max_depth + b) for c, b in _compiled("lang") + _compiled("category")]
    batch = pkg.Batch(buf.data_ptr(), buf.numel(), table, queries,
                      flags=pkg.GPJ_BATCH_AUTOTUNE if case["tuned"] else 0, stream=_stream())
    batch.input = buf
    v = batch.view()

    def view(ptr, count, typestr):
        return torch.as_tensor(_DeviceArray(batch, ptr, count, typestr), device="cuda")

    out = {"results": view(v.d_results, v.result_ints, "<i4"),
           "files": view(v.d_file_info, v.num_files * pkg.FILE_INFO_WORDS, "<i8"),
           "string": view(v.d_string, v.string_words, "<i8"),
           "leveled": view(v.d_leveled, v.leveled_words, "<i8"),
           "newline": view(v.d_newline, v.newline_slots, "<i8")}
    return {"batch": batch, "out": out}


def _run_batch(s):
    s["batch"].run(_stream())
    return s["out"]


def _prepare_host(case, seed):
    """Pinned input and result buffers, the whole call from host to host."""
    data = _partition(case["source"], seed, case["bytes"]).cpu().pin_memory()
    lines = int((data == 10).sum()) + 1
    compiled = _compiled(case["queries"])
    outs = [torch.empty((lines, c.num_result_slots, 2), dtype=torch.int32).pin_memory()
            for c, _ in compiled]
    return {"data": data, "levels": _levels(case["queries"]), "compiled": [c for c, _ in compiled],
            "bases": [b for _, b in compiled], "outs": outs}


def _run_host(s):
    lines = _context().query_host(s["data"].data_ptr(), s["data"].numel(), s["levels"],
                                  s["compiled"], [o.data_ptr() for o in s["outs"]],
                                  [o.numel() for o in s["outs"]], stream=_stream(),
                                  base_levels=s["bases"])
    return {"results": s["outs"], "lines": lines}


def _prepare_server(case, seed):
    """A burst of requests, 30% for files whose index the server may keep."""
    rng = np.random.default_rng(case["requests"])
    base = _base("posts_deep", seed, 9 * MIB)
    comp = [(c, b, c.max_depth + b) for c, b in _compiled("posts")]
    sizes = np.clip(rng.lognormal(math.log(case["bytes"]), 1.0, case["requests"]), 16 * KIB, 8 * MIB)
    items = []
    for r, size in enumerate(sizes):
        picks = sorted(int(q) for q in rng.choice(4, int(rng.integers(1, 4)), replace=False))
        key = (seed * 4096 + r + 1) if rng.random() < 0.3 else 0
        data = torch.from_numpy(_piece("posts_deep", base, 97 * r, int(size))).pin_memory()
        items.append((data.numpy(), [comp[q] for q in picks], key, 0))
    return {"items": items, "server": _server(case["budget"])}


def _run_server(s):
    srv = s["server"]
    ids = srv.submit_prepared(srv.prepare(s["items"]))
    left = set(ids)
    while left:
        left.difference_update(srv.poll(timeout_us=1_000_000))
    done = [srv.response(rid) for rid in ids]
    if any(r.status for r in done):
        raise RuntimeError(next(r.message for r in done if r.status))
    return [np.concatenate([x.reshape(-1) for x in r.results]) for r in done]


_KINDS = {
    "index": (_prepare_index, _run_index),
    "query": (_prepare_query, _run_query),
    "engine": (_prepare_engine, _run_engine),
    "compact": (_prepare_compact, _run_compact),
    "batch": (_prepare_batch, _run_batch),
    "host": (_prepare_host, _run_host),
    "server": (_prepare_server, _run_server),
}


def listed():
    return [
        # the index of one small request's file, queued into buffers the
        # caller owns: launch count and latency
        {"name": "index_request", "kind": "index", "source": "posts", "bytes": 100_000,
         "levels": 4},
        # one uploaded partition of ordinary size, with the escape and quote
        # bitmaps that a consumer of every reference bitmap asks for
        {"name": "index_partition", "kind": "index", "source": "posts_deep",
         "bytes": 24 * MIB + 777, "levels": 4, "verify": True},
        # the benchmark's 1 GiB product array
        {"name": "index_array", "kind": "index", "source": "products", "bytes": 1 << 30,
         "levels": 4},
        # the benchmark's 64 MiB posts: one key path over a resident index
        {"name": "query_key", "kind": "query", "source": "posts", "bytes": 64 * MIB,
         "queries": "lang"},
        # array elements as records, a slice with two slots
        {"name": "query_array", "kind": "query", "source": "products", "bytes": 500_000_000,
         "queries": "category"},
        # eight slots per record with 64-bit offsets, as partitions of 2 GiB
        # and more need them
        {"name": "query_slots", "kind": "query", "source": "posts_deep", "bytes": 700 * MIB,
         "queries": "tags", "wide": True},
        # descend and filter queries, whose index holds every level they reach:
        # build, queries, status, release
        {"name": "engine_descend", "kind": "engine", "source": "posts_deep", "bytes": 96 * MIB,
         "queries": "descend"},
        # the executor's result compaction, matches and their text
        {"name": "compact_tags", "kind": "compact", "source": "posts_deep", "bytes": 256 * MIB,
         "queries": "tags"},
        # many files in one captured chain, as the benchmark packs them
        {"name": "batch_many", "kind": "batch", "files": 2000, "bytes": 1500 * MIB,
         "tuned": True},
        # a small batch of small files
        {"name": "batch_small", "kind": "batch", "files": 60, "bytes": 4 * MIB, "tuned": False},
        # host to host: one file of a driver run with the four benchmark queries
        {"name": "host_file", "kind": "host", "source": "posts_deep", "bytes": 6 * MIB + 4321,
         "queries": "posts"},
        # a burst at the server, log-normal files around 128 KiB
        {"name": "server_burst", "kind": "server", "requests": 40, "bytes": 128 * KIB,
         "budget": 1 << 30},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["index", "index", "query", "query", "engine", "compact", "batch", "batch",
                       "host", "server"])
    if kind == "index":
        case = {"kind": kind, "source": rng.choice(["posts", "posts_deep", "products"]),
                "bytes": _log(rng, 20 * KIB, 700 * MIB),
                "levels": rng.choice([2, 3, 4, 4, 5, 6, 8, 12, 15])}
        if rng.random() < 0.2:
            case["verify"] = True
        if rng.random() < 0.1:
            case["skew"] = rng.randint(1, 15)
        return case
    if kind in ("query", "compact"):
        q = rng.choice(["lang", "tags", "country", "retweet", "category", "last_tags", "followed",
                        "any_id"])
        case = {"kind": kind, "bytes": _log(rng, 64 * KIB, 400 * MIB), "queries": q,
                "source": "products" if q == "category" else rng.choice(["posts", "posts_deep"])}
        if kind == "query" and rng.random() < 0.25:
            case["wide"] = True
        return case
    if kind == "engine":
        q = rng.choice(["lang", "posts", "filters", "descend", "category"])
        return {"kind": kind, "bytes": _log(rng, 64 * KIB, 200 * MIB), "queries": q,
                "source": "products" if q == "category" else rng.choice(["posts", "posts_deep"])}
    if kind == "batch":
        files = _log(rng, 8, 3000)
        return {"kind": kind, "files": files, "tuned": False,
                "bytes": min(700 * MIB, int(files * _log(rng, 16 * KIB, 600 * KIB)))}
    if kind == "host":
        q = rng.choice(["lang", "posts", "category"])
        return {"kind": kind, "bytes": _log(rng, 64 * KIB, 80 * MIB), "queries": q,
                "source": "products" if q == "category" else "posts_deep"}
    return {"kind": kind, "requests": rng.randint(4, 60), "bytes": _log(rng, 32 * KIB, 512 * KIB),
            "budget": 1 << 30}


def prepare(case, seed):
    return {"kind": case["kind"], "state": _KINDS[case["kind"]][0](case, seed)}


def run(state):
    return _KINDS[state["kind"]][1](state["state"])


def _index_bytes(n: int, levels: int, verify: bool = False) -> int:
    """Input read once, S, the levels (and E, Q) and the newline index written."""
    return n + n // 8 * (1 + levels + (2 if verify else 0)) + 8 * (n // RECORD_BYTES)


def _query_bytes(n: int, name: str, width: int = 4) -> int:
    """The newline index and one level's bitmap words read, the results written."""
    total = 0
    for compiled, _ in _compiled(name):
        total += n // 8 + (n // RECORD_BYTES) * (8 + 2 * width * compiled.num_result_slots)
    return total


def work(case):
    n = case["bytes"]
    kind = case["kind"]
    if kind == "index":
        b = _index_bytes(n, case["levels"], case.get("verify", False))
    elif kind == "query":
        b = _query_bytes(n, case["queries"], 8 if case.get("wide") else 4)
    elif kind == "engine":
        b = _index_bytes(n, _levels(case["queries"])) + _query_bytes(n, case["queries"])
    elif kind == "compact":
        # every pair read; about half the slots match, with some 10 bytes of text
        items = (n // RECORD_BYTES) * _compiled(case["queries"])[0][0].num_result_slots
        b = items * 8 + items // 2 * (40 + 2 * 10)
    elif kind == "batch":
        b = _index_bytes(n, 4) + _query_bytes(n, "lang")
    elif kind == "host":
        b = n + _index_bytes(n, _levels(case["queries"])) + 2 * _query_bytes(n, case["queries"])
    else:
        total = n * case["requests"]
        b = total + _index_bytes(total, 4) + 2 * _query_bytes(total, "lang")
    return {"bytes": b, "flops": 0}


def exact(case, seed):
    """Index builds up to 32 MiB, in plain numpy; elsewhere every output is a
    whole number that a general JSON parser would take minutes to restate."""
    if case["kind"] != "index" or case["bytes"] > 32 * MIB:
        return None
    data = _partition(case["source"], seed, case["bytes"], case.get("skew", 0)).cpu().numpy()
    n = data.size
    words = (n + 63) // 64
    bs = data == ord("\\")
    # a byte is escaped when the backslash run before it has odd length (runs
    # of the inputs are far shorter than a 64-byte word, but count inside it)
    escaped = np.zeros(n + 1, bool)
    for i in np.flatnonzero(bs):
        escaped[i + 1] = not escaped[i]
    escaped = escaped[:n]
    quote = (data == ord('"')) & ~escaped
    inside = np.cumsum(quote, dtype=np.int64) % 2 == 1
    opens = ((data == ord("{")) | (data == ord("["))) & ~inside
    closes = ((data == ord("}")) | (data == ord("]"))) & ~inside
    depth = np.cumsum(opens.astype(np.int32) - closes, dtype=np.int32) - 1
    level = np.where(closes, depth + 1, depth)
    marks = (opens | closes | (((data == ord(":")) | (data == ord(","))) & ~inside))

    def pack(bits):
        padded = np.zeros(words * 64, bool)
        padded[:n] = bits
        return np.packbits(padded, bitorder="little").view("<i8")

    newline = np.concatenate([[0], np.flatnonzero(data == 10)]).astype(np.int64)
    string = pack(inside)
    if n % 64:  # the state after the last byte fills the word's tail
        tail = np.uint64(~((1 << (n % 64)) - 1) & (2**64 - 1)) if inside[-1] else np.uint64(0)
        string[-1] = (string[-1].view(np.uint64) | tail).view(np.int64)
    out = {"string": string,
           "leveled": np.concatenate([pack(marks & (level == l)) for l in range(case["levels"])]),
           "newline": newline,
           "summary": np.array([newline.size, int(inside[-1]), int(depth[-1]), 0], np.int64)}
    if case.get("verify"):
        out["escape"], out["quote"] = pack(escaped), pack(quote)
    return out
