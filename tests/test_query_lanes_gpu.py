"""The query kernel runs a record with 32, 16, 8 or 1 lanes, by the number of
records: each split against the oracle, bit for bit, on records that reach the
edges of its searches (dense and long records, keys across words, escaped
quotes, blanks, broken nesting, garbage), at both ends of each range."""
import random

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

QUERIES = [
    ("$.k", 0), ("$.ab", 0), ("$.key.ab", 0), ("$.long_key_name.x", 0), ("$.arr[2]", 0),
    ("$.arr[1:4].k", 0), ("$.arr[-1]", 0), ("$.arr[-2:]", 0), ('$.key[?(@.ab == "v")].k', 0),
    ("$.key[?(@.n >= 10)].k", 0), ("$.arr[*]", 4), ("$.arr[1:-1].k", 4), ("$..k", 3),
    ("$.%s" % ("q" * 130), 0),
]


def _value(rng, depth):
    r = rng.random()
    if depth > 2 or r < 0.45:
        return rng.choice(['"v"', "1", "10.5", "null", '"x\\"k\\":1"', '"\\\\"', '"%s"' % ("y" * 90),
                           '"{[,:]}"', "-3e2"])
    pad = rng.choice(["", "", " ", "   "])
    if r < 0.7:
        return "[" + ("," + pad).join(_value(rng, depth + 1) for _ in range(rng.randint(0, 5))) + "]"
    return _object(rng, depth + 1)


def _object(rng, depth=0):
    keys = rng.sample(["k", "ab", "key", "long_key_name", "arr", "n", "x", "abc", "q" * 130, "zz"],
                      rng.randint(0, 7))
    pad = rng.choice(["", "", "", " "])
    items = ['"%s"%s:%s%s' % (k, pad, pad, str(rng.randint(0, 30)) if k == "n" else
                              _value(rng, depth)) for k in keys]
    return "{" + ",".join(items) + "}"


def _line(rng):
    r = rng.random()
    if r < 0.8:
        return _object(rng)
    if r < 0.84:  # more structural characters than one round looks at
        return '{%s,"k":7,"arr":[%s]}' % (",".join('"a%d":1' % i for i in range(90)),
                                          "," * rng.randint(0, 200))
    if r < 0.86:
        return '{"abc":"%s","ab":%s}' % ("t" * rng.randint(50, 2500), _value(rng, 0))
    if r < 0.88:
        return "{" + ":" * rng.randint(1, 130) + "}"
    return "".join(rng.choices('{}[]:,"\\ kab', weights=[6, 6, 3, 3, 5, 5, 8, 1, 3, 8, 4, 4],
                               k=rng.randint(0, 120)))


def _lines(seed, count):
    rng = random.Random(seed)
    pool = [_line(rng) for _ in range(1500)]
    return "\n".join(rng.choice(pool) for _ in range(count)).encode()


def _counts():
    """(lanes, number of records) at both ends of each range."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() \
        else 148
    top = {g: sms * 1024 // g for g in (32, 16, 8)}
    return [(32, 40), (32, top[32]), (16, top[32] + 1), (16, top[16]), (8, top[16] + 1),
            (8, top[8]), (1, top[8] + 1)]


@pytest.mark.parametrize("end", range(7))
@pytest.mark.parametrize("skew", [0, 5], ids=["aligned", "unaligned"])
def test_every_split_matches_oracle(cuda_ctx, gpj, end, skew):
    lanes, count = _counts()[end]
    data = np.frombuffer(_lines(end, count), np.uint8)
    buf = torch.zeros(data.size + 64, dtype=torch.uint8, device="cuda")
    buf[skew:skew + data.size] = torch.from_numpy(data.copy())
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in QUERIES]
    levels = min(6, max(c.max_depth for c in comp))
    want_ix = oracle.OracleIndex(data, levels)
    ix = cuda_ctx.build_index(buf.data_ptr() + skew, data.size, levels)
    try:
        assert ix.num_lines == count
        for c in comp:
            for wide in (False, True):
                out = torch.full((count, c.num_result_slots, 2), -7, device="cuda",
                                 dtype=torch.int64 if wide else torch.int32)
                cuda_ctx.query(ix, c, out.data_ptr(), wide=wide)
                torch.cuda.synchronize()
                np.testing.assert_array_equal(
                    out.cpu().numpy().astype(np.int64),
                    want_ix.query(c.ir_bytes, c.num_result_slots),
                    err_msg=f"{lanes} lanes, {c.query_text}")
                overflow = want_ix.last_status & oracle.OracleIndex.STATUS_OVERFLOW
                assert cuda_ctx.query_status() == (gpj.GPJ_QUERY_OVERFLOW if overflow else 0)
    finally:
        cuda_ctx.free_index(ix)


@pytest.mark.parametrize("end", range(7))
def test_every_split_of_a_batch_matches_oracle(gpj, end):
    """Files of several queries share a launch: records of different files,
    queries and empty files meet in one warp."""
    _, count = _counts()[end]
    rng = random.Random(100 + end)
    cuts = [max(1, count // 3), 0, count // 4, 1, 2]
    cuts.append(max(1, count - sum(max(c, 1) for c in cuts)))
    files = [_lines(1000 + 10 * end + i, c) if c else b"" for i, c in enumerate(cuts)]
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in
            [("$.k", 0), ("$.arr[1:4].k", 0), ("$.key.ab", 0)]]
    queries = [(c, 0, c.max_depth) for c in comp]
    packed, offsets = gpj.pack_files(files)
    kinds = [rng.randrange(3) for _ in files]
    dev = torch.from_numpy(packed).cuda()
    table = [(o, len(f), k) for o, f, k in zip(offsets, files, kinds)]
    with gpj.Batch(dev.data_ptr(), packed.size, table, queries) as b:
        b.run()
        torch.cuda.synchronize()
        v = b.view()
        from devmem import d2h
        info = d2h(v.d_file_info, len(files) * 8, np.uint64).reshape(-1, 8)
        got = d2h(v.d_results, v.result_ints, np.int32)
        for f, k, row in zip(files, kinds, info):
            c = comp[k]
            lines, off = int(row[0]), int(row[3])
            res = got[off:off + lines * c.num_result_slots * 2].reshape(lines, -1, 2)
            if not f:
                assert (res == -1).all()
                continue
            want = oracle.OracleIndex(np.frombuffer(f, np.uint8), c.max_depth).query(
                c.ir_bytes, c.num_result_slots)
            np.testing.assert_array_equal(res.astype(np.int64), want, err_msg=c.query_text)


@pytest.mark.parametrize("blocks", [4, 5, 6])
@pytest.mark.parametrize("query", ["$.key.ab", "$.arr[*]"])
def test_one_lane_at_every_block_count(cuda_ctx, gpj, blocks, query):
    """One lane per record in launches of one full wave of 4, 5 or 6 blocks per
    SM, plus the records of a half block."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = sms * 256 * blocks - 128
    part = _lines(77, 20000)
    data = np.frombuffer(b"\n".join([part] * (count // 20000 + 1)), np.uint8)
    ends = np.flatnonzero(data == 10)
    data = data[: int(ends[count - 1])]
    c = gpj.compile(query, wildcard_limit=4)
    buf = torch.from_numpy(data.copy()).cuda()
    ix = cuda_ctx.build_index(buf.data_ptr(), data.size, c.max_depth)
    try:
        assert ix.num_lines == count
        out = torch.full((count, c.num_result_slots, 2), -7, dtype=torch.int32, device="cuda")
        cuda_ctx.query(ix, c, out.data_ptr())
        torch.cuda.synchronize()
        cuda_ctx.query_status()
        want = oracle.OracleIndex(data, c.max_depth).query(c.ir_bytes, c.num_result_slots)
        np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64), want)
    finally:
        cuda_ctx.free_index(ix)


@pytest.mark.parametrize("waves", [(4, 0), (4, 1), (5, 0), (5, 1), (9, 1)], ids=str)
def test_one_lane_batch_at_every_block_count(gpj, waves):
    """A batch's one-lane launches at both ends of the range that takes five
    blocks per SM, and one whose warps take further runs of records."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = sms * 256 * waves[0] + waves[1]
    part = _lines(78, 20000)
    tail = b"\n".join(part.split(b"\n")[: count % 20000])
    files = [part] * (count // 20000) + [tail]
    c = gpj.compile("$.key.ab")
    packed, offsets = gpj.pack_files(files)
    dev = torch.from_numpy(packed).cuda()
    table = [(o, len(f), 0) for o, f in zip(offsets, files)]
    want = {f: oracle.OracleIndex(np.frombuffer(f, np.uint8), c.max_depth).query(
        c.ir_bytes, c.num_result_slots) for f in (part, tail)}
    with gpj.Batch(dev.data_ptr(), packed.size, table, [(c, 0, c.max_depth)]) as b:
        for _ in range(2):
            b.run()
        torch.cuda.synchronize()
        v = b.view()
        from devmem import d2h
        info = d2h(v.d_file_info, len(files) * 8, np.uint64).reshape(-1, 8)
        got = d2h(v.d_results, v.result_ints, np.int32)
        assert sum(int(row[0]) for row in info) == count
        for f, row in zip(files, info):
            lines, off = int(row[0]), int(row[3])
            res = got[off:off + lines * c.num_result_slots * 2].reshape(lines, -1, 2)
            np.testing.assert_array_equal(res.astype(np.int64), want[f])


@pytest.mark.parametrize("kind", ["one", "eight", "nine", "long_ir"])
@pytest.mark.parametrize("count", [60, 9000, 40000])
def test_queries_of_one_host_call_share_launches(cuda_ctx, gpj, kind, count):
    """gpj_query_host launches as many queries together as fit (8 queries, 4 KiB
    of IR): plain, extension and descend queries side by side."""
    data = np.frombuffer(_lines(5, count), np.uint8)
    texts = {"one": QUERIES[:1], "eight": QUERIES[:8], "nine": QUERIES[4:13],
             "long_ir": [("$.%s" % (ch * 1500), 0) for ch in "abcq"] + QUERIES[:2]}[kind]
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in texts]
    levels = min(8, max(c.max_depth for c in comp))
    host = torch.from_numpy(data.copy()).pin_memory()
    outs = [torch.full((count, c.num_result_slots, 2), -7, dtype=torch.int32).pin_memory()
            for c in comp]
    try:
        lines = cuda_ctx.query_host(host.data_ptr(), data.size, levels, comp,
                                    [o.data_ptr() for o in outs], [o.numel() for o in outs])
        assert lines == count
    except gpj.CapacityError:  # raised after the copies: a slice was truncated
        assert any(k for _, k in texts)
    want_ix = oracle.OracleIndex(data, levels)
    for c, o in zip(comp, outs):
        np.testing.assert_array_equal(o.numpy().astype(np.int64),
                                      want_ix.query(c.ir_bytes, c.num_result_slots),
                                      err_msg=c.query_text)
