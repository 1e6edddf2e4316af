"""\"..name\" runs a record with 32, 8 or one lane, by the number of records and
their length, and other queries take one lane on records of a bitmap word: each
against the oracle at both ends of its range, alone, in batches and 64 bits
wide."""
import random

import numpy as np
import pytest
import torch

import oracle
from devmem import d2h
from kernel_trace import launches

pytestmark = pytest.mark.gpu


def _member(rng, depth=0):
    r = rng.random()
    if depth > 3 or r < 0.4:
        return rng.choice(["1", '"k"', '"\\"k\\":1"', "null", "[]", "{}", '{"k":2}', "-1e3"])
    if r < 0.6:
        return "[" + ",".join(_member(rng, depth + 1) for _ in range(rng.randint(1, 4))) + "]"
    keys = rng.sample(["k", "kk", "key", "K", "name", "ab"], rng.randint(1, 4))
    return "{" + ",".join('"%s"%s:%s%s' % (k, rng.choice(["", " "]), rng.choice(["", "  "]),
                                           _member(rng, depth + 1)) for k in keys) + "}"


def _line(rng, mean):
    r = rng.random()
    if r < 0.05:
        return "".join(rng.choices('{}[]:,"\\k ', k=rng.randint(0, mean)))
    if r < 0.08:
        return "{" + '"k":' * rng.randint(1, max(1, mean // 5)) + "}"
    text = _member(rng)
    if text[0] != "{":
        text = '{"k":%s}' % text
    fill = max(0, int(rng.expovariate(1 / mean)) - len(text) - 8)
    body = '"%s":"%s",' % (rng.choice(["k", "f"]), "x" * (fill // 2)) if fill else ""
    tail = ',"k":[%s]' % ",".join("7" * rng.randint(1, 9) for _ in range(fill // 12)) if fill else ""
    return "{" + body + text[1:-1] + (tail if len(text) > 2 else "") + "}"


def _data(count, mean):
    rng = random.Random(count + mean)
    pool = [_line(rng, mean) for _ in range(700)]
    if mean < 64:
        pool = [x for x in pool if len(x) < mean] + ['{"k":1}', '{"k":{"k":"k"}}', "{}", "", "[]"]
    # the mean decides the lanes: padded to it by blanks in front of the lines
    lines = [rng.choice(pool) for _ in range(count)]
    short = mean * count - sum(len(x) + 1 for x in lines)
    if short > 0:
        pad = short // count
        lines = [" " * pad + x for x in lines]
    return np.frombuffer("\n".join(lines).encode(), np.uint8)


def _lanes(count, size, descends):
    threads = torch.cuda.get_device_properties(0).multi_processor_count * 1024
    mean = size // count
    if count * 32 <= threads:
        return 32
    if descends:
        if mean <= 1024:
            return 8 if count * 8 <= threads else 1
        return 8 if mean <= 2048 else 32
    if mean <= 64:
        return 1
    return next((g for g in (16, 8) if count * g <= threads), 1)


QUERIES = [("$..k", 3), ("$.k..key", 2), ("$.k", 0), ("$.k[?(@.k >= 1)].k", 0)]


@pytest.mark.parametrize("count,mean", [(300, 30), (4800, 30), (9000, 40), (4800, 66), (19100, 40),
                                        (18900, 90), (19100, 90), (4800, 1500), (9000, 900),
                                        (19500, 900), (19500, 1400), (5000, 2300)])
def test_lanes_by_records_and_length(cuda_ctx, gpj, count, mean):
    data = _data(count, mean)
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in QUERIES]
    levels = 5
    dev = torch.from_numpy(data.copy()).cuda()
    want_ix = oracle.OracleIndex(data, levels)
    want = [want_ix.query(c.ir_bytes, c.num_result_slots) for c in comp]
    ix = cuda_ctx.build_index(dev.data_ptr(), data.size, levels)
    try:
        assert ix.num_lines == count
        for c, w in zip(comp, want):
            for wide in (False, True):
                out = torch.full((count, c.num_result_slots, 2), -7, device="cuda",
                                 dtype=torch.int64 if wide else torch.int32)

                def run():
                    cuda_ctx.query(ix, c, out.data_ptr(), wide=wide)

                (name, _, _), = launches(run, "query_kernel")
                got = name.split("query_kernel<")[1].split(">")[0].split(", ")
                assert int(got[3]) == _lanes(count, data.size, ".." in c.query_text)
                np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64), w,
                                              err_msg=f"{c.query_text}, wide {wide}")
        cuda_ctx.query_status()
    finally:
        cuda_ctx.free_index(ix)
    for c, w in zip(comp, want):
        with gpj.Batch(dev.data_ptr(), data.size, [(0, data.size, 0)], [(c, 0, levels)]) as b:
            b.run()
            torch.cuda.synchronize()
            v = b.view()
            got = d2h(v.d_results, v.result_ints, np.int32).reshape(w.shape)
        np.testing.assert_array_equal(got.astype(np.int64), w, err_msg=c.query_text)


def test_two_gib_of_short_records(cuda_ctx, gpj):
    """64-bit positions: one lane for short records, 32 otherwise."""
    for line, count in ((b'{"k":1,"a":{"k":[2,{"k":3}]}}\n', 72_000_000),
                        (b'{"a":{"k":[2,{"k":3}]},"f":"%s","k":4}\n' % (b"x" * 1200), 1_750_000)):
        data = torch.from_numpy(np.frombuffer(line, np.uint8).copy()).cuda().repeat(count)
        assert data.numel() > 1 << 31
        c = gpj.compile("$..k", wildcard_limit=2)
        ix = cuda_ctx.build_index(data.data_ptr(), data.numel(), 5)
        try:
            one = torch.from_numpy(oracle.OracleIndex(line, 5).query(c.ir_bytes, 2)[:1]).cuda()
            out = torch.full((ix.num_lines, 2, 2), -7, dtype=torch.int64, device="cuda")
            cuda_ctx.query(ix, c, out.data_ptr(), wide=True)
            starts = torch.arange(count, dtype=torch.int64, device="cuda")[:, None, None] * len(line)
            assert torch.equal(out[:count], one + starts)
            assert (out[count:] == -1).all()
            assert cuda_ctx.query_status() == gpj.GPJ_QUERY_OVERFLOW
        finally:
            cuda_ctx.free_index(ix)
        del out, data, starts
