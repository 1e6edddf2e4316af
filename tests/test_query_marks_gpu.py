"""Queries whose IR holds many bytes equal to the mark opcode (seven-letter
keys, element 7) or many open marks, on partitions of 2 GiB and more: the
64-bit kernels run them in every split.  Also one 16-level query with 16 open
marks on small partitions, in batches too."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

MARK, RESET = b"\x07", b"\x08"


def _deep(gpj):
    """16 open marks, then 15 levels down."""
    ir = MARK * 16 + RESET * 16 + b"\x04\x01d\x03" * 15 + b"\x01\x00"
    return gpj.CompiledQuery("", ir, 16, 1)


def _queries(gpj):
    return [gpj.compile("$.orders[*].country", wildcard_limit=16),
            gpj.compile("$.a.b.c[0:16].message"),
            gpj.compile("$.entities.user_mentions[*].profile.country", wildcard_limit=16),
            gpj.compile("$.entities[?(@.user_mentions[7].profile.country == 7)]"
                        ".user_mentions[-2:].profile.country"),
            gpj.compile("$..country", wildcard_limit=16), _deep(gpj)]


def _line(size):
    items = ",".join('{"country":"c%d","message":"m"}' % i for i in range(12))
    mentions = ",".join('{"profile":{"country":%d}}' % i for i in range(9))
    text = '{"orders":[%s],"a":{"b":{"c":[%s]}},"entities":{"user_mentions":[%s]},"d":%s,"fill":"' \
        % (items, items, mentions, '{"d":' * 14 + "5" + "}" * 14)
    return (text + "f" * (size - len(text) - 3) + '"}\n').encode()


@pytest.mark.parametrize("records", [2, 2300, 5600], ids=["32 lanes", "32 lanes, waves", "1 lane"])
def test_two_gib_partition_with_many_mark_bytes(cuda_ctx, gpj, records):
    line = _line(((2200 << 20) // records))
    data = torch.from_numpy(np.frombuffer(line, np.uint8).copy()).cuda().repeat(records)
    n = data.numel()
    assert n > 1 << 31
    ix = cuda_ctx.build_index(data.data_ptr(), n, 16)
    try:
        short = _line(4097)  # the same record without most of its filler
        assert short[:3000] == line[:3000]
        want_ix = oracle.OracleIndex(short, 16)
        for c in _queries(gpj):
            out = torch.full((ix.num_lines, c.num_result_slots, 2), -7, dtype=torch.int64,
                             device="cuda")
            cuda_ctx.query(ix, c, out.data_ptr(), wide=True)
            torch.cuda.synchronize()
            one = torch.from_numpy(want_ix.query(c.ir_bytes, c.num_result_slots)[:1])
            starts = torch.arange(records, dtype=torch.int64)[:, None, None] * len(line)
            want = torch.where(one >= 0, one + starts, -1)
            got = out.cpu()
            assert torch.equal(got[:records], want), c.query_text
            assert (got[records:] == -1).all()
        cuda_ctx.query_status()
    finally:
        cuda_ctx.free_index(ix)


@pytest.mark.parametrize("count", [40, 40000], ids=["32 lanes", "1 lane"])
@pytest.mark.parametrize("wide", [False, True], ids=["int32", "int64"])
def test_sixteen_marks_and_levels(cuda_ctx, gpj, count, wide):
    from devmem import d2h
    line = _line(1501)
    data = np.frombuffer(line * count, np.uint8)[:-1]
    want = oracle.OracleIndex(data, 16)
    dev = torch.from_numpy(data.copy()).cuda()
    ix = cuda_ctx.build_index(dev.data_ptr(), data.size, 16)
    try:
        for c in _queries(gpj):
            out = torch.full((count, c.num_result_slots, 2), -7, device="cuda",
                             dtype=torch.int64 if wide else torch.int32)
            cuda_ctx.query(ix, c, out.data_ptr(), wide=wide)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64),
                                          want.query(c.ir_bytes, c.num_result_slots),
                                          err_msg=c.query_text)
        cuda_ctx.query_status()
    finally:
        cuda_ctx.free_index(ix)
    c = _deep(gpj)
    with gpj.Batch(dev.data_ptr(), data.size, [(0, data.size, 0)], [(c, 0, 16)]) as b:
        b.run()
        torch.cuda.synchronize()
        v = b.view()
        got = d2h(v.d_results, v.result_ints, np.int32).reshape(count, 1, 2)
    np.testing.assert_array_equal(got.astype(np.int64), want.query(c.ir_bytes, 1))
