"""Partitions of 2^31 - 2, 2^31 - 1 and 2^31 bytes: the largest that 32-bit
positions hold and the first beyond, with one record from the first byte to the
last, and with a last record that is an empty object up to the last byte (32
lanes and one lane per record)."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

HEAD = b'{"arr":[10,{"k":5},"x"],"key":{"ab":7},"fill":"'


@pytest.mark.parametrize("n", [(1 << 31) - 2, (1 << 31) - 1, 1 << 31])
def test_one_record_of_two_gib(cuda_ctx, gpj, n):
    data = torch.full((n,), ord("f"), dtype=torch.uint8, device="cuda")
    data[:len(HEAD)] = torch.from_numpy(np.frombuffer(HEAD, np.uint8).copy())
    data[-2:] = torch.tensor(list(b'"}'), dtype=torch.uint8)
    want_ix = oracle.OracleIndex(HEAD + b'f"}', 4)
    ix = cuda_ctx.build_index(data.data_ptr(), n, 4)
    try:
        assert ix.num_lines == 1
        for text, limit in [("$.arr[1].k", 0), ("$.arr[2]", 0), ("$.arr[-1]", 0), ("$.arr[*]", 4),
                            ("$.arr[1:-1].k", 4), ("$.key.ab", 0), ("$.nokey", 0), ("$..k", 2)]:
            c = gpj.compile(text, wildcard_limit=limit)
            want = want_ix.query(c.ir_bytes, c.num_result_slots)
            for wide in ((False, True) if n < 1 << 31 else (True,)):
                out = torch.full((1, c.num_result_slots, 2), -7, device="cuda",
                                 dtype=torch.int64 if wide else torch.int32)
                cuda_ctx.query(ix, c, out.data_ptr(), wide=wide)
                torch.cuda.synchronize()
                np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64), want,
                                              err_msg=f"{text}, wide {wide}")
        c = gpj.compile("$.fill")
        out = torch.full((2,), -7, dtype=torch.int64, device="cuda")
        cuda_ctx.query(ix, c, out.data_ptr(), wide=True)
        assert out.tolist() == [len(HEAD) - 1, n - 1]
        assert cuda_ctx.query_status() == 0
    finally:
        cuda_ctx.free_index(ix)


@pytest.mark.parametrize("before", [40, 20000], ids=["32 lanes", "1 lane"])
def test_empty_object_up_to_the_last_byte(cuda_ctx, gpj, before):
    n = (1 << 31) - 1
    line = (n - 20) // before  # records of one long string, then "{   }"
    data = np.full(n, ord("f"), np.uint8)
    rows = data[:line * before].reshape(before, line)
    rows[:, :6] = np.frombuffer(b'{"f":"', np.uint8)
    rows[:, -3:] = np.frombuffer(b'"}\n', np.uint8)
    data[line * before:] = ord(" ")
    data[line * before], data[-1] = ord("{"), ord("}")
    dev = torch.from_numpy(data).cuda()
    ix = cuda_ctx.build_index(dev.data_ptr(), n, 3)
    want_ix = oracle.OracleIndex(data, 3)
    try:
        for text in ("$.a", "$.f", "$.a.b", "$.a[1].b"):
            c = gpj.compile(text)
            want = want_ix.query(c.ir_bytes, 1)
            for wide in (False, True):
                out = torch.full((before + 1, 1, 2), -7, device="cuda",
                                 dtype=torch.int64 if wide else torch.int32)
                cuda_ctx.query(ix, c, out.data_ptr(), wide=wide)
                torch.cuda.synchronize()
                np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64), want,
                                              err_msg=f"{text}, wide {wide}")
        assert want[-1].tolist() == [[-1, -1]] and want_ix.query(gpj.compile("$.a").ir_bytes, 1)[
            -1].tolist() == [[n, n - 1]]
    finally:
        cuda_ctx.free_index(ix)
