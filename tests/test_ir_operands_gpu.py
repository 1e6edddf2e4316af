"""IR whose operands claim more text than there is: lengths up to 2^31 - 1 end
the record, in every split of the query kernel and in batches, as the oracle
(64-bit positions) has it."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

HUGE = b"\xff\xff\xff\xff\x07"  # 2^31 - 1
END, STORE, DOWN, KEY, INDEX, EQUALS, NUMBER, DESCEND = (
    bytes([b]) for b in (0, 1, 3, 4, 5, 9, 10, 11))
IRS = [
    KEY + HUGE + b"k" + DOWN + STORE + END,
    KEY + b"\x01k" + DOWN + STORE + KEY + HUGE + b"k" + END,
    KEY + b"\x01k" + DOWN + KEY + HUGE,
    KEY + b"\xff\xff\xff\xff\x0f" + b"k" + DOWN + STORE + END,  # -1
    KEY + b"\xff\xff\xff\xff\xff\x07" + DOWN + STORE + END,  # six bytes
    KEY + b"\x05k" + DOWN + STORE + END,  # past the end by one
    KEY + b"\x04k" + DOWN + STORE + END,  # to the end
    KEY + b"\x01k" + DOWN + STORE,  # no END
    STORE + EQUALS + HUGE + b'"v"' + STORE + END,
    KEY + b"\x01n" + DOWN + NUMBER + b"\x04" + HUGE + b"10" + STORE + END,
    KEY + b"\x01n" + DOWN + NUMBER + b"\x04\x03" + b"10",
    DESCEND + HUGE + b"k" + END,
    DESCEND + b"\x02k",
    DESCEND + b"\x01k" + DESCEND + HUGE,
    KEY + b"\x01a" + DOWN + INDEX + HUGE + DOWN + STORE + END,
]
LINES = [b"{}", b'{"k":1}', b'{"k":{"k":2}, "a":[1,2,3]}', b'{"n":12,"k":"v"}', b"[]", b'"v"',
         b'{"a":[{"k":3}],"n":9}', b"{:}", b""]


def _data(count):
    return np.frombuffer(b"\n".join(LINES[i % len(LINES)] for i in range(count)), np.uint8)


@pytest.mark.parametrize("count", [40, 9000, 15000, 40000])  # 32, 16, 8 and one lane
@pytest.mark.parametrize("wide", [False, True], ids=["int32", "int64"])
def test_overlong_operands_match_oracle(cuda_ctx, gpj, count, wide):
    data = _data(count)
    buf = torch.from_numpy(data.copy()).cuda()
    want_ix = oracle.OracleIndex(data, 4)
    ix = cuda_ctx.build_index(buf.data_ptr(), data.size, 4)
    try:
        for ir in IRS:
            out = torch.full((count, 2, 2), -7, device="cuda",
                             dtype=torch.int64 if wide else torch.int32)
            cuda_ctx.query(ix, gpj.CompiledQuery("", ir, 4, 2), out.data_ptr(), wide=wide)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(out.cpu().numpy().astype(np.int64),
                                          want_ix.query(ir, 2), err_msg=ir.hex())
        cuda_ctx.query_status()
    finally:
        cuda_ctx.free_index(ix)


@pytest.mark.parametrize("count", [40, 40000])
def test_overlong_operands_in_a_batch(gpj, count):
    from devmem import d2h
    for at in range(0, len(IRS), 5):
        irs = IRS[at:at + 5]
        files = [bytes(_data(count // len(irs)))] * len(irs)
        packed, offsets = gpj.pack_files(files)
        dev = torch.from_numpy(packed).cuda()
        table = [(o, len(f), k) for k, (o, f) in enumerate(zip(offsets, files))]
        with gpj.Batch(dev.data_ptr(), packed.size, table,
                       [(gpj.CompiledQuery("", ir, 4, 2), 0, 4) for ir in irs]) as b:
            b.run()
            torch.cuda.synchronize()
            v = b.view()
            info = d2h(v.d_file_info, len(files) * 8, np.uint64).reshape(-1, 8)
            got = d2h(v.d_results, v.result_ints, np.int32)
        want_ix = oracle.OracleIndex(np.frombuffer(files[0], np.uint8), 4)
        for ir, row in zip(irs, info):
            lines, off = int(row[0]), int(row[3])
            np.testing.assert_array_equal(
                got[off:off + lines * 4].reshape(lines, 2, 2).astype(np.int64),
                want_ix.query(ir, 2), err_msg=ir.hex())
