"""The server moves small pinned inputs and small results by one kernel for all
requests of a pass and the others by copies of their own: both ways, at the
sizes and alignments between them, against the oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _file(size, seed):
    """`size` bytes of short records."""
    rng = np.random.default_rng(seed)
    line = b'{"a":%d,"b":["x",{"c":"y"}]}\n'
    text = b"".join(line % int(v) for v in rng.integers(0, 10**6, max(1, size // 30)))
    return np.frombuffer((text + b" " * size)[:size], np.uint8)


@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
@pytest.mark.parametrize("offset", [0, 16, 4, 1])
def test_inputs_and_results_of_every_size(gpj, pinned, offset):
    sizes = [1, 15, 16, 17, 4095, 16384, 16385, 100_001, MIB - 1, MIB, MIB + 1, 3 * MIB + 5, 0, 333]
    step = 4 * MIB
    host = torch.zeros(step * len(sizes), dtype=torch.uint8)
    host = host.pin_memory() if pinned else host
    view = host.numpy()
    comp = [gpj.compile("$.a"), gpj.compile("$.b[1].c")]
    queries = [(c, 0, c.max_depth) for c in comp]
    datas = []
    for i, n in enumerate(sizes):
        part = view[i * step + offset:i * step + offset + n]
        part[:] = _file(n, i)
        datas.append(part)
    srv = gpj.Server(0, num_slots=32, hbm_budget_bytes=512 * MIB, host_result_bytes=64 * MIB)
    try:
        ids = srv.submit_prepared(srv.prepare([(d, queries, 0, 0) for d in datas]))
        left = set(ids)
        while left:
            left.difference_update(srv.poll(timeout_us=2_000_000))
        for rid, d in zip(ids, datas):
            got = srv.response(rid)
            assert got.status == 0, got.message
            if d.size == 0:
                continue
            want_ix = oracle.OracleIndex(d, max(c.max_depth for c in comp))
            assert got.num_lines == want_ix.num_lines
            for c, res in zip(comp, got.results):
                np.testing.assert_array_equal(res.astype(np.int64),
                                              want_ix.query(c.ir_bytes, c.num_result_slots))
    finally:
        srv.close()
