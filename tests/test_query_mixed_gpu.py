"""Queries of different kinds in one call: each query's answer and status are
those it has alone."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _data(count):
    lines = ['{"arr":[%d,2,3],"user":{"lang":"l%d","n":%d},"n":7}' % (i, i % 9, i % 40)
             for i in range(count)]
    return np.frombuffer("\n".join(lines).encode(), np.uint8)


def _narrow(gpj):
    """Reference syntax with fewer slots than its IR stores: what does not fit
    is dropped without a status, as only the extensions have one."""
    c = gpj.compile("$.arr[0:3]")
    return gpj.CompiledQuery(c.query_text, c.ir_bytes, c.max_depth, 1)


OTHERS = [("$.user[?(@.n >= 10)].lang", 0), ("$.arr[*]", 3), ("$..n", 2)]


@pytest.mark.parametrize("other", OTHERS, ids=str)
@pytest.mark.parametrize("count", [50, 40000])
def test_dropped_results_of_a_plain_query_raise_no_status(cuda_ctx, gpj, other, count):
    data = _data(count)
    ext = gpj.compile(other[0], wildcard_limit=other[1])
    comp = [_narrow(gpj), ext]
    levels = min(3, max(c.max_depth for c in comp))
    want_ix = oracle.OracleIndex(data, levels)
    want = [want_ix.query(c.ir_bytes, c.num_result_slots) for c in comp]
    host = torch.from_numpy(data.copy()).pin_memory()
    outs = [torch.full((count, c.num_result_slots, 2), -7, dtype=torch.int32).pin_memory()
            for c in comp]
    assert cuda_ctx.query_host(host.data_ptr(), data.size, levels, comp,
                               [o.data_ptr() for o in outs], [o.numel() for o in outs]) == count
    for o, w in zip(outs, want):
        np.testing.assert_array_equal(o.numpy().astype(np.int64), w)
    # a batch of one file per query
    packed, offsets = gpj.pack_files([data, data])
    packed_host = torch.from_numpy(packed).pin_memory()
    dev = torch.from_numpy(packed).cuda()
    with gpj.Batch(dev.data_ptr(), packed.size, [(o, data.size, k) for k, o in enumerate(offsets)],
                   [(c, 0, levels) for c in comp]) as b:
        v = b.view()
        got = torch.zeros(v.result_ints, dtype=torch.int32).pin_memory()
        b.run_host(packed_host.data_ptr(), got.data_ptr())
    first = count * 2
    np.testing.assert_array_equal(got[:first].numpy().reshape(count, 1, 2), want[0])
    np.testing.assert_array_equal(got[first:].numpy().reshape(count, -1, 2), want[1])
    # two requests of one server pass
    with gpj.Server(0, num_slots=4, hbm_budget_bytes=256 << 20, host_result_bytes=16 << 20) as srv:
        ids = srv.submit_prepared(srv.prepare([(data, [(c, 0, levels)], 0, 0) for c in comp]))
        for rid, w in zip(ids, want):
            srv.wait(rid)
            r = srv.response(rid)
            assert r.status == 0, r.message
            np.testing.assert_array_equal(r.results[0].astype(np.int64), w)


def test_an_extension_query_beside_a_plain_one_keeps_its_status(cuda_ctx, gpj):
    data = _data(50)
    comp = [gpj.compile("$.user.lang"), gpj.compile("$.arr[*]", wildcard_limit=2)]
    host = torch.from_numpy(data.copy()).pin_memory()
    outs = [torch.full((50, c.num_result_slots, 2), -7, dtype=torch.int32).pin_memory()
            for c in comp]
    with pytest.raises(gpj.CapacityError):
        cuda_ctx.query_host(host.data_ptr(), data.size, 2, comp, [o.data_ptr() for o in outs],
                            [o.numel() for o in outs])
    assert cuda_ctx.query_status() == gpj.GPJ_QUERY_OVERFLOW  # and clears it
