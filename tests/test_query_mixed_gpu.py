"""Queries of different kinds in one call: each query's answer and status are
those it has alone."""
import re

import numpy as np
import pytest
import torch

import oracle
from kernel_trace import launches

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


def _query_kernels(run):
    """Variants that ran: the types or the extensions, the lanes per record, the
    blocks per SM (not whether a batch's launch is one of two)."""
    names = [name for name, _, _ in launches(run, "query_kernel")]
    variants = [re.search(r"query_kernel<([^>]*)>", name)[1].split(", ") for name in names]
    return {tuple(v[:3] if "batch" in name else v) for name, v in zip(names, variants)}


def test_a_descending_query_leaves_the_others_their_kernels(cuda_ctx, gpj):
    """One "..name" query in a call: the rest runs with the lanes per record
    that it has alone."""
    data = _data(40000)
    host = torch.from_numpy(data.copy()).pin_memory()
    lang, any_n = gpj.compile("$.user.lang"), gpj.compile("$..n", wildcard_limit=4)

    def host_call(comp):
        outs = [torch.empty((40000, c.num_result_slots, 2), dtype=torch.int32).pin_memory()
                for c in comp]
        return _query_kernels(lambda: cuda_ctx.query_host(
            host.data_ptr(), data.size, 3, comp, [o.data_ptr() for o in outs],
            [o.numel() for o in outs]))

    alone = [host_call([c]) for c in (lang, any_n)]
    assert all(len(k) == 1 for k in alone) and alone[0] != alone[1]
    assert host_call([lang, any_n]) == alone[0] | alone[1]

    packed, offsets = gpj.pack_files([data, _data(300)])
    dev = torch.from_numpy(packed).cuda()
    sizes = [data.size, _data(300).size]

    def batch_run(kinds):
        table = [(o, s, k) for o, s, k in zip(offsets, sizes, kinds)]
        with gpj.Batch(dev.data_ptr(), packed.size, table, [(lang, 0, 2), (any_n, 0, 3)]) as b:
            return _query_kernels(b.run)

    alone = [batch_run([0, 0]), batch_run([1, 1])]
    assert all(len(k) == 1 for k in alone) and alone[0] != alone[1]
    assert batch_run([0, 1]) == alone[0] | alone[1]


@pytest.mark.parametrize("count", [70, 9000, 15000, 40000, 260000])
@pytest.mark.parametrize("graph", [True, False], ids=["graph", "direct"])
def test_batches_of_descending_and_other_queries_match_oracle(gpj, count, graph):
    """Files of four queries, two of which descend, from empty and one-line
    files to most of the records, in every order."""
    import random

    from devmem import d2h
    from test_query_lanes_gpu import _lines
    rng = random.Random(count)
    cuts = [0, 1, 1, 1, 2, 0, 3, 40, 1, 0, 7, 1]
    while sum(max(c, 1) for c in cuts) < count:
        left = count - sum(max(c, 1) for c in cuts)
        cuts.append(min(left, rng.choice([1, 1, 5, 33, 700, count // 3, count])))
    rng.shuffle(cuts)
    files = [_lines(i, c) if c else b"" for i, c in enumerate(cuts)]
    kinds = [rng.randrange(4) for _ in files]
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in
            [("$.k", 0), ("$..k", 3), ("$.arr[1:-1].k", 4), ("$.key..ab", 2)]]
    levels = [2, 6, 3, 5]
    packed, offsets = gpj.pack_files(files)
    dev = torch.from_numpy(packed).cuda()
    table = [(o, len(f), k) for o, f, k in zip(offsets, files, kinds)]
    with gpj.Batch(dev.data_ptr(), packed.size, table,
                   [(c, 0, lv) for c, lv in zip(comp, levels)],
                   flags=0 if graph else gpj.GPJ_BATCH_NO_GRAPH) as b:
        v = b.view()
        assert v.num_records == count
        for _ in range(3):
            b.run()
        torch.cuda.synchronize()
        info = d2h(v.d_file_info, len(files) * 8, np.uint64).reshape(-1, 8)
        got = d2h(v.d_results, v.result_ints, np.int32)
    for f, k, row in zip(files, kinds, info):
        c = comp[k]
        lines, off = int(row[0]), int(row[3])
        res = got[off:off + lines * c.num_result_slots * 2].reshape(lines, -1, 2)
        want = oracle.OracleIndex(np.frombuffer(f, np.uint8), levels[k]).query(
            c.ir_bytes, c.num_result_slots) if f else np.full_like(res, -1)
        np.testing.assert_array_equal(res.astype(np.int64), want, err_msg=c.query_text)


def test_one_server_pass_of_descending_and_other_queries(gpj):
    from test_query_lanes_gpu import _lines
    comp = [gpj.compile(q, wildcard_limit=k) for q, k in
            [("$.k", 0), ("$..k", 3), ("$.arr[*]", 4), ("$.key.ab", 0)]]
    files = [np.frombuffer(_lines(50 + i, 5 + 200 * i), np.uint8) for i in range(12)]
    items = [(f, [(comp[(i + j) % 4], 0, 4) for j in range(1 + i % 3)], 0, 0)
             for i, f in enumerate(files)]
    with gpj.Server(0, num_slots=16, hbm_budget_bytes=256 << 20,
                    host_result_bytes=64 << 20) as srv:
        ids = srv.submit_prepared(srv.prepare(items))
        for rid, (data, queries, _, _) in zip(ids, items):
            srv.wait(rid)
            r = srv.response(rid)
            want_ix = oracle.OracleIndex(data, 4)
            overflow = False
            want = []
            for c, _, _ in queries:
                want.append(want_ix.query(c.ir_bytes, c.num_result_slots))
                overflow |= bool(want_ix.last_status & oracle.OracleIndex.STATUS_OVERFLOW)
            assert r.status == (gpj.GPJ_ERR_CAPACITY if overflow else 0)
            for got, w in zip(r.results, want):
                np.testing.assert_array_equal(got.astype(np.int64), w)
