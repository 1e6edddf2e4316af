"""The calls whose launches overlap one another, captured in a CUDA graph and
replayed on other inputs, and with a summary at any address."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _index(gpj, words, levels, lines):
    new = lambda k: torch.zeros(k, dtype=torch.int64, device="cuda")  # noqa: E731
    out = {"d_string": new(words), "d_leveled": new(words * levels), "d_newline": new(lines)}
    ix = gpj.Index()
    for name, t in out.items():
        setattr(ix, name, t.data_ptr())
    ix.newline_capacity = lines
    return ix, out


@pytest.mark.parametrize("noalloc", [False, True], ids=["context", "noalloc"])
def test_build_query_and_compaction_in_a_graph(gpj, noalloc):
    from gpjson_b200 import datagen
    size, levels = 3 << 20, 4
    texts = [datagen.tweets(s, size)[:size] for s in (1, 2, 3)]
    c = gpj.compile("$.entities.hashtags[0:8].text")
    wants = [oracle.OracleIndex(t, levels) for t in texts]
    lines = max(w.num_lines for w in wants)
    buf = torch.from_numpy(texts[0].copy()).cuda()
    words = (size + 63) // 64
    ix, out = _index(gpj, words, levels, lines)
    ix.num_lines = lines
    summary = torch.zeros(4, dtype=torch.int64, device="cuda")
    res = torch.zeros((lines, c.num_result_slots, 2), dtype=torch.int32, device="cuda")
    pairs = res.numel() // 2
    matches = torch.zeros((pairs, 5), dtype=torch.int64, device="cuda")
    arena = torch.zeros(pairs * 64, dtype=torch.uint8, device="cuda")
    counts = torch.zeros(3, dtype=torch.int64, device="cuda")
    with gpj.Context(0) as ctx:
        def work(stream):
            if noalloc:
                gpj.build_index_noalloc(buf.data_ptr(), size, levels, ix, summary.data_ptr(),
                                        stream=stream)
            else:
                ctx.build_index_async(buf.data_ptr(), size, levels, ix, summary.data_ptr(),
                                      stream=stream)
            ctx.query(ix, c, res.data_ptr(), stream=stream)
            ctx.compact(res.data_ptr(), lines, c.num_result_slots, buf.data_ptr(), size, 0,
                        matches.data_ptr(), pairs, arena.data_ptr(), arena.numel(),
                        counts.data_ptr(), stream=stream)

        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            work(side.cuda_stream)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            work(side.cuda_stream)
        for text, want in list(zip(texts, wants)) * 2:
            buf.copy_(torch.from_numpy(text.copy()))
            out["d_newline"].fill_(size - 1)  # the lines past the last one are empty
            graph.replay()
            torch.cuda.synchronize()
            got = [int(v) for v in summary.cpu()]
            assert got[0] == want.num_lines and got[3] == 0
            np.testing.assert_array_equal(out["d_string"].cpu().numpy().view(np.uint64), want.S)
            np.testing.assert_array_equal(out["d_leveled"].cpu().numpy().view(np.uint64), want.LB)
            expect = want.query(c.ir_bytes, c.num_result_slots)
            have = res.cpu().numpy()[: want.num_lines].astype(np.int64)
            np.testing.assert_array_equal(have[:-1], expect[:-1])
            some = (res.cpu().numpy().reshape(-1, 2) >= 0).all(1)
            m = int(counts[0])
            assert m == int(some.sum()) and int(counts[2]) == 0
            got_m = matches.cpu().numpy().view(gpj.MATCH_DTYPE).reshape(-1)[:m]
            np.testing.assert_array_equal(got_m["start"], res.cpu().numpy().reshape(-1, 2)[some, 0])
            blob = b"".join(text[s:e].tobytes() for s, e in zip(got_m["start"], got_m["end"]))
            assert arena[: len(blob)].cpu().numpy().tobytes() == blob
        del graph


@pytest.mark.parametrize("skew", [0, 4, 1])
@pytest.mark.parametrize("size", [0, 100, 100_000])
@pytest.mark.parametrize("noalloc", [False, True], ids=["context", "noalloc"])
def test_summary_at_any_address(cuda_ctx, gpj, noalloc, size, skew):
    from gpjson_b200 import datagen
    data = datagen.tweets(9, 200_000)[:size]
    want = oracle.OracleIndex(data, 2) if size else None
    buf = torch.zeros(max(size, 1), dtype=torch.uint8, device="cuda")
    buf[:size] = torch.from_numpy(data.copy())
    ix, _ = _index(gpj, max(1, (size + 63) // 64), 2, want.num_lines if size else 1)
    if size == 0 and noalloc and skew:
        pytest.skip("an empty build writes its words in a kernel")
    raw = torch.full((64,), 0xEE, dtype=torch.uint8, device="cuda")
    if noalloc:
        gpj.build_index_noalloc(buf.data_ptr(), size, 2, ix, raw.data_ptr() + skew)
    else:
        cuda_ctx.build_index_async(buf.data_ptr(), size, 2, ix, raw.data_ptr() + skew)
    torch.cuda.synchronize()
    got = raw.cpu().numpy()[skew:skew + 32].copy().view(np.int64)
    assert got.tolist()[0] == (want.num_lines if size else 1) and got[3] == 0
    assert raw.cpu().numpy()[skew + 32] == 0xEE
