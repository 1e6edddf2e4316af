"""Result compaction at the edges of its blocks (512 pairs; the counting blocks
take 2,048) and of its ways to copy a text (8 lanes, a warp, the block), against
the same compaction in numpy; whole numbers and bytes, no tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(ctx, gpj, res, slots, data, base, skew, match_cap=None, arena_cap=None):
    lines = res.shape[0] // slots
    buf = torch.zeros(res.size + 8, dtype=torch.int32, device="cuda")
    buf[skew:skew + res.size] = torch.from_numpy(res.reshape(-1)).cuda()
    text = torch.from_numpy(data).cuda()
    some = (res >= 0).all(1)
    bad = some & ((res[:, 0] > res[:, 1]) | (res[:, 1] > data.size))
    idx = np.flatnonzero(some & ~bad)
    start, end = res[idx, 0].astype(np.int64), res[idx, 1].astype(np.int64)
    length = end - start
    offset = np.cumsum(length) - length
    match_cap = idx.size if match_cap is None else match_cap
    arena_cap = int(length.sum()) if arena_cap is None else arena_cap
    matches = torch.full((max(match_cap, 1) * 5,), -1, dtype=torch.int64, device="cuda")
    arena = torch.full((max(arena_cap, 1) + 64,), 0xEE, dtype=torch.uint8, device="cuda")
    counts = torch.full((3,), 77, dtype=torch.int64, device="cuda")
    ctx.compact(buf[skew:].data_ptr(), lines, slots, text.data_ptr(), data.size, base,
                matches.data_ptr(), match_cap, arena.data_ptr(), arena_cap, counts.data_ptr())
    torch.cuda.synchronize()
    assert counts.cpu().tolist() == [idx.size, int(length.sum()), int(bad.sum())]
    got = matches.cpu().numpy().view(gpj.MATCH_DTYPE)[: min(match_cap, idx.size)]
    keep = slice(0, got.size)
    for name, want in (("line", idx // slots), ("slot", idx % slots), ("length", length),
                       ("start", start + base), ("end", end + base), ("text_offset", offset)):
        np.testing.assert_array_equal(got[name], want[keep], err_msg=name)
    want_arena = np.full(arena.numel(), 0xEE, np.uint8)
    for s, e, o in zip(start, end, offset):
        if o + (e - s) <= arena_cap:
            want_arena[o:o + e - s] = data[s:e]
    np.testing.assert_array_equal(arena.cpu().numpy(), want_arena)


@pytest.mark.parametrize("skew", [0, 1, 2], ids=["aligned", "skew1", "skew2"])
@pytest.mark.parametrize("slots,lines", [(1, 1), (1, 511), (1, 512), (1, 2049), (2, 1025), (3, 4099),
                                         (8, 2600), (7, 147000)])
def test_blocks_and_order(cuda_ctx, gpj, slots, lines, skew):
    rng = np.random.default_rng(lines)
    data = rng.integers(0, 256, 1 << 20, dtype=np.uint8)
    start = rng.integers(0, data.size - 40, lines * slots)
    res = np.stack([start, start + rng.integers(0, 24, start.size)], 1).astype(np.int32)
    res[rng.random(start.size) < 0.5] = -1
    res[rng.random(start.size) < 0.01, 0] = -1  # one side only: no match
    bad = rng.random(start.size) < 0.003
    res[bad, 0], res[bad, 1] = 9, 5
    _run(cuda_ctx, gpj, res, slots, data, 5_000_000_000, skew)


@pytest.mark.parametrize("caps", [(None, None), (300, 40_000), (2048, None), (5, 0)])
def test_long_texts_and_capacities(cuda_ctx, gpj, caps):
    rng = np.random.default_rng(3)
    data = rng.integers(0, 256, 1 << 20, dtype=np.uint8)
    length = rng.choice([0, 1, 7, 8, 255, 256, 257, 1000, 16384, 16385, 70001], 4500,
                        p=[0.1, 0.2, 0.2, 0.2, 0.1, 0.09, 0.09, 0.01, 0.004, 0.004, 0.002])
    start = rng.integers(0, data.size - 80_000, length.size)
    res = np.stack([start, start + length], 1).astype(np.int32)
    _run(cuda_ctx, gpj, res, 2, data, 0, 0, *caps)
