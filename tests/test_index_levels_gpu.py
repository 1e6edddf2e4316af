"""Indexes of more than eight levels take their levels in passes of eight; a
warp walks a later pass only where its depths may reach those levels.  Checked
against the oracle where warps skip passes, walk them, and wrap the
signed-char depth from either end."""
import random

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _text(seed, kind):
    rng = random.Random(seed)
    parts = []
    for _ in range(70):
        r = rng.random()
        if kind == "shallow" or r < 0.3:
            parts.append(b'{"a":[1,2,{"b":{"c":[3]}}],"d":"x' + b"]" * rng.randrange(0, 900) + b'"}\n')
        elif r < 0.5:
            n = rng.randrange(6, 24)
            parts.append(b'{"k":' * n + b"1,2" + b"}" * n + b",\n")
        elif r < 0.65:
            parts.append(b"[" * rng.randrange(1, 300))
        elif r < 0.85:
            parts.append(b"]" * rng.randrange(1, 300))
        else:
            parts.append(bytes(rng.choices(b"{}[]:,", k=rng.randrange(100, 5000))))
    return np.frombuffer(b"".join(parts), np.uint8)


@pytest.mark.parametrize("kind", ["shallow", "deep"])
@pytest.mark.parametrize("levels", [8, 9, 15, 16, 17, 22])
def test_levels_in_passes(cuda_ctx, gpj, levels, kind):
    data = _text(levels, kind)
    n, words = data.size, (data.size + 63) // 64
    want = oracle.OracleIndex(data, levels)
    dev = torch.from_numpy(data.copy()).cuda()
    new = lambda k: torch.full((k,), -1, dtype=torch.int64, device="cuda")  # noqa: E731
    lb, s, nl, summary = new(words * levels), new(words), new(want.num_lines), new(4)
    ix = gpj.Index()
    ix.d_leveled, ix.d_string, ix.d_newline = lb.data_ptr(), s.data_ptr(), nl.data_ptr()
    ix.newline_capacity = want.num_lines
    cuda_ctx.build_index_async(dev.data_ptr(), n, levels, ix, summary.data_ptr())
    torch.cuda.synchronize()
    assert summary.cpu().tolist()[3] == 0
    got = lb.cpu().numpy().view(np.uint64).reshape(levels, words)
    np.testing.assert_array_equal(got, np.asarray(want.LB).reshape(levels, words))
    assert (got[8:] != 0).any() == (kind == "deep" and levels > 8)
