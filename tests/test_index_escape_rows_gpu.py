"""The escape carry into the first row of a warp (every 4 KiB) is read back from
the row before it: backslash runs of every length up to and over a word ending
there, in rows that are staged, in the last rows of a file and on unaligned
inputs, against the oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _text(tail):
    """Quotes and backslash runs of 0 .. 70 that end at multiples of 4 KiB."""
    parts = bytearray()
    for run in list(range(0, 8)) + [31, 32, 33, 62, 63, 64, 65, 66, 70]:
        fill = 4096 - run
        block = (b'{"k":"' + b"x" * 4096)[:fill - 3] + b'"' + b"y" * 2
        parts += block[:fill] + b"\\" * run
    parts += b'"' + b"z" * tail
    return np.frombuffer(bytes(parts), np.uint8)


@pytest.mark.parametrize("flags", [0, 2], ids=["tma", "no_tma"])
@pytest.mark.parametrize("skew", [0, 3])
@pytest.mark.parametrize("tail", [0, 1, 127, 128, 129, 4095, 20000])
def test_runs_that_end_before_a_warps_first_row(cuda_ctx, gpj, tail, skew, flags):
    data = _text(tail)
    n, words, levels = data.size, (data.size + 63) // 64, 3
    want = oracle.OracleIndex(data, levels)
    buf = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    buf[skew:skew + n] = torch.from_numpy(data.copy())
    new = lambda k: torch.full((k,), -1, dtype=torch.int64, device="cuda")  # noqa: E731
    out = {"d_escape": new(words), "d_quote": new(words), "d_string": new(words),
           "d_leveled": new(words * levels), "d_newline": new(want.num_lines)}
    ix = gpj.Index()
    for name, t in out.items():
        setattr(ix, name, t.data_ptr())
    ix.newline_capacity = want.num_lines
    summary = new(4)
    cuda_ctx.build_index_async(buf.data_ptr() + skew, n, levels, ix, summary.data_ptr(),
                               flags=flags | gpj.GPJ_INDEX_EMIT_ESCAPE_QUOTE)
    torch.cuda.synchronize()
    assert summary.cpu().tolist()[3] == 0
    for name, exp in (("d_escape", want.E), ("d_quote", want.Q), ("d_string", want.S),
                      ("d_leveled", want.LB)):
        np.testing.assert_array_equal(out[name].cpu().numpy().view(np.uint64),
                                      np.asarray(exp).reshape(-1), err_msg=name)
