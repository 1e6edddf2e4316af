"""Array indexes far into an array, forward and from the end, in every split of
the query kernel: dense arrays (several commas a bitmap word), elements longer
than a round of words, arrays that end early, and broken ones, against the
oracle."""
import random

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

QUERIES = ["$.arr[%s]" % i for i in ("0", "1", "63", "64", "150", "400", "-1", "-2", "-64", "-150",
                                     "-400", "-3:", "62:66", "5,2,90,3")] + ["$[7]", "$[-7]"]


def _line(rng):
    r = rng.random()
    n = rng.choice([0, 1, 2, 63, 64, 65, 151, 399, 401])
    if r < 0.5:
        body = ("," + " " * rng.randint(0, 2)).join(str(rng.randint(0, 9)) for _ in range(n))
    elif r < 0.7:
        body = ",".join('"%s"' % ("x" * rng.choice([0, 5, 60, 130, 2100])) for _ in range(n % 70))
    elif r < 0.8:
        body = "," * n
    else:
        body = ",".join('{"k":[%d,1]}' % i for i in range(n))
    if r > 0.95:  # not closed, closed twice, or cut by another closing bracket
        return '{"arr":[' + body + rng.choice(["", "]]", "}", "}]", ",", "]}}", ":1]}"])
    if 0.78 < r < 0.8:
        return "[" + body + "]"
    return rng.choice(['{"a":1,"arr":[%s],"z":[1,2]}', '{"arr":[%s]}', '{"arr" : [ %s ] }']) % body


@pytest.mark.parametrize("count", [60, 5000, 10000, 20000], ids=["32", "16", "8", "1"])
@pytest.mark.parametrize("base_level", [0, 1])
def test_index_steps_match_oracle(cuda_ctx, gpj, count, base_level):
    rng = random.Random(count)
    pool = [_line(rng) for _ in range(300)]
    data = np.frombuffer("\n".join(rng.choice(pool) for _ in range(count)).encode(), np.uint8)
    comp = [gpj.compile(q) for q in QUERIES]
    levels = max(c.max_depth for c in comp) + base_level
    dev = torch.from_numpy(data.copy()).cuda()
    want_ix = oracle.OracleIndex(data, levels)
    ix = cuda_ctx.build_index(dev.data_ptr(), data.size, levels)
    try:
        assert ix.num_lines == count
        for c in comp[::1 if count < 10000 else 4]:
            out = torch.full((count, c.num_result_slots, 2), -7, dtype=torch.int32, device="cuda")
            cuda_ctx.query(ix, c, out.data_ptr(), base_level=base_level)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(
                out.cpu().numpy().astype(np.int64),
                want_ix.query(c.ir_bytes, c.num_result_slots, base_level), err_msg=c.query_text)
    finally:
        cuda_ctx.free_index(ix)
