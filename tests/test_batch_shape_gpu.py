"""The view of a batch reports the query launch that runs: its block and grid,
tuned or not, with every number of lanes per record."""
import numpy as np
import pytest
import torch

from kernel_trace import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned", [False, True], ids=["default", "tuned"])
@pytest.mark.parametrize("count", [40, 4000, 9000, 15000, 40000, 170000, 300000])
def test_view_reports_the_launched_grid(gpj, count, tuned):
    data = np.frombuffer(b'{"a":{"b":%d}}\n' % 7 * count, np.uint8)[:-1]
    dev = torch.from_numpy(data.copy()).cuda()
    c = gpj.compile("$.a.b")
    with gpj.Batch(dev.data_ptr(), data.size, [(0, data.size, 0)], [(c, 0, 2)],
                   flags=gpj.GPJ_BATCH_NO_GRAPH | (gpj.GPJ_BATCH_AUTOTUNE if tuned else 0)) as b:
        v = b.view()
        assert v.num_records == count
        got = launches(b.run, "batch_query_kernel")
        assert {(grid, block) for _, grid, block in got} == {(v.query_grid, v.query_block)}
