"""The view of a batch reports the query launch that runs: its block and grid,
tuned or not, with every number of lanes per record."""
import json

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _query_launch(run, path):
    run()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    found = [e["args"] for e in json.loads(path.read_text())["traceEvents"]
             if "batch_query_kernel" in e.get("name", "") and "grid" in e.get("args", {})]
    assert len(found) == 1
    return found[0]["grid"][0], found[0]["block"][0]


@pytest.mark.parametrize("tuned", [False, True], ids=["default", "tuned"])
@pytest.mark.parametrize("count", [40, 4000, 9000, 15000, 40000, 170000, 300000])
def test_view_reports_the_launched_grid(gpj, tmp_path, count, tuned):
    data = np.frombuffer(b'{"a":{"b":%d}}\n' % 7 * count, np.uint8)[:-1]
    dev = torch.from_numpy(data.copy()).cuda()
    c = gpj.compile("$.a.b")
    with gpj.Batch(dev.data_ptr(), data.size, [(0, data.size, 0)], [(c, 0, 2)],
                   flags=gpj.GPJ_BATCH_NO_GRAPH | (gpj.GPJ_BATCH_AUTOTUNE if tuned else 0)) as b:
        v = b.view()
        assert v.num_records == count
        assert _query_launch(b.run, tmp_path / "trace.json") == (v.query_grid, v.query_block)
