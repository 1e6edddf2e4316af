"""The kernels a call launches, as torch's profiler records them."""
import json
import tempfile
import time
from pathlib import Path

import torch


def launches(run, name):
    """{(kernel name, grid x, block x)} of the kernels with `name` in theirs.

    The profiler drops records that its clock puts outside the profiled span,
    most easily late in a long process: the call runs several times, away from
    the span's ends, and again where nothing was recorded."""
    run()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA],
                                    acc_events=True) as prof:
            time.sleep(0.05)
            for _ in range(8):
                run()
                torch.cuda.synchronize()
                time.sleep(0.005)
            time.sleep(0.05)
        with tempfile.TemporaryDirectory() as tmp:
            path = Path(tmp) / "trace.json"
            prof.export_chrome_trace(str(path))
            events = json.loads(path.read_text())["traceEvents"]
        found = {(e["name"], e["args"]["grid"][0], e["args"]["block"][0]) for e in events
                 if name in e.get("name", "") and "grid" in e.get("args", {})}
        if found:
            return found
    raise AssertionError("the profiler recorded no kernel")
