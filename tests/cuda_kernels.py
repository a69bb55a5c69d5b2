"""The CUDA kernels that a piece of code launched, as the CUDA profiling
interface of PyTorch saw them."""
import json
import time
import warnings

import pytest

_MARKS = 4      # kernels of PyTorch's own before and after, which show that nothing was lost
_APART = 0.1    # s between the ends of the record and what is recorded: events close to them may be cut off


def _record(run, tmp_path):
    import torch
    from torch.profiler import ProfilerActivity, profile
    mark = torch.zeros(1, device="cuda")

    def marks():
        for _ in range(_MARKS):
            mark.add_(1)
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            time.sleep(_APART)
            marks()
            run()
            torch.cuda.synchronize()
            marks()
            time.sleep(_APART)
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]
    events.sort(key=lambda e: e["ts"])
    return [(e["name"], e["args"]["registers per thread"]) for e in events]


def kernels(run, tmp_path):
    """[(name, registers per thread), ...] of this library's kernels launched by
    run(), in order of their start."""
    for _ in range(3):   # the first records of a process may lack some
        if len(_record(lambda: None, tmp_path)) == 2 * _MARKS:
            break
    else:
        pytest.skip("no complete record of kernels here")
    ran = _record(run, tmp_path)
    mine = [k for k in ran if "h3d::" in k[0]]
    if len(ran) - len(mine) < 2 * _MARKS:
        pytest.skip("the record lacks kernels")
    return mine
