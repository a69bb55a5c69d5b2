"""The CUDA kernels that a piece of code launched, as the CUDA profiling
interface of PyTorch saw them."""
import json
import warnings

import pytest


def kernels(run, tmp_path):
    """[(name, registers per thread), ...] of the kernels launched by run(), in order of their start."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            run()
            torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]
    if not events:
        pytest.skip("no CUDA profiling interface here")
    events.sort(key=lambda e: e["ts"])
    return [(e["name"], e["args"]["registers per thread"]) for e in events]
