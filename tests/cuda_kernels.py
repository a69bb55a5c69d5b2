"""The CUDA kernels that a piece of code launched, as the CUDA profiling
interface of PyTorch saw them.  In a process of its own: late in a long one its
records lack kernels."""
import json
import os
import subprocess
import sys
import tempfile
import textwrap
import time
import warnings

import pytest

_HERE = os.path.dirname(os.path.abspath(__file__))
_MARKS = 4      # kernels of PyTorch's own before and after, which show that nothing was lost
_LACKS = 77     # exit status of a process whose record lacks some
_APART = 0.1    # s between the ends of the record and what is recorded: events close to them may be cut off


def _record(run):
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
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as f:
            events = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]
    events.sort(key=lambda e: e["ts"])
    return [(e["name"], e["args"]["registers per thread"]) for e in events]


def kernels(run):
    """[(name, registers per thread), ...] of this library's kernels launched by
    run(), in order of their start."""
    for _ in range(3):   # the first records of a process may lack some
        if len(_record(lambda: None)) == 2 * _MARKS:
            break
    ran = _record(run)
    mine = [k for k in ran if "h3d::" in k[0]]
    if len(ran) - len(mine) < 2 * _MARKS:
        sys.exit(_LACKS)
    return mine


def in_child(body, **env):
    """What `body` leaves in `out`, run by a fresh Python with `env` set, after
    the imports of a GPU test, kernels() among them."""
    code = textwrap.dedent("""\
        import json, os, sys
        sys.path[:0] = [%r, %r, %r]
        import numpy as np
        import torch
        from cuda_kernels import kernels
        from helpers import mode_n_solver, rand_c, small_problem
        """) % (_HERE, os.path.dirname(_HERE), os.path.join(os.path.dirname(_HERE),
                                                            "iterative-helmholtz-solver-with-pardiso_b200"))
    code += textwrap.dedent(body) + "\nprint('OUT' + json.dumps(out))\n"
    kept = {k: v for k, v in os.environ.items() if not k.startswith("HELM3D_")}
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", code], env=dict(kept, **env), capture_output=True, text=True, timeout=300)
        if r.returncode != _LACKS:
            break
    else:
        pytest.skip("no complete record of kernels here")
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(next(ln for ln in r.stdout.splitlines() if ln.startswith("OUT"))[3:])
