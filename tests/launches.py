"""The kernel launches of a call, as the CUDA profiling interface reports them."""
import json
import os
import re
import tempfile
from collections import namedtuple

import pytest

Launch = namedtuple("Launch", "name args threads blocks registers shared")
_started = False


def _kernels(call):
    """The kernel events of a profiled session around `call`."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    fd, path = tempfile.mkstemp(suffix=".json")
    os.close(fd)
    try:
        prof.export_chrome_trace(path)
        with open(path) as f:
            events = json.load(f)["traceEvents"]
    finally:
        os.unlink(path)
    return sorted((e for e in events if e.get("cat") == "kernel"), key=lambda e: e["ts"])


def launches(call):
    """Runs `call` and returns its launches of this library's kernels in order:
    kernel name, template arguments as texts, threads per block, blocks,
    registers per thread and shared memory per block.  Skips the test where the
    profiling interface reports nothing (another tool may hold it)."""
    import torch
    global _started
    if not _started:  # (a process's first session may miss launches)
        probe = torch.zeros(1, device="cuda")
        _kernels(lambda: probe.add_(1))
        if not _kernels(lambda: probe.add_(1)):
            pytest.skip("no kernel records from the CUDA profiling interface")
        _started = True
    out = []
    for e in _kernels(call):
        m = re.search(r"\b(k_\w+)(?:<([^()]*(?:\(\w+\)[^()]*)*)>)?\(", e["name"])
        if not m:
            continue
        args = [re.sub(r"^\(\w+\)", "", x.strip()) for x in m.group(2).split(",")] if m.group(2) else []
        a = e["args"]
        prod = lambda d: d[0] * d[1] * d[2]  # noqa: E731
        out.append(Launch(m.group(1), args, prod(a["block"]), prod(a["grid"]), a["registers per thread"],
                          a.get("shared memory", 0)))
    return out
