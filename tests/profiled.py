"""What a call launches and which CUDA runtime functions it uses, from torch's profiler."""
import json
import os
import tempfile
import time


def profiled(call):
    """(the call's result, {name: count} of kernels, copies and runtime calls, the kernels' records).
    The margins on both sides keep the call's records inside the profiler's window, whose GPU and host
    clocks differ; a kernel in each shows that it was open."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    x = torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        for part in ("before", "call", "after"):
            if part == "call":
                out = call()
            else:
                x.add_(1)
                torch.cuda.synchronize()
                time.sleep(0.05)
                x.add_(1)
            torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        p.export_chrome_trace(path)
        with open(path) as f:
            events = json.load(f)["traceEvents"]
    kernels = [e for e in events if e.get("cat") == "kernel"]
    assert any("elementwise" in e["name"] for e in kernels), "the profiler's window was not open"
    counts = {}
    for e in events:
        if e.get("cat") in ("kernel", "gpu_memcpy", "gpu_memset", "cuda_runtime", "cuda_driver"):
            counts[e["name"]] = counts.get(e["name"], 0) + 1
    return out, counts, [e for e in kernels if "uegccd" in e["name"]]
