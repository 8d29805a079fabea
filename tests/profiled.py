"""What a call launches and which CUDA runtime functions it uses, from torch's profiler."""
import json
import os
import tempfile


def profiled(call, complete=lambda counts, kernels: True, tries=6):
    """(the call's result, {name: count} of kernels, copies and runtime calls, the kernels' records).
    The profiler always records the runtime calls, but in a process of some minutes it loses the first
    GPU records (kernels, copies) of a window: copies and kernels of no interest go first, and the call
    is made again, at most `tries` times, until complete(counts, kernels) says that what the test
    needs was recorded.  Where it records nothing (another profiler has the GPU), the test is
    skipped."""
    import pytest
    import torch
    from torch.profiler import ProfilerActivity, profile, record_function

    x, host = torch.zeros(64, device="cuda"), torch.zeros(64)
    for _ in range(tries):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            for _ in range(50):
                x.copy_(host)
                x.add_(1)
                x.cpu()
            torch.cuda.synchronize()
            with record_function("the call"):
                out = call()
                torch.cuda.synchronize()
        with tempfile.TemporaryDirectory() as d:
            path = os.path.join(d, "trace.json")
            p.export_chrome_trace(path)
            with open(path) as f:
                events = json.load(f)["traceEvents"]
        span = next(e for e in events if e.get("cat") == "user_annotation" and e["name"] == "the call")
        runtime = [e for e in events if e.get("cat") in ("cuda_runtime", "cuda_driver")
                   and span["ts"] <= e["ts"] <= span["ts"] + span["dur"]]
        ids = {e["args"]["correlation"] for e in runtime}
        gpu = [e for e in events if e.get("cat") in ("kernel", "gpu_memcpy", "gpu_memset")
               and e["args"].get("correlation") in ids]
        kernels = [e for e in gpu if e["cat"] == "kernel" and "uegccd" in e["name"]]
        counts = {}
        for e in runtime + gpu:
            counts[e["name"]] = counts.get(e["name"], 0) + 1
        if complete(counts, kernels):
            break
    else:
        if not gpu:
            pytest.skip("the profiler lost the GPU's records")
    if not runtime:
        pytest.skip("the profiler records no CUDA calls")
    return out, counts, kernels
