"""The kernels a call launches, from the CUDA profiling interface."""

import json
import re


def kernels(call, tmp_path):
    """[(name with its first template arguments, grid, device microseconds)] of
    the kernels that ``call()`` launches, in time order."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    path = tmp_path / "trace.json"
    prof.export_chrome_trace(str(path))
    events = [ev for ev in json.loads(path.read_text())["traceEvents"] if ev.get("cat") == "kernel"]
    out = []
    for ev in sorted(events, key=lambda ev: ev["ts"]):
        m = re.search(r"(k_\w+(?:<[^(]*>)?)\(", ev["name"])
        out.append((m.group(1) if m else ev["name"], tuple(ev["args"]["grid"]), ev["dur"]))
    return out


def resolve_kernels(engine, tmp_path):
    """``kernels()`` of a resolve, repeated (three times at most) where the
    profiler lost a record: the engine counts its launches itself."""
    for _ in range(3):
        out = kernels(engine.resolve, tmp_path)
        if len(out) == engine.timings()["kernel_launches"]:
            break
    return out


def count(launched, prefix):
    """How many of ``kernels()``'s launches carry a name with that prefix."""
    return sum(name.startswith(prefix) for name, _, _ in launched)
