"""Names and CUDA runtime calls of what a function launches, as torch's profiler traces them."""
import pytest
import torch


def trace(fn):
    """{event name: count} of one call of `fn`, after a call that is not traced."""
    from torch.profiler import ProfilerActivity, profile
    fn()
    torch.cuda.synchronize()
    for _ in range(2):  # the first trace of a process starts late
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            fn()
            torch.cuda.synchronize()
        out = {}
        for e in p.events():
            out[e.name] = out.get(e.name, 0) + 1
    if not any('cgb::' in k for k in out):
        pytest.skip('no kernel trace on this machine')
    return out


def ran(fn, *names):
    """Which of the kernels `names` one call of `fn` launches."""
    t = trace(fn)
    return [any('::' + n in k for k in t) for n in names]
