"""Kernels that a call launches, by the profiler, for the tests that say which
kernel form ran or how many."""

from __future__ import annotations

import time

import pytest


def record(run):
    """``(result of run, [(kernel name, launches)])``.

    The profiler drops what lies before its own start by its converted clock,
    and a clock that is off by a fraction of a millisecond takes the first
    kernels of a short run with it.  So ``run`` stands between two marks, with
    a pause on either side, and a record that lacks a mark is taken again."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    for pause in (0.02, 0.2, 2.0):
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            time.sleep(pause)
            torch.cuda._sleep(1000)
            out = run()
            torch.cuda._sleep(1000)
            torch.cuda.synchronize()
            time.sleep(pause)
        events = [(e.key, e.count) for e in prof.key_averages()]
        if sum(n for key, n in events if "spin_kernel" in key) == 2:
            return out, [(key, n) for key, n in events if "spin_kernel" not in key]
    pytest.skip("the profiler's record is not whole on this machine")
