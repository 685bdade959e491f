"""Kernels that a call launches, by the profiler, for the tests that say which
kernel form ran or how many."""

from __future__ import annotations

import time

import pytest

TRIES = 20


def record(run, whole):
    """``(result of run, [(kernel name, launches)])``, the record taken again
    until ``whole(record)`` holds, ``TRIES`` times at most.

    The profiler loses records: those before its own start by its converted
    clock, which takes the first kernels of a short run with it when the clock
    is off by a fraction of a millisecond, and in a process that has run for
    minutes also single ones in between, of a graph loop's kernels above all.
    It never invents one.  So ``run`` stands between two marks with pauses on
    either side, a record without a mark does not count, and a caller that
    finds fewer kernels than it expects says ``lost``."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    last = None
    for k in range(TRIES):
        pause = 0.01 if k < 10 else 0.2
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            time.sleep(pause)
            torch.cuda._sleep(1000)
            out = run()
            torch.cuda._sleep(1000)
            torch.cuda.synchronize()
            time.sleep(pause)
        events = [(e.key, e.count) for e in prof.key_averages()]
        if sum(n for key, n in events if "spin_kernel" in key) == 2:
            last = out, [(key, n) for key, n in events if "spin_kernel" not in key]
            if whole(last[1]):
                return last
    return last if last is not None else lost()


def lost():
    pytest.skip("the profiler loses records on this machine")
