"""Streams of the lockstep lane: a case that cannot be built, or is refused
after it was built, gives its stream back, and the requests served after it on
the same streams have the bits that they have in a fresh engine."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gridfoam_b200.serving import CavityRequest  # noqa: E402

pytestmark = pytest.mark.gpu


def _engine():
    from gridfoam_b200.serving import BatchedEngine

    eng = BatchedEngine(max_slots=3, max_outer=6, p_tol=1e-30, keep_fields=True)
    eng.prepare((8, 12, 16))
    return eng


def _mix():
    sizes = [8, 16, 12, 8, 12, 16, 8]
    return [CavityRequest(i, n, 50.0 + 40.0 * i, 0.6 + 0.2 * i, 0.0) for i, n in enumerate(sizes)]


@pytest.mark.parametrize("where", ["build", "hook"])
def test_rejected_admissions_give_their_streams_back(where, monkeypatch):
    from gridfoam_b200.algorithms import pressure_velocity

    want = {r.id: r for r in _engine().run(_mix())}
    eng = _engine()
    first = {id(s) for s in eng._streams}
    assert len(first) == 1  # the start-up's cases used one stream in turn
    build = pressure_velocity.create_algorithm
    bad = {2, 5}

    def failing(grid, *a, **k):
        algo = build(grid, *a, **k)
        if where == "build" and any(abs(algo.nu - r.lid / r.re) < 1e-12 for r in _mix() if r.id in bad):
            raise RuntimeError("planted")
        return algo

    def hook(case):
        if where == "hook" and case.req.id in bad:
            raise ValueError("planted")

    monkeypatch.setattr(pressure_velocity, "create_algorithm", failing)
    eng.case_hook = hook
    for _ in range(3):
        got = {r.id: r for r in eng.run(_mix())}
        assert {i for i, r in got.items() if r.status.startswith("rejected")} == bad
        for i in set(want) - bad:
            assert got[i].iterations == want[i].iterations
            np.testing.assert_array_equal(got[i].U, want[i].U)
            np.testing.assert_array_equal(got[i].p, want[i].p)
        # at most as many streams as there are slots, the first one among them
        assert len(eng._streams) <= 3 and first <= {id(s) for s in eng._streams}


def test_a_lone_failing_case_leaves_the_streams_as_they_were(monkeypatch):
    from gridfoam_b200.algorithms import pressure_velocity

    def failing(*a, **k):
        raise RuntimeError("planted")

    eng = _engine()
    before = [id(s) for s in eng._streams]
    with monkeypatch.context() as m:
        m.setattr(pressure_velocity, "create_algorithm", failing)
        (r,) = eng.run(_mix()[:1])
    assert r.status == "rejected: RuntimeError"
    assert [id(s) for s in eng._streams] == before


@pytest.mark.parametrize("free,emptied", [(1 << 20, True), (1 << 33, False)])
def test_a_capture_on_a_full_device_empties_the_allocators_cache(free, emptied, monkeypatch):
    """The allocator cannot give cached blocks back during a capture."""
    eng = _engine()
    calls = []
    empty = torch.cuda.empty_cache
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, 1 << 37))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: (calls.append(1), empty()))
    (r,) = eng.run(_mix()[:1])
    assert r.iterations == 6 and eng.captures > 0
    assert bool(calls) == emptied
