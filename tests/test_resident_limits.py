"""The largest systems of the on-chip CG forms, one cell on either side.

The form that ran is read from the profiler; bounds of the solutions as derived
in ``test_resident_cg`` and ``test_cluster_krylov``."""

from __future__ import annotations

import re

import pytest

torch = pytest.importorskip("torch")

from tests.test_resident_cg import _ring, _solve  # noqa: E402

pytestmark = pytest.mark.gpu

SIX = r"k_pcg_resident(<6, true>|ILi6ELb1E)"  # the name as written or as linked


def _ran(run, form):
    """``run``'s result and whether a kernel of the form ran."""
    from tests.profiled import lost, record

    names = lambda events: " ".join(key for key, _ in events if "gf::k_" in key or "_ZN2gf" in key)  # noqa: E731
    out, events = record(run, lambda events: re.search(form, names(events)))
    if not names(events):
        lost()
    return out, names(events)


# cells, block cap, wide rows: six cells a thread (chunks of 2,049 to 2,106
# cells) with room for all further entries and for some, and the first chunk
# without room for two a cell
@pytest.mark.parametrize("n,cap,form", [(4098, 2, SIX), (4200, 2, SIX),
                                        (4212, 2, SIX), (4214, 2, "k_pcg1_qrec_ell")])
@pytest.mark.parametrize("reach,long_every", [(4, 3), (5, 1), (5, 2)])
def test_resident_cg_of_six_cells_a_thread_with_wide_rows(n, cap, form, reach, long_every):
    s, diag, val = _ring(n, reach, long_every)
    g = torch.Generator(device="cuda").manual_seed(5)
    rhs = torch.randn((1, n), dtype=torch.float64, device="cuda", generator=g)
    (x, st), kernels = _ran(lambda: _solve(s, diag, val, rhs, 10, cap), form)
    assert re.search(form, kernels), kernels
    ref, st_ref = _solve(s, diag, val, rhs, 0, 148)
    assert st.status == st_ref.status == "ok"
    assert float((x - ref).norm()) < 4e-11


# rows of six: 2,801 cells a block of 16
@pytest.mark.parametrize("shape,form", [((16, 2801, 1), "k_cluster_cg"), ((44817, 1, 1), "k_pcg_resident")])
@pytest.mark.parametrize("layout", ["box", "sym", "ell6"])
def test_cluster_cg_at_its_largest_system(shape, form, layout):
    from tests.test_cluster_krylov import _solve as solve
    from tests.test_cluster_krylov import _system

    s = _system(shape, layout)
    g = torch.Generator(device="cuda").manual_seed(7)
    rhs = torch.randn((1, s.num_cells), dtype=torch.float64, device="cuda", generator=g)
    (x, st), kernels = _ran(lambda: solve(s, "cg", rhs, False, "l_2", layout), form)
    assert re.search(form, kernels), kernels
    ref, st_ref = solve(s, "cg", rhs, True, "l_2", layout)
    assert st[0].status == st_ref[0].status == "ok"
    assert float((x[0] - ref[0]).norm()) < 4e-11
