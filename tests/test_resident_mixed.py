"""FP32-inner CG with the system resident on the grid's SMs against the FP64
register kernel.  Systems ``L + I`` as in ``test_resident_cg``: the FP64
residuals of both solutions are below 1e-9, so they differ by at most 2e-9 in
the 2-norm; twice that is allowed for rounding."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from tests.test_resident_cg import _ring  # noqa: E402

pytestmark = pytest.mark.gpu


def _solve(s, diag, val, rhs, variant, cap, precision, symmetric=False, norm="l_2"):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import CGSolver

    solver = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=1e-9, rel_tolerance=0.0,
                                   max_iter=2000, norm_type=norm, inner_precision=precision))
    solver.variant = variant
    solver.block_cap = cap
    x = torch.zeros_like(rhs)
    return x, solver.solve_arrays(s, diag, val, rhs, x, symmetric=symmetric)[0]


# cells, block cap: one, two, four and five cells a thread, ragged chunks;
# 16,384 is the smallest with room for the flags; 16,383 cells and six cells a
# thread take the form before
@pytest.mark.parametrize("n,cap", [(16383, 148), (16384, 148), (16385, 17), (16387, 9), (16385, 7), (16385, 6), (80001, 148)])
@pytest.mark.parametrize("reach,long_every", [(3, 1), (4, 3), (5, 1), (5, 2)])
def test_resident_mixed_cg_matches_fp64(n, cap, reach, long_every):
    s, diag, val = _ring(n, reach, long_every)
    g = torch.Generator(device="cuda").manual_seed(6)
    rhs = torch.randn((1, n), dtype=torch.float64, device="cuda", generator=g)
    x, st = _solve(s, diag, val, rhs, 10, cap, "float32")
    ref, st_ref = _solve(s, diag, val, rhs, 0, 148, "float64")
    assert st.status == st_ref.status == "ok"
    assert float((x - ref).norm()) < 4e-9


@pytest.mark.parametrize("symmetric", [False, True])
def test_resident_mixed_cg_on_boxes_and_infinity_norm(symmetric):
    from gridfoam_b200.solvers.autotune import BoxSystem

    s = BoxSystem(37, 41, 43, device=torch.device("cuda"))
    diag = s.diag - 1.0
    x, st = _solve(s, diag, s.val, s.rhs, 10, 0, "float32", symmetric, "l_inf")
    ref, st_ref = _solve(s, diag, s.val, s.rhs, 0, 0, "float64", symmetric, "l_inf")
    assert st.status == st_ref.status == "ok"
    # |r| < 1e-9 in the largest value is |r| < 1e-9 sqrt(n) in the 2-norm
    assert float((x - ref).norm()) < 4e-9 * s.num_cells**0.5
