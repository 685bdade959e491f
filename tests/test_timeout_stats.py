"""A solve whose first wait ran out reports no convergence and no residual.

A solve of a zero right-hand side runs first on the same blocks: its sums are
zeros, and a kernel that took what is left of them for its own would report a
residual of zero, and convergence, beside the timeout."""

from __future__ import annotations

import math

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _box(size):
    from gridfoam_b200.solvers.autotune import BoxSystem

    s = BoxSystem(*size, device=torch.device("cuda"))
    return s, s.diag - 1.0, s.val


def _wide(n):
    from tests.test_resident_cg import _ring

    return _ring(n, 5, 2)


# register form, halo form, rows and vectors on the SMs (box and long rows, FP64
# and FP32-inner), q-recurrence, grid BiCGStab of one and three components
@pytest.mark.parametrize("system,size", [(_box, (24, 24, 48)), (_wide, 27648)])
@pytest.mark.parametrize("method,variant,precision,ncomp", [
    ("cg", 0, "float64", 1), ("cg", 8, "float64", 1), ("cg", 10, "float64", 1), ("cg", 11, "float64", 1),
    ("cg", 10, "float32", 1), ("bicgstab", None, "float64", 1), ("bicgstab", None, "float64", 3)])
def test_a_timeout_is_not_convergence(system, size, method, variant, precision, ncomp):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver, CGSolver

    s, diag, val = system(size)
    n = s.val.shape[1] if hasattr(s, "val") else val.shape[1]
    rhs = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda").expand(ncomp, n).contiguous()
    zero = torch.zeros_like(rhs)
    cls = CGSolver if method == "cg" else BiCGSTABSolver
    cfg = SolverConfig(method=method, preconditioner="jacobi", tolerance=1e-10, rel_tolerance=0.0, max_iter=500,
                       inner_precision=precision)
    timeouts = 0
    for _ in range(20):
        full = cls(cfg)
        full.variant, full.block_cap = variant, 148  # a bound on the blocks keeps it on the grid
        st = full.solve_arrays(s, diag, val, zero, torch.zeros_like(rhs))
        assert all(q.converged and q.initial_residual == 0.0 for q in st)
        short = cls(cfg)
        short.variant, short.block_cap, short.spin_limit = variant, 148, 1
        x = torch.zeros_like(rhs)
        st = short.solve_arrays(s, diag, val, rhs, x)
        for q in st:
            if q.status == "timeout":
                timeouts += 1
                assert not q.converged
                assert not 0.0 < q.initial_residual < 1e-3
                assert math.isnan(q.final_residual) or q.final_residual == 0.0 or q.final_residual > 1e-10
        # the next solve on the stream runs normally
        st = full.solve_arrays(s, diag, val, rhs, torch.zeros_like(rhs))
        assert all(q.status == "ok" and q.converged for q in st)
    assert timeouts > 0
