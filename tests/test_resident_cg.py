"""CG with the system resident on the grid's SMs against the register kernel.

The systems are ``L + I`` (``L`` a graph Laplacian, so the smallest
eigenvalue is at least 1): two solutions whose residuals are below 1e-11
differ by at most 2e-11 in the 2-norm; twice that is allowed for the rounding
of the recursive residuals."""

from __future__ import annotations

from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _ring(n, reach, long_every):
    """Couplings to +-1 .. +-3 on a ring, and to +-4 .. +-reach between the
    cells whose number divided by 64 is a multiple of ``long_every``: rows of
    six and of 2 reach entries, as at the level interfaces of an octree."""
    c = torch.arange(n, device="cuda")
    width = 2 * reach
    nbr = c.expand(width, n).clone()
    val = torch.zeros((width, n), dtype=torch.float64, device="cuda")
    is_long = (c // 64) % long_every == 0
    slot = 0
    length = torch.full((n,), 6, dtype=torch.uint8, device="cuda")
    for d in range(1, reach + 1):
        for sign in (-1, 1):
            j = (c + sign * d) % n
            on = torch.ones_like(is_long) if d <= 3 else is_long & is_long[j]
            nbr[slot] = torch.where(on, j, c)
            val[slot] = on.to(torch.float64) * (1.0 / d)
            length = torch.where(on, torch.full_like(length, slot + 1), length)
            slot += 1
    s = SimpleNamespace(device=torch.device("cuda"), ell_width=width, box_strides=None,
                        dev={"ell_nbr": nbr.to(torch.int32).contiguous(), "ell_len": length.contiguous()})
    return s, -(val.sum(0) + 1.0), val.contiguous()


def _solve(s, diag, val, rhs, variant, cap, norm="l_2"):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import CGSolver

    solver = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=1e-11, rel_tolerance=0.0,
                                   max_iter=2000, norm_type=norm))
    solver.variant = variant
    solver.block_cap = cap
    x = torch.zeros_like(rhs)
    return x, solver.solve_arrays(s, diag, val, rhs, x)[0]


# cells, block cap: one cell a thread and ragged chunks, two, four and six
# cells a thread; on one block of 3,300 cells the further entries of width 10
# have room for some rows only; 3,300 is the smallest with room for the flags
@pytest.mark.parametrize("n,cap", [(3300, 148), (7177, 9), (6000, 3), (5000, 2), (16385, 6), (80001, 148)])
@pytest.mark.parametrize("reach,long_every", [(3, 1), (4, 3), (5, 1), (5, 2)])
def test_resident_cg_matches_register_kernel(n, cap, reach, long_every):
    s, diag, val = _ring(n, reach, long_every)
    g = torch.Generator(device="cuda").manual_seed(5)
    rhs = torch.randn((1, n), dtype=torch.float64, device="cuda", generator=g)
    x, st = _solve(s, diag, val, rhs, 10, cap)
    ref, st_ref = _solve(s, diag, val, rhs, 0, 148)
    assert st.status == st_ref.status == "ok"
    assert float((x - ref).norm()) < 4e-11


@pytest.mark.parametrize("symmetric", [False, True])
def test_resident_cg_on_boxes_and_infinity_norm(symmetric):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.autotune import BoxSystem
    from gridfoam_b200.solvers.krylov import CGSolver

    s = BoxSystem(37, 41, 43, device=torch.device("cuda"))
    diag = s.diag - 1.0
    out = []
    for variant in (10, 0):
        solver = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=1e-11, rel_tolerance=0.0,
                                       max_iter=2000, norm_type="l_inf"))
        solver.variant = variant
        x = torch.zeros_like(s.rhs)
        st = solver.solve_arrays(s, diag, s.val, s.rhs, x, symmetric=symmetric)[0]
        assert st.status == "ok"
        out.append(x)
    # |r| < 1e-11 in the largest value is |r| < 1e-11 sqrt(n) in the 2-norm
    assert float((out[0] - out[1]).norm()) < 4e-11 * s.num_cells**0.5
