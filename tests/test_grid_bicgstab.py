"""Grid BiCGStab against the cluster form and a dense solve.

The systems are ``L + I`` plus a skew part (``L`` the box Laplacian, the
smallest eigenvalue of the symmetric part at least 1), so ``|x - y|`` of two
solutions is at most the sum of their residuals' 2-norms: 2e-11 for residuals
below 1e-11; twice that is allowed for the rounding of the recursions."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# one cell; a block's threads and one more; several cells a thread on few
# blocks; a ragged box; more cells than one pass of the whole grid covers
SHAPES = [(1, 1, 1, 148), (1024, 1, 1, 148), (1025, 1, 1, 148), (16, 16, 32, 3), (37, 29, 41, 148), (54, 53, 55, 148)]


def _system(shape, layout):
    from gridfoam_b200.solvers.autotune import BoxSystem

    s = BoxSystem(*shape, device=torch.device("cuda"))
    s.diag = s.diag - 1.0
    # convection-like skew part: the "+" coefficients up, the "-" ones down
    skew = torch.tensor([-0.3, 0.3] * 3, dtype=torch.float64, device="cuda")[:, None]
    s.val = (s.val * (1.0 + skew)).contiguous()
    if layout != "box":
        s.box_strides = None
    if layout == "ell8":
        n = s.num_cells
        own = torch.arange(n, dtype=torch.int32, device="cuda").expand(2, n)
        s.ell_width = 8
        s.dev["ell_nbr"] = torch.cat([s.dev["ell_nbr"], own]).contiguous()
        s.dev["ell_len"] = torch.full((n,), 6, dtype=torch.uint8, device="cuda")
        s.val = torch.cat([s.val, torch.zeros((2, n), dtype=torch.float64, device="cuda")]).contiguous()
    return s


def _apply(s, x):
    y = s.diag * x
    for k in range(s.ell_width):
        y += s.val[k] * x[:, s.dev["ell_nbr"][k].long()]
    return y


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", ["box", "ell6", "ell8"])
@pytest.mark.parametrize("ncomp,norm", [(1, "l_2"), (2, "l_inf"), (3, "l_2"), (3, "l_inf")])
def test_grid_bicgstab_solves_the_system(shape, layout, ncomp, norm):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver

    s = _system(shape[:3], layout)
    g = torch.Generator(device="cuda").manual_seed(3)
    rhs = torch.randn((ncomp, s.num_cells), dtype=torch.float64, device="cuda", generator=g)
    rhs[-1] *= 1e3  # the components converge at different iterations
    solver = BiCGSTABSolver(SolverConfig(method="bicgstab", preconditioner="jacobi", tolerance=1e-11,
                                         rel_tolerance=0.0, max_iter=500, norm_type=norm))
    solver.block_cap = shape[3]  # a bound on the blocks keeps small solves on the grid
    x = torch.zeros_like(rhs)
    st = solver.solve_arrays(s, s.diag, s.val, rhs, x)
    # the true residual against the recursive one: rounding of a few dozen
    # updates of values up to |b|
    scale = float(rhs.abs().max())
    tol = 4e-11 * (s.num_cells**0.5 if norm == "l_inf" else 1.0) + 1e-13 * scale * s.num_cells**0.5
    r = rhs - _apply(s, x)
    for k in range(ncomp):
        assert st[k].status == "ok" and st[k].iterations < 500
        assert float(r[k].norm()) < tol


def test_grid_bicgstab_restarts_and_gives_up_like_the_cluster_form():
    """An antisymmetric system breaks down at once (r_hat.v = 0); both forms
    use up the permitted restarts and report it."""
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver

    s = _system((64, 1, 1), "ell6")
    s.diag = torch.full_like(s.diag, 1.0)
    s.val = torch.zeros_like(s.val)
    s.val[0, 1::2] = -1e12
    s.val[1, 0::2] = 1e12  # pairs coupled by a rotation, the diagonal lost in rounding
    rhs = torch.ones((3, 64), dtype=torch.float64, device="cuda")
    out = []
    for cap in (0, 148):
        solver = BiCGSTABSolver(SolverConfig(method="bicgstab", preconditioner="jacobi", tolerance=1e-30,
                                             rel_tolerance=0.0, max_iter=50, max_restart=2))
        solver.block_cap = cap
        x = torch.zeros_like(rhs)
        st = solver.solve_arrays(s, s.diag, s.val, rhs, x)
        out.append([(q.status, q.iterations, q.converged) for q in st])
    assert out[0] == out[1] == [("breakdown", 3, False)] * 3
