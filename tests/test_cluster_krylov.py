"""Krylov solves on one thread-block cluster against the grid kernels.

The systems are ``L + I`` (L the box Laplacian, so the smallest eigenvalue is
at least 1): two solutions whose residuals are below 1e-11 differ by at most
2e-11 in the 2-norm; the tests allow twice that for the rounding of the
recursive residuals."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# one cell; one block full and one cell more; 16 blocks at one, two and eight
# cells a thread; a ragged shape; the largest systems and the first ones beyond
SHAPES = [(1, 1, 1), (16, 16, 1), (257, 1, 1), (16, 16, 16), (4097, 1, 1), (23, 17, 21), (32, 32, 32),
          (32769, 1, 1), (43, 31, 32), (45057, 1, 1)]


def _system(shape, layout):
    from gridfoam_b200.solvers.autotune import BoxSystem

    s = BoxSystem(*shape, device=torch.device("cuda"))
    s.diag = s.diag - 1.0
    if layout.startswith("ell"):
        s.box_strides = None
    if layout == "ell8":  # two unused slots behind rows of six
        n = s.num_cells
        own = torch.arange(n, dtype=torch.int32, device="cuda").expand(2, n)
        s.ell_width = 8
        s.dev["ell_nbr"] = torch.cat([s.dev["ell_nbr"], own]).contiguous()
        s.dev["ell_len"] = torch.full((n,), 6, dtype=torch.uint8, device="cuda")
        s.val = torch.cat([s.val, torch.zeros((2, n), dtype=torch.float64, device="cuda")]).contiguous()
    return s


def _solve(s, method, rhs, grid_kernels, norm, layout):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver, CGSolver

    cfg = SolverConfig(method=method, preconditioner="jacobi", tolerance=1e-11, rel_tolerance=0.0, max_iter=2000,
                       norm_type=norm)
    solver = (CGSolver if method == "cg" else BiCGSTABSolver)(cfg)
    solver.variant = 0 if grid_kernels else 10
    solver.block_cap = 148 if grid_kernels else 0  # a bound on the blocks keeps the solve on the grid
    x = torch.zeros_like(rhs)
    return x, solver.solve_arrays(s, s.diag, s.val, rhs, x, symmetric=layout == "sym")


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout,norm", [("box", "l_2"), ("sym", "l_inf"), ("ell6", "l_2"), ("ell8", "l_2")])
@pytest.mark.parametrize("method,ncomp", [("cg", 1), ("bicgstab", 1), ("bicgstab", 3)])
def test_cluster_solve_matches_grid_kernels(shape, layout, norm, method, ncomp):
    s = _system(shape, layout)
    g = torch.Generator(device="cuda").manual_seed(7)
    rhs = torch.randn((ncomp, s.num_cells), dtype=torch.float64, device="cuda", generator=g)
    x, st = _solve(s, method, rhs, False, norm, layout)
    ref, st_ref = _solve(s, method, rhs, True, norm, layout)
    # |r| < 1e-11 in the largest value is |r| < 1e-11 sqrt(n) in the 2-norm
    tol = 4e-11 * (s.num_cells**0.5 if norm == "l_inf" else 1.0)
    for k in range(ncomp):
        assert st[k].status == st_ref[k].status == "ok"
        assert float((x[k] - ref[k]).norm()) < tol


def test_cluster_solve_ends_with_the_right_status():
    """A zero right-hand side, the iteration limit and a NaN."""
    s = _system((16, 16, 16), "box")
    zero = torch.zeros((1, s.num_cells), dtype=torch.float64, device="cuda")
    one = torch.ones_like(zero)
    one[0, 0] = 2.0
    bad = one.clone()
    bad[0, 5] = float("nan")
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver, CGSolver

    for cls, method in ((CGSolver, "cg"), (BiCGSTABSolver, "bicgstab")):
        cfg = dict(method=method, preconditioner="jacobi", rel_tolerance=0.0)
        for rhs, tol, limit, want in ((zero, 1e-12, 50, ("ok", 0, True)), (one, 1e-30, 3, ("max_iter", 3, False)),
                                      (one, 1e-30, 0, ("max_iter", 0, False)),
                                      (bad, 1e-12, 50, ("nonfinite", 0, False))):
            solver = cls(SolverConfig(tolerance=tol, max_iter=max(limit, 1), **cfg))
            solver.max_iter = limit
            x = torch.zeros_like(rhs)
            st = solver.solve_arrays(s, s.diag, s.val, rhs, x)[0]
            assert (st.status, st.iterations, st.converged) == want


def test_cluster_solve_under_stream_capture():
    """A captured solve replays on new right-hand sides with the same bits."""
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import CGSolver

    s = _system((16, 16, 16), "box")
    solver = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=1e-11, rel_tolerance=0.0))
    rhs = s.rhs.clone()
    x = torch.zeros_like(rhs)
    solver.solve_arrays(s, s.diag, s.val, rhs, x)
    solver.host_stats = False
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solver.solve_arrays(s, s.diag, s.val, rhs, x)
    for seed in (1, 2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rhs.normal_(generator=g)
        x.zero_()
        graph.replay()
        want = torch.zeros_like(rhs)
        solver.solve_arrays(s, s.diag, s.val, rhs, want)
        assert torch.equal(x, want)
