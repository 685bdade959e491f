"""BiCGStab with strides that no box layout has (rows wider than six slots, or
descending strides) goes by the index table: the same bits as without them."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from tests.test_grid_bicgstab import _system  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout,strides", [("ell8", (23, 23 * 17)), ("ell6", (23 * 17, 23)), ("ell8", (7, 3))])
@pytest.mark.parametrize("cap", [0, 148])  # on a cluster and on the grid
@pytest.mark.parametrize("ncomp", [1, 3])
def test_strides_without_a_box_are_ignored(layout, strides, cap, ncomp):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import BiCGSTABSolver

    s = _system((23, 17, 21), layout)
    g = torch.Generator(device="cuda").manual_seed(3)
    rhs = torch.randn((ncomp, s.num_cells), dtype=torch.float64, device="cuda", generator=g)
    out = []
    for box in (None, strides):
        s.box_strides = box
        solver = BiCGSTABSolver(SolverConfig(method="bicgstab", preconditioner="jacobi", tolerance=1e-11,
                                             rel_tolerance=0.0, max_iter=500))
        solver.block_cap = cap
        x = torch.zeros_like(rhs)
        st = solver.solve_arrays(s, s.diag, s.val, rhs, x)
        assert all(q.status == "ok" for q in st)
        out.append(x)
    assert torch.equal(out[0], out[1])
