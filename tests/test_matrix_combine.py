"""Sums of matrices in one pass, and the time derivative's own assembly,
against the same arithmetic on whole tensors: products by one are exact and
general factors differ by one rounding of each product and of the sum."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

EPS = 2.0**-52


@pytest.fixture(scope="module", params=["box", "pipe", "wake"])
def grid(request):
    from gridfoam_b200.cases import build_mesh, cavity_case, cylinder_wake_case, pipe_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = {"box": lambda: cavity_case(9), "pipe": lambda: pipe_case(16, 17),
            "wake": lambda: cylinder_wake_case((40, 27, 5))}[request.param]()
    return AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")


@pytest.mark.parametrize("shape", [(), (3,)])
def test_one_pass_sum_and_time_derivative(grid, shape):
    from gridfoam_b200.core.field import CellField
    from gridfoam_b200.fv import fvm

    gen = torch.Generator(device="cuda").manual_seed(3)
    f = CellField(grid, "U" if shape else "p", "transient", shape)
    f.data = torch.randn(f.data.shape, generator=gen, dtype=torch.float64, device="cuda")
    # a poisoned allocator: what an operator leaves unwritten shows as NaN
    del_me = [torch.full((grid.ell_width * grid.num_cells,), float("nan"), dtype=torch.float64, device="cuda")
              for _ in range(8)]
    del del_me
    lap, ddt = fvm.laplacian(0.7, f), fvm.ddt(f)

    assert torch.count_nonzero(ddt.val) == 0
    vdt = grid.cell_volumes / grid.dt
    # one division and one product against the same: a rounding each
    assert torch.all((ddt.diag_store - vdt).abs() <= 2 * EPS * vdt.abs())
    old = f.old_store.reshape(-1, grid.num_cells)
    assert torch.all((ddt.source_store - vdt * old).abs() <= 3 * EPS * (vdt * old).abs())

    for a, b in ((1.0, 1.0), (1.0, -1.0), (0.3, 1.7)):
        out = lap._combine(ddt, a, b)
        for name in ("diag_store", "val", "source_store"):
            x, y = getattr(lap, name), getattr(ddt, name)
            bound = 0.0 if (abs(a), abs(b)) == (1.0, 1.0) else 2 * EPS * ((a * x).abs() + (b * y).abs())
            assert torch.all((getattr(out, name) - (a * x + b * y)).abs() <= bound), (name, a, b)
