"""Operators whose matrices start as unset memory write every entry: the same
matrices from a poisoned allocator as from a cleared one."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _poison(grid, value):
    """Blocks of the sizes of a matrix's arrays, filled and given back."""
    n = grid.num_cells
    del_me = [torch.full((k * n,), value, dtype=torch.float64, device="cuda") for k in (1, 3, grid.ell_width)
              for _ in range(6)]
    del del_me


@pytest.fixture(scope="module", params=["box", "pipe", "wake"])
def mesh(request):
    from gridfoam_b200.cases import build_mesh, cavity_case, cylinder_wake_case, pipe_case

    case = {"box": lambda: cavity_case(9), "pipe": lambda: pipe_case(16, 17),
            "wake": lambda: cylinder_wake_case((40, 27, 5))}[request.param]()
    return case, build_mesh(case["mesh"], device="cuda")


@pytest.mark.parametrize("shape", [(), (3,)])
@pytest.mark.parametrize("scheme", ["upwind", "linear", "vanleer", "minmod"])
def test_operators_write_every_entry(mesh, shape, scheme):
    from gridfoam_b200.core.field import CellField, FaceField
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.fv import fvm
    from gridfoam_b200.meta.config import SimulatorConfig

    case, m = mesh
    case["simulator"]["fvSchemes"]["divSchemes"] = {"default": scheme}
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), m, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    f = CellField(grid, "U" if shape else "p", "transient", shape)
    f.data = torch.randn(f.data.shape, generator=gen, dtype=torch.float64, device="cuda")
    phi = FaceField(grid, "phi")
    phi.store.normal_(generator=gen)
    gamma = torch.rand(grid.num_cells, generator=gen, dtype=torch.float64, device="cuda") + 0.5
    for op in (lambda: fvm.div(phi, f), lambda: fvm.laplacian(gamma, f), lambda: fvm.laplacian(0.3, f),
               lambda: fvm.ddt(f), lambda: fvm.ddt(f) + fvm.div(phi, f) - fvm.laplacian(0.3, f)):
        out = []
        for value in (float("nan"), 0.0):
            _poison(grid, value)
            out.append(op())
        for name in ("diag_store", "val", "source_store"):
            a, b = getattr(out[0], name), getattr(out[1], name)
            assert not bool(a.isnan().any()) and torch.equal(a, b), (name, scheme)
