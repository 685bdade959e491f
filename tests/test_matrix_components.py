"""Sums, negation, copies and new sources of matrices whose field has another
number of components than one or three, against the same arithmetic on whole
tensors (products by +-1 and 0 of finite values and sums of two are exact to
the one rounding that both sides make)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

STORES = ("diag_store", "val", "source_store")


@pytest.mark.parametrize("shape", [(2,), (3, 3)])
@pytest.mark.parametrize("mesh", ["box", "wake"])
def test_matrix_algebra_takes_any_component_count(shape, mesh):
    from gridfoam_b200.cases import build_mesh, cavity_case, cylinder_wake_case
    from gridfoam_b200.core.field import CellField
    from gridfoam_b200.core.fvmatrix import FvMatrix
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = cavity_case(7) if mesh == "box" else cylinder_wake_case((40, 27, 5))
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")
    # two components: a hand-built system, as BiCGStab takes it
    field = (CellField(grid, "T", "local", shape) if shape == (3, 3)
             else SimpleNamespace(grid=grid, num_components=2, component_shape=shape))
    gen = torch.Generator(device="cuda").manual_seed(4)
    a, b = FvMatrix(field), FvMatrix(field)
    for m in (a, b):
        for name in STORES:
            getattr(m, name).normal_(generator=gen)
    for got, want in ((a + b, lambda x, y: x + y), (a - b, lambda x, y: x - y), (-a, lambda x, y: -x),
                      (a.clone(), lambda x, y: x)):
        for name in STORES:
            assert torch.equal(getattr(got, name), want(getattr(a, name), getattr(b, name))), name
    source = torch.randn(a.source.shape, generator=gen, dtype=torch.float64, device="cuda")
    c = a.with_source(source)
    assert torch.equal(c.source, source) and torch.equal(c.val, a.val) and torch.equal(c.diag_store, a.diag_store)
