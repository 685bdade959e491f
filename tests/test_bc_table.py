"""A boundary table whose kinds need no values (no condition, slip, fixed flux
pressure) may come without them: the same state as with values that are there."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,shape", [("p", ()), ("U", (3,))])
def test_state_of_kinds_without_values(name, shape):
    from gridfoam_b200._lib import GfBc, call, ptr, stream_ptr
    from gridfoam_b200.cases import build_mesh, pipe_case
    from gridfoam_b200.core.field import CellField
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = pipe_case(11, 12)
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")
    f = CellField(grid, name, "local", shape)
    gen = torch.Generator(device="cuda").manual_seed(1)
    f.data = torch.randn(f.data.shape, generator=gen, dtype=torch.float64, device="cuda")
    t = f.table
    # none, slip and fixed flux pressure in turn
    t.kind.copy_(torch.tensor([0, 3, 5], dtype=torch.int8, device="cuda").repeat(grid.num_bnd)[: grid.num_bnd])
    out = []
    for value in (torch.randn(t.refv.shape, generator=gen, dtype=torch.float64, device="cuda"), None):
        bc = GfBc()
        bc.ncomp, bc.kind, bc.value = f.num_components, ptr(t.kind), ptr(value)
        for a in (t.frac, t.refv, t.refg, t.psib):
            a.fill_(float("nan"))
        call("gf_bc_state", ctypes.byref(grid.cmesh), ctypes.byref(bc), ptr(f.store), None, ctypes.byref(t.cstate),
             stream_ptr())
        out.append([a.clone() for a in (t.frac, t.refv, t.refg, t.psib)])
    for a, b in zip(*out):
        assert torch.equal(a, b) and not bool(b.isnan().any())
