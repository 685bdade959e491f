"""Where the regular cells' own gradient kernel takes over: below that size a
gradient is one launch and has the general path's bits, from there on it is
within the bound of ``test_regular_cells`` (whose derivation holds here too)."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

from tests.test_regular_cells import _general  # noqa: E402

pytestmark = pytest.mark.gpu

LINE = 327680


def _grid(name, size):
    from gridfoam_b200.cases import build_mesh, cylinder_wake_case, pipe_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    if name == "wake":
        case = cylinder_wake_case(size)
    else:
        case = pipe_case(33, 34)
        case["mesh"] |= {"res": list(size), "upper": [n / 64 for n in size]}
        body = case["mesh"]["bodies"][0] | {"center": [size[0] / 128, size[1] / 128], "radius": 0.4 * size[0] / 64}
        case["mesh"]["bodies"] = [body] * (name == "pipe")
    return AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")


@pytest.mark.parametrize("name,size,own", [("box", (64, 64, 79), False), ("box", (64, 64, 80), True),
                                           ("box", (127, 26, 101), True), ("pipe", (55, 55, 55), False),
                                           ("pipe", (71, 69, 70), True), ("wake", (104, 65, 13), False),
                                           ("wake", (116, 74, 14), True)])
def test_gradient_on_both_sides_of_the_line(name, size, own):
    from gridfoam_b200._lib import call, ptr, stream_ptr
    from gridfoam_b200.core.field import CellField
    from gridfoam_b200.fv.fvc import _eval_state

    grid = _grid(name, size)
    assert (grid.num_cells >= LINE) == own and grid.num_cells > 131072
    gen = torch.Generator(device="cuda").manual_seed(1)
    tol = 4 * 2.0**-52 * float(grid.cell_centers.abs().max()) / float(grid.cell_sizes.min())
    for field, shape in (("p", ()), ("U", (3,))):
        f = CellField(grid, field, "local", shape)
        f.data = torch.randn(f.data.shape, generator=gen, dtype=torch.float64, device="cuda")
        _eval_state(f)
        out = []
        for m in (grid.cmesh, _general(grid)):
            g = torch.full((3 * f.num_components, grid.num_cells), float("nan"), dtype=torch.float64, device="cuda")
            call("gf_lsq_grad", ctypes.byref(m), f.num_components, ptr(f.store), ptr(f.table.kind),
                 ptr(f.table.psib), ptr(g), stream_ptr())
            out.append(g)
        if own:
            assert float((out[0] - out[1]).abs().max()) <= tol * float(out[1].abs().max())
        else:
            assert torch.equal(out[0], out[1])
