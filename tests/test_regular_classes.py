"""The regular cells of a mesh against a plain numpy restatement, on the CPU."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _restated(h):
    C = h.cell_sizes.shape[0]
    size = h.cell_sizes.min(axis=0)
    out = np.full(C, 255)
    faces: list = [[] for _ in range(C)]
    for f, (o, n) in enumerate(zip(h.owner, h.neighbour)):
        faces[o].append((f, n))
        faces[n].append((f, o))
    dom = np.bincount(h.domain_owner, minlength=C)
    for c in range(C):
        level = int(round(float(np.log2(h.cell_sizes[c, 0] / size[0]))))
        regular = dom[c] == 0 and len(faces[c]) == 6 and np.array_equal(h.cell_sizes[c], size * 2.0**level)
        for f, n in faces[c]:
            want = np.zeros(3)
            want[h.axis[f]] = h.cell_sizes[c, h.axis[f]]
            d = np.abs(h.cell_centers[n] - h.cell_centers[c])
            regular = (regular and not h.immersed[f] and np.array_equal(h.cell_sizes[n], h.cell_sizes[c])
                       and bool(np.all(np.abs(d - want) <= 1e-9 * h.cell_sizes[c].min())))
        if regular:
            out[c] = level
    return size, out


@pytest.mark.parametrize("name", ["cavity", "pipe", "wake", "one layer"])
def test_regular_cells_match_the_restatement(name):
    from gridfoam_b200.cases import build_mesh, cavity_case, cylinder_wake_case, pipe_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = {"cavity": lambda: cavity_case(9), "pipe": lambda: pipe_case(16, 17),
            "wake": lambda: cylinder_wake_case((40, 27, 5)), "one layer": lambda: cavity_case(1)}[name]()
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cpu"),
                             device="cpu")
    size, want = _restated(grid.host)
    assert np.array_equal(grid.dev["reg_level"].numpy(), want)
    assert np.array_equal(grid.dev["irr_cells"].numpy(), np.nonzero(want == 255)[0])
    assert np.allclose(tuple(grid.cmesh.reg_h), size, rtol=0, atol=0)
    assert grid.cmesh.n_irr == int((want == 255).sum())
    if name == "wake":
        assert {0, 2, 255} <= set(want.tolist())  # the finest and the coarsest level have regular cells


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("value,whole_axis", [(0.0, False), (-1.0, False), (float("nan"), False), (float("inf"), False),
                                              (0.0, True), (-1.0, True)])
def test_sizes_without_a_level_are_not_regular(value, whole_axis):
    """A mesh with such sizes was accepted before there were classes."""
    from gridfoam_b200.cases import build_mesh, cavity_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = cavity_case(5)
    mesh = build_mesh(case["mesh"], device="cpu")
    sizes = np.array(mesh.cell_sizes, dtype=np.float64)
    cells = slice(None) if whole_axis else [62]  # the middle cell
    sizes[cells, 0] = value
    mesh.cell_sizes = sizes
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), mesh, device="cpu")
    assert (grid.dev["reg_level"].numpy()[cells] == 255).all()
