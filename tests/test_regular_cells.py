"""Kernels that take a regular cell's geometry from its level against the
general path (the same mesh without the classification), and the gradient at
the hanging cells against the full one.

The general path takes distances as differences of cell centres: with centres
up to X and cells of size h they carry a rounding of at most 2^-52 X / h,
relative; the tests allow four times that (three differences meet in a sum)."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _grid(name):
    from gridfoam_b200.cases import build_mesh, cylinder_wake_case, pipe_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    if name == "wake":
        case = cylinder_wake_case((80, 54, 10))
    else:
        case = pipe_case(33, 34)
        case["mesh"] |= {"res": [51, 53, 55], "upper": [51 / 64, 53 / 64, 55 / 64]}
        case["mesh"]["bodies"] = [case["mesh"]["bodies"][0] | {"center": [0.4, 0.41], "radius": 0.3}] * (name == "pipe")
    grid = AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")
    assert grid.num_cells >= 131072  # the size from which the regular cells get their own path
    return grid


@pytest.fixture(scope="module", params=["box", "pipe", "wake"])
def setting(request):
    from gridfoam_b200.core.field import CellField
    from gridfoam_b200.fv.fvc import _eval_state

    grid = _grid(request.param)
    gen = torch.Generator(device="cuda").manual_seed(1)
    fields = []
    for name, shape in (("p", ()), ("U", (3,))):
        f = CellField(grid, name, "local", shape)
        f.data = torch.randn(f.data.shape, generator=gen, dtype=torch.float64, device="cuda")
        _eval_state(f)
        fields.append(f)
    h = float(grid.cell_sizes.min())
    tol = 4 * 2.0**-52 * float(grid.cell_centers.abs().max()) / h
    return grid, fields, tol


def _general(grid):
    """The mesh without its classification of cells."""
    from gridfoam_b200._lib import GfMesh

    m = GfMesh()
    ctypes.pointer(m)[0] = grid.cmesh
    m.reg_level = None
    m.hang_cells = None
    return m


def test_classification(setting):
    """A regular cell has six neighbours of its own size; the rest are listed."""
    grid, _, _ = setting
    level = grid.dev["reg_level"].cpu()
    irr = grid.dev["irr_cells"].cpu().long()
    assert torch.equal(irr, torch.nonzero(level == 255).reshape(-1))
    assert 0 < irr.numel() < grid.num_cells
    sizes = grid.cell_sizes.cpu()
    W, C = grid.ell_width, grid.num_cells
    nbr = grid.dev["ell_nbr"].cpu().long().reshape(W, C)
    reg = torch.nonzero(level != 255).reshape(-1)
    for s in range(6):
        assert torch.equal(sizes[reg], sizes[nbr[s, reg]])
        d = grid.cell_centers.cpu()[nbr[s, reg]] - grid.cell_centers.cpu()[reg]
        want = torch.zeros_like(d)
        want[:, s // 2] = (2 * (s % 2) - 1) * sizes[reg, s // 2]
        assert float((d - want).abs().max()) < 1e-9


def test_gradient_matches_general_path(setting):
    from gridfoam_b200._lib import call, ptr, stream_ptr

    grid, fields, tol = setting
    for f in fields:
        out = []
        for m in (grid.cmesh, _general(grid)):
            g = torch.full((3 * f.num_components, grid.num_cells), float("nan"), dtype=torch.float64, device="cuda")
            call("gf_lsq_grad", ctypes.byref(m), f.num_components, ptr(f.store), ptr(f.table.kind),
                 ptr(f.table.psib), ptr(g), stream_ptr())
            out.append(g)
        scale = float(out[1].abs().max())
        assert float((out[0] - out[1]).abs().max()) <= tol * scale


def test_hanging_gradient_matches_general_path(setting):
    from gridfoam_b200._lib import call, ptr, stream_ptr

    grid, fields, _ = setting
    if grid.num_hanging == 0:
        pytest.skip("no hanging faces")
    cells = grid.dev["hang_cells"].long()
    for f in fields:
        out = []
        for m in (grid.cmesh, _general(grid)):
            g = torch.full((3 * f.num_components, grid.num_cells), float("nan"), dtype=torch.float64, device="cuda")
            call("gf_lsq_grad_hang", ctypes.byref(m), f.num_components, ptr(f.store), ptr(f.table.kind),
                 ptr(f.table.psib), ptr(g), stream_ptr())
            out.append(g)
        assert torch.equal(out[0][:, cells], out[1][:, cells])
        other = torch.ones(grid.num_cells, dtype=torch.bool, device="cuda")
        other[cells] = False
        assert bool(out[0][:, other].isnan().all()) and not bool(out[1].isnan().any())


def test_divergence_of_unit_fluxes_counts_faces(setting):
    """fvc.div against a sum over faces in plain torch."""
    from gridfoam_b200.core.field import FaceField
    from gridfoam_b200.fv import fvc

    grid, _, _ = setting
    gen = torch.Generator(device="cuda").manual_seed(2)
    phi = FaceField(grid, "phi_div")
    phi.store.normal_(generator=gen)
    F, C = grid.num_internal_faces, grid.num_cells
    inner = phi.store[0, :F] * ~grid.ap_is_immersed_faces  # an immersed face enters by its two sides
    bnd_cell = grid.dev["bnd_cell"].long()
    total = torch.zeros(C, dtype=torch.float64, device="cuda")
    total.index_add_(0, grid.owner, inner).index_add_(0, grid.neighbour, -inner)
    total.index_add_(0, bnd_cell, phi.store[0, F:])
    # sums of at most twelve values of size one in another order
    assert float((fvc.div(phi).data * grid.cell_volumes - total).abs().max()) < 12 * 12 * 2.0**-52 * 6


def test_face_values_match_plain_torch(setting):
    """fvc.interpolate and fvc.sn_grad on the faces that are not hanging."""
    from gridfoam_b200.fv import fvc

    grid, (p, U), _ = setting
    F = grid.num_internal_faces
    plain = ~grid.ap_is_immersed_faces
    if grid.num_hanging:
        plain = plain.clone()
        plain[grid.dev["hang_face"].long()] = False
    w, delta = grid.dev["weight"], grid.dev["delta"]
    for f in (p, U):
        po, pn = f.store[:, grid.owner], f.store[:, grid.neighbour]
        v = fvc.interpolate(f).store
        want = w * po + (1.0 - w) * pn
        assert float((v[:, :F] - want)[:, plain].abs().max()) < 4 * 2.0**-52 * float(want.abs().max())
        assert bool((v[:, :F][:, grid.ap_is_immersed_faces] == 0).all())
        assert torch.equal(v[:, F:], f.table.psib)
        g = fvc.sn_grad(f).store[:, :F]
        want = delta * (pn - po)
        assert float((g - want)[:, plain].abs().max()) < 4 * 2.0**-52 * float(want.abs().max())
