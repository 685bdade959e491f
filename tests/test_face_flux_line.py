"""Face fluxes on octrees on both sides of the size from which the internal
faces get a kernel of their own: one kernel below, two from there on, and the
general kernel's bits."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

from tests.test_launch_count import _grid  # noqa: E402

pytestmark = pytest.mark.gpu

LINE = 655360  # internal faces


@pytest.mark.parametrize("size,kernels", [((40, 27, 5), 1), ((92, 60, 12), 1), ((96, 62, 12), 2), ((116, 74, 14), 2)])
@pytest.mark.parametrize("ddt", [False, True])
def test_octree_face_flux(size, kernels, ddt):
    from gridfoam_b200._lib import GfDdtCorr, GfMesh, call, ptr, stream_ptr
    from gridfoam_b200.core.field import CellField, FaceField
    from gridfoam_b200.fv.fvc import _eval_state, _hanging_grad
    from tests.profiled import lost, record

    grid = _grid("wake", size)
    F = grid.num_internal_faces
    assert (F >= LINE) == (kernels == 2)
    gen = torch.Generator(device="cuda").manual_seed(2)
    rand = lambda *n: torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")  # noqa: E731
    U = CellField(grid, "U", "local", (3,))
    U.data = rand(*U.data.shape)
    _eval_state(U)
    grad, t, d = _hanging_grad(U), U.table, None
    if ddt:
        keep = rau, u_old, u_older, phi_old, phi_older = (rand(grid.num_cells), rand(3, grid.num_cells),
                                                         rand(3, grid.num_cells), rand(F + grid.num_bnd),
                                                         rand(F + grid.num_bnd))
        d = GfDdtCorr()
        d.rau, d.u_old, d.u_older, d.phi_old, d.phi_older = (ptr(a) for a in keep)
        d.b, d.c, d.dt = 2.0, 0.5, 1e-3
    general = GfMesh()
    ctypes.pointer(general)[0] = grid.cmesh
    general.face_axis = None

    def run():
        out = []
        for m in (general, grid.cmesh):
            phi = FaceField(grid, "phi")
            phi.store.fill_(float("nan"))
            call("gf_face_flux", ctypes.byref(m), 0, ptr(U.store), ptr(t.kind), ptr(t.psib),
                 None if d is None else ctypes.byref(d), ptr(grad), ptr(phi.store), stream_ptr())
            out.append(phi.store)
        return out

    seen = lambda events: sum(n for key, n in events if "k_face_flux" in key)  # noqa: E731
    out, events = record(run, lambda events: seen(events) > kernels)
    assert not bool(out[0].isnan().any()) and torch.equal(out[0], out[1])
    if seen(events) < 1 + kernels:
        lost()
    assert seen(events) == 1 + kernels
