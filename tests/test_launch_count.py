"""Launch accounting: what ``launch_total`` says against the kernels that the
profiler sees, for the calls whose kernel count depends on the mesh or on the
iterations."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _grid(mesh, size):
    from gridfoam_b200.cases import build_mesh, cylinder_wake_case, pipe_case
    from gridfoam_b200.core.grid import AxisProjectedGrid
    from gridfoam_b200.meta.config import SimulatorConfig

    case = cylinder_wake_case(size) if mesh == "wake" else pipe_case(33, 34)
    if mesh == "box":
        case["mesh"] |= {"res": list(size), "upper": [n / 64 for n in size], "bodies": []}
    return AxisProjectedGrid(SimulatorConfig.model_validate(case["simulator"]), build_mesh(case["mesh"], device="cuda"),
                             device="cuda")


def _kernels(run):
    """The package's kernels launched by ``run``, by the profiler and by the account."""
    from gridfoam_b200 import _lib
    from tests.profiled import lost, record

    def counted():
        _lib.clear_launches()
        run()

    seen = lambda events: sum(n for key, n in events if "gf::k_" in key)  # noqa: E731
    run()
    _, events = record(counted, lambda events: seen(events) >= _lib.launch_total())
    if seen(events) < _lib.launch_total():
        lost()
    return seen(events), _lib.launch_total()


@pytest.mark.parametrize("mesh,size", [("box", (20, 21, 22)), ("box", (72, 71, 70)), ("wake", (40, 27, 5)),
                                       ("wake", (116, 74, 14))])
def test_gradients_and_face_fluxes(mesh, size):
    from gridfoam_b200.core.field import CellField, FaceField
    from gridfoam_b200.fv import fvc

    grid = _grid(mesh, size)
    p, U, phi = CellField(grid, "p", "local", ()), CellField(grid, "U", "local", (3,)), FaceField(grid, "phi")

    def run():
        fvc.grad(p)
        fvc.grad(U)
        fvc.interpolate(U)
        fvc.face_flux(phi, U)

    seen, counted = _kernels(run)
    assert seen == counted


@pytest.mark.parametrize("iterations", [0, 2, 3, 4, 7, 8])
def test_split_cg_loop(iterations):
    from gridfoam_b200 import _lib
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import CGSolver
    from tests.test_resident_cg import _ring

    s, diag, val = _ring(7177, 4, 3)
    solver = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=0.0, rel_tolerance=0.0,
                                   max_iter=max(1, iterations)))
    solver.max_iter = iterations
    solver.variant = 29
    rhs = torch.ones((1, 7177), dtype=torch.float64, device="cuda")
    stats = []
    _lib.TRACK_DEFERRED = True
    try:
        seen, counted = _kernels(lambda: stats.append(solver.solve_arrays(s, diag, val, rhs, torch.zeros_like(rhs))[0]))
    finally:
        _lib.TRACK_DEFERRED = False
        _lib.clear_launches()
    assert stats[-1].iterations == iterations
    assert seen == counted
