"""Solves of two sizes from two host threads at once, on kernels whose dynamic
shared memory grows with the system: every solve has the bits it has alone.

Each pair of sizes goes to the same kernel instance with different amounts of
shared memory.  A run is many solves of two iterations, each going on from the
last one's solution, and the threads do nothing else between them.
"""

from __future__ import annotations

import ctypes
from concurrent.futures import ThreadPoolExecutor

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROUNDS = 2000


def _solver(variant, precision):
    from gridfoam_b200.meta.config import SolverConfig
    from gridfoam_b200.solvers.krylov import CGSolver

    s = CGSolver(SolverConfig(method="cg", preconditioner="jacobi", tolerance=0.0, rel_tolerance=0.0, max_iter=2,
                              inner_precision=precision, max_outer=1))
    s.variant = variant
    s.host_stats = False
    return s


# rows and vectors on the SMs (FP64, FP32-inner), vectors in shared memory
# (halo and q-recurrence forms), staged box tiles
@pytest.mark.parametrize("variant,precision,shapes", [
    (10, "float64", [(48, 48, 80), (64, 64, 72)]),
    (10, "float32", [(48, 48, 80), (60, 64, 64)]),
    (11, "float64", [(48, 48, 80), (64, 64, 72)]),
    (8, "float64", [(64, 64, 80), (80, 80, 80)]),
    (5, "float64", [(32, 32, 32), (128, 64, 16)]),
])
def test_two_threads_with_systems_of_two_sizes(variant, precision, shapes):
    from gridfoam_b200._lib import load
    from gridfoam_b200.solvers.autotune import BoxSystem

    dev = torch.device("cuda")
    lib = load()
    runs = []
    for shape in shapes:
        s, solver = BoxSystem(*shape, device=dev), _solver(variant, precision)
        x = torch.zeros_like(s.rhs)
        runs.append((x, solver.describe(s, s.diag, s.val, s.rhs, x, symmetric=True)[0], torch.cuda.Stream(), (s, solver)))

    def solves(run):
        x, k, stream, _ = run
        torch.cuda.set_device(x.device)
        status = [lib.gf_pcg_solve(ctypes.byref(k), ctypes.c_void_p(stream.cuda_stream)) for _ in range(ROUNDS)]
        stream.synchronize()
        return sum(st != 0 for st in status)

    torch.cuda.synchronize()
    want = []
    for run in runs:
        assert solves(run) == 0
        want.append(run[0].clone())
        run[0].zero_()
    torch.cuda.synchronize()
    with ThreadPoolExecutor(2) as pool:
        assert list(pool.map(solves, runs)) == [0, 0]
    for run, x in zip(runs, want):
        assert torch.equal(run[0], x)
