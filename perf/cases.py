"""What the speed of this package is measured on.

Each case is one call, or one short run of calls, that a program makes on
fields it already has on the GPU:

* ``solve``     a pressure equation assembled once, solved to a tight
                tolerance (CG; ``inner`` gives the precision of its inner
                iterations);
* ``momentum``  a hand-written momentum predictor: ddt + div - laplacian,
                the BiCGStab solve, then H/A;
* ``explicit``  the explicit operators of one time step: gradients of U and
                p, face values, face-normal gradient, face flux, divergence;
* ``adjoint``   a diffusion solve and its reverse pass (gradient in the
                diffusivity), as an inverse problem runs it;
* ``step``      one whole time step or outer iteration of an algorithm;
* ``serve``     the solve server on a handful of small cavities.

Meshes: ``box`` (uniform duct without bodies), ``pipe`` (uniform box with an
immersed pipe), ``wake`` (octree around an immersed cylinder), ``cavity``.
``n`` are the cells per direction, of the base level for ``wake`` (refined
two levels around the cylinder).
"""

from __future__ import annotations

import functools
import math

import torch

from gridfoam_b200 import cases as gc
from gridfoam_b200.algorithms.pressure_velocity import create_algorithm
from gridfoam_b200.core.boundary import DirichletBC
from gridfoam_b200.core.equation import equation
from gridfoam_b200.core.field import CellField, FaceField
from gridfoam_b200.core.grid import AxisProjectedGrid
from gridfoam_b200.fv import fvc, fvm
from gridfoam_b200.meta.config import SimulatorConfig, SolverConfig
from gridfoam_b200.serving import BatchedEngine
from gridfoam_b200.serving.requests import CavityRequest
from gridfoam_b200.solvers.factory import create_solver

DEV = "cuda"
F64 = dict(dtype=torch.float64, device=DEV)
H = 1.0 / 64  # cell size of the box and pipe meshes
NU = 0.02


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, mesh, nx, ny, nz, **more):
    return {"kind": kind, "mesh": mesh, "nx": nx, "ny": ny, "nz": nz, **more}


def listed():
    return [
        # one pressure solve of a case small enough to be bound by latency
        {"name": "solve 16x16x32", **_case("solve", "box", 16, 16, 32, inner="float64")},
        # an odd-sized one of the size that fits the caches
        {"name": "solve 61x67x131", **_case("solve", "box", 61, 67, 131, inner="float64")},
        # FP32 inner iterations in FP64 refinement, the pipe of the benchmark's second workload at half length
        {"name": "solve pipe 64x64x128 fp32", **_case("solve", "pipe", 64, 64, 128, inner="float32")},
        # the pressure system of the octree wake, beyond the caches (most of the benchmark's time)
        {"name": "solve wake 256x160x32", **_case("solve", "wake", 256, 160, 32, inner="float64")},
        # momentum predictors as a user's own algorithm writes them
        {"name": "momentum 47x53x59", **_case("momentum", "box", 47, 53, 59, div="upwind")},
        {"name": "momentum wake 256x160x32", **_case("momentum", "wake", 256, 160, 32, div="linear")},
        # explicit operators of one step, with and without refinement
        {"name": "explicit 96x96x96", **_case("explicit", "box", 96, 96, 96)},
        {"name": "explicit wake 256x160x32", **_case("explicit", "wake", 256, 160, 32)},
        # forward and reverse of a diffusion solve
        {"name": "adjoint 40x40x72", **_case("adjoint", "box", 40, 40, 72)},
        # the lid-driven cavity of the benchmark, one SIMPLE iteration
        {"name": "step cavity 32", **_case("step", "cavity", 32, 32, 32)},
        # one PISO step of a small octree wake
        {"name": "step wake 96x64x12", **_case("step", "wake", 96, 64, 12)},
        # the solve server: eight small cavities, ten outer iterations each
        {"name": "serve 8", **_case("serve", "cavity", 32, 32, 32, count=8, outer=10)},
    ]


def _size(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "momentum", "momentum", "explicit", "explicit", "adjoint", "step",
                       "serve"])
    if kind == "serve":
        n = rng.choice([24, 32, 40])
        return _case("serve", "cavity", n, n, n, count=rng.randint(3, 8), outer=rng.randint(4, 10))
    if kind == "step":
        if rng.random() < 0.5:
            n = _size(rng, 14, 40)
            return _case("step", "cavity", n, n, n)
        nx = rng.randint(60, 96)
        return _case("step", "wake", nx, rng.randint(40, 64), rng.randint(8, 12))
    mesh = rng.choice(["box", "box", "pipe", "wake"]) if kind != "adjoint" else "box"
    if mesh == "wake":
        f = math.exp(rng.uniform(math.log(0.3), 0.0))
        nx, ny, nz = int(256 * f), int(160 * f), max(6, int(32 * f))
    else:
        top = {"solve": 96, "momentum": 80, "explicit": 110, "adjoint": 56}[kind]
        nx, ny, nz = _size(rng, 14, top), _size(rng, 14, top), _size(rng, 16, top)
    more = {}
    if kind == "solve":
        more["inner"] = rng.choice(["float64", "float64", "float32"])
    if kind == "momentum":
        more["div"] = rng.choice(["upwind", "linear", "vanleer"])
    return _case(kind, mesh, nx, ny, nz, **more)


# ---------------------------------------------------------------------------
# meshes and configurations
# ---------------------------------------------------------------------------
def _definition(case):
    """The package's own case definition that a case stands on."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["mesh"] == "wake":
        d = gc.cylinder_wake_case((nx, ny, nz))
    elif case["mesh"] == "cavity":
        d = gc.cavity_case(nx)
    else:
        d = gc.pipe_case(nx, nz)
        d["mesh"] |= {"upper": [nx * H, ny * H, nz * H], "res": [nx, ny, nz]}
        if case["mesh"] == "box":
            d["mesh"]["bodies"] = []
            for field in d["simulator"]["conditions"].values():
                for bc in field["boundary"].values():
                    bc["patches"] = [p for p in bc["patches"] if p != "pipe"]
        else:
            d["mesh"]["bodies"][0] |= {"center": [0.5 * nx * H, 0.5 * ny * H], "radius": 0.4 * min(nx, ny) * H}
        d["inlet_profile"] = None
        d["simulator"]["control"]["deltaT"] = 0.25 * H
    sim = d["simulator"]
    if "div" in case:
        sim["fvSchemes"]["divSchemes"] = {"default": case["div"]}
    if case["kind"] == "step":  # solved until the tolerances of the package's own small cases
        for name, s in sim["fvSolution"]["solvers"].items():
            s |= {"tolerance": 1e-10 if name == "U" else 1e-9, "rel_tolerance": 0.0}
    return d


@functools.lru_cache(maxsize=32)
def _topology(mesh, nx, ny, nz):
    """Mesh and device layout of one mesh: what a program builds once and
    shares between its cases (``AxisProjectedGrid.with_config``)."""
    d = _definition({"kind": "", "mesh": mesh, "nx": nx, "ny": ny, "nz": nz})
    m = gc.build_mesh(d["mesh"], device=DEV)
    return AxisProjectedGrid(SimulatorConfig.model_validate(d["simulator"]), m, device=DEV)


def _grid(case):
    sim = SimulatorConfig.model_validate(_definition(case)["simulator"])
    return _topology(case["mesh"], case["nx"], case["ny"], case["nz"]).with_config(sim)


def _smooth(x, gen, waves=3):
    """A smooth random field with values of about -1..1: a few waves a domain length, and a little noise."""
    lo, hi = x.min(0).values, x.max(0).values
    u = (x - lo) / (hi - lo)
    out = torch.zeros(x.shape[0], **F64)
    for _ in range(4):
        k = torch.randint(1, waves + 1, (3,), generator=gen).to(**F64)
        a = torch.rand(1, generator=gen, dtype=torch.float64).item()
        out += 0.25 * torch.sin(2 * math.pi * (u @ k) + 2 * math.pi * a)
    g = torch.Generator(device=DEV).manual_seed(int(torch.randint(1 << 30, (1,), generator=gen)))
    return out + 0.02 * torch.randn(x.shape[0], generator=g, **F64)


def _velocity(x, gen, main):
    """A velocity field with mean flow 1 along axis ``main``."""
    u = torch.stack([0.3 * _smooth(x, gen) for _ in range(3)], 1)
    u[:, main] += 1.0
    return u


def _inputs(case, x, seed):
    """The random inputs of a case at the cell centres ``x`` [C, 3]."""
    gen = torch.Generator().manual_seed(int(seed))
    main = 2 if case["mesh"] in ("box", "pipe") else 0
    return {
        "U": _velocity(x, gen, main),
        "p": 0.5 * _smooth(x, gen),
        "gamma": 0.01 * (1.0 + 0.5 * _smooth(x, gen).clamp(-1.5, 1.5)),
        "rhs": _smooth(x, gen, 6),
        "weight": _smooth(x, gen, 6),
    }


def _solver(case, method):
    more = {"inner_precision": case["inner"]} if "inner" in case else {}
    rtol = 1e-11 if case.get("inner") == "float32" else 1e-10
    return create_solver(SolverConfig(method=method, preconditioner="jacobi", tolerance=0.0, rel_tolerance=rtol,
                                      max_iter=5000, **more))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _server(outer):
    """A server that has been started for its sizes (once a program)."""
    eng = BatchedEngine(device=DEV, max_slots=8, max_outer=outer, p_tol=1e-9, keep_fields=True)
    eng.prepare((16, 24, 32))
    return eng


def prepare(case, seed):
    if case["kind"] == "serve":
        gen = torch.Generator().manual_seed(int(seed))
        r = torch.rand(2, case["count"], generator=gen, dtype=torch.float64).tolist()
        sizes = [n for n in (case["nx"], 16, 24, 32) if n <= case["nx"]]
        reqs = [CavityRequest(i, sizes[i % len(sizes)], 10.0 ** (1 + 2 * r[0][i]), 0.5 + 1.5 * r[1][i], 0.0)
                for i in range(case["count"])]
        return {"case": case, "engine": _server(case["outer"]), "requests": reqs}
    grid = _grid(case)
    v = _inputs(case, grid.cell_centers, seed)
    s = {"case": case, "grid": grid, **v}
    if case["kind"] == "step":
        transient = grid.sim_config.fvSolution.algorithm.type in gc.TRANSIENT
        U = CellField(grid, "U", "transient" if transient else "local", (3,))
        U.data = v["U"]
        algo = create_algorithm(grid)  # sets the face flux from U
        s |= {"algo": algo, "phi": algo.phi.store.clone()}
        return s
    U = CellField(grid, "U", "transient", (3,))
    p = CellField(grid, "p", "local", ())
    U.data, p.data = v["U"], v["p"]
    U.update_history(reset=True)
    phi = FaceField(grid, "phi")
    fvc.face_flux(phi, U)
    s |= {"Ufield": U, "pfield": p, "phi": phi}
    if case["kind"] == "solve":
        mat = -fvm.laplacian(v["gamma"], p)
        mat.source = mat.source - v["rhs"] * grid.cell_volumes
        s |= {"matrix": mat, "solver": _solver(case, "cg")}
    elif case["kind"] == "momentum":
        s["solver"] = _solver(case, "bicgstab")
    elif case["kind"] == "adjoint":
        s["gamma"].requires_grad_(True)
        s["solver"] = _solver(case, "cg")
    return s


def run(s):
    return {"solve": _run_solve, "momentum": _run_momentum, "explicit": _run_explicit, "adjoint": _run_adjoint,
            "step": _run_step, "serve": _run_serve}[s["case"]["kind"]](s)


def _run_solve(s):
    return {"x": s["solver"].solve(equation(s["pfield"], s["matrix"])).solution}


def _run_momentum(s):
    U = s["Ufield"]
    eqn = fvm.ddt(U) + fvm.div(s["phi"], U) - fvm.laplacian(NU, U)
    u = s["solver"].solve(equation(U, eqn)).solution
    rAU = 1.0 / eqn.A()
    return {"u": u, "rAU": rAU, "HbyA": rAU[:, None] * eqn.H(u)}


def _run_explicit(s):
    U, p, phi = s["Ufield"], s["pfield"], s["phi"]
    out = {"grad_U": fvc.grad(U).store, "grad_p": fvc.grad(p).store, "U_f": fvc.interpolate(U).store,
           "sn_p": fvc.sn_grad(p).store}
    fvc.face_flux(phi, U)
    return {**out, "phi": phi.store, "div": fvc.div(phi).store}


def _run_adjoint(s):
    p, gamma = s["pfield"], s["gamma"]
    gamma.grad = None
    mat = -fvm.laplacian(gamma, p)
    mat.source = mat.source - s["rhs"] * s["grid"].cell_volumes
    x = s["solver"].solve(equation(p, mat)).solution
    (s["weight"] * x).sum().backward()
    return {"x": x.detach(), "grad": gamma.grad}


def _run_step(s):
    a = s["algo"]
    a.U.data, a.p.data = s["U"], s["p"]
    a.phi.store.copy_(s["phi"])
    if a.transient:
        a.U.update_history(reset=True)
        a.phi.update_history(reset=True)
    a.step()
    return {"U": a.U.data, "p": a.p.data, "phi": a.phi.store}


def _run_serve(s):
    done = sorted(s["engine"].run(s["requests"]), key=lambda r: r.id)
    return {"U": [r.U for r in done], "p": [r.p for r in done], "iterations": [r.iterations for r in done]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _cells(case):
    n = case["nx"] * case["ny"] * case["nz"]
    # the wake's band around the cylinder is refined twice
    return 3.13 * n if case["mesh"] == "wake" else n


def _iterations(case):
    """CG iterations of a pressure solve: they grow with the cells along the longest way to the outlet."""
    long = max(case["nx"], case["ny"], case["nz"]) * (4 if case["mesh"] == "wake" else 1)
    cycles = 2.0 if case.get("inner") == "float32" else 1.0
    return cycles * (1.55 if case["mesh"] == "wake" else 6.0) * long


def work(case):
    """Bytes and operations of one pass, each array of the path read or
    written once: fields of 8 bytes a cell value, three faces a cell."""
    C, kind = _cells(case), case["kind"]
    it = _iterations(case)
    cg = (14 * 8 + 3 * 16) * C, 26 * C  # an iteration: five vectors, diagonal, rows
    if kind == "solve":
        half = 0.6 if case["inner"] == "float32" else 1.0
        return {"bytes": it * half * cg[0], "flops": it * cg[1]}
    if kind == "momentum":  # three operators, their sum, some ten BiCGStab iterations, H/A
        return {"bytes": (400 + 10 * 500) * C, "flops": 10 * 150 * C}
    if kind == "explicit":
        return {"bytes": 8 * (3 + 1 + 9 + 3 + 3 * 5 + 1 + 3 * 8) * C, "flops": 200 * C}
    if kind == "adjoint":
        return {"bytes": (2 * it * cg[0] + 500 * C), "flops": 2 * it * cg[1]}
    if kind == "step":
        passes = 1 if case["mesh"] == "cavity" else 2
        return {"bytes": (passes * it * cg[0] + 6000 * C), "flops": passes * it * cg[1] + 1500 * C}
    each = case["outer"] * (0.5 * it * cg[0] + 6000 * C) / 2
    return {"bytes": case["count"] * each, "flops": case["count"] * each / 8}


# ---------------------------------------------------------------------------
# exact values on boxes without bodies, in plain torch
# ---------------------------------------------------------------------------
def _box_centres(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [(torch.arange(n, **F64) + 0.5) * H for n in (nx, ny, nz)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack([x, y, z], -1).reshape(-1, 3)


def _sides(a, axis):
    """Values of ``a`` [..., z, y, x] below and above the inner faces across axis 0 (x), 1 (y) or 2 (z)."""
    d, n = -1 - axis, a.shape[-1 - axis]
    return a.narrow(d, 0, n - 1), a.narrow(d, 1, n - 1)


def _end(a, axis, top):
    d = -1 - axis
    return a.narrow(d, a.shape[d] - 1 if top else 0, 1)


class _Box:
    """-div(gamma grad p) on the duct: p = 0 on z_plus, zero gradient elsewhere, times a cell's volume."""

    def __init__(self, gamma):
        self.k = [0.5 * sum(_sides(gamma, a)) * H for a in range(3)]
        self.out = 2.0 * H * _end(gamma, 2, True)

    def apply(self, p):
        y = torch.zeros_like(p)
        for a in range(3):
            lo, hi = _sides(p, a)
            f = self.k[a] * (lo - hi)
            ylo, yhi = _sides(y, a)
            ylo += f
            yhi -= f
        top = _end(y, 2, True)
        top += self.out * _end(p, 2, True)
        return y

    def diag(self):
        d = torch.zeros(self.k[2].shape[0] + 1, self.k[1].shape[1] + 1, self.k[0].shape[2] + 1, **F64)
        for a in range(3):
            lo, hi = _sides(d, a)
            lo += self.k[a]
            hi += self.k[a]
        top = _end(d, 2, True)
        top += self.out
        return d


def _solve_cg(A, b):
    """Conjugate gradients to rounding, started again from the true residual."""
    d, x = A.diag(), torch.zeros_like(b)
    for _ in range(4):
        r = b - A.apply(x)
        z = r / d
        p, rz, r0 = z.clone(), (r * z).sum(), r.norm().item()
        if r0 <= 1e-15 * b.norm().item():
            break
        for it in range(4000):
            q = A.apply(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            z = r / d
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
            if it % 25 == 0 and r.norm().item() < 1e-13 * r0:
                break
    return x


def _bc_velocity(U):
    """Boundary values of U [3, z, y, x]: zero on walls and inlet, the cell's value on z_plus."""
    return [[0.0 * _end(U, a, False), 0.0 * _end(U, a, True) if a < 2 else _end(U, a, True)] for a in range(3)]


def _box_flux(U):
    """(inner, lower, upper) volume fluxes across each axis, from linear face values."""
    b = _bc_velocity(U)
    return [(0.5 * (lambda s: s[0] + s[1])(_sides(U[a], a)) * H * H, b[a][0][a] * H * H, b[a][1][a] * H * H)
            for a in range(3)]


def exact(case, seed):
    if case["mesh"] != "box" or case.get("div", "upwind") == "vanleer":
        return None
    shape = (case["nz"], case["ny"], case["nx"])
    v = _inputs(case, _box_centres(case), seed)
    t = {k: (a.t().reshape(3, *shape) if a.dim() == 2 else a.reshape(shape)) for k, a in v.items()}
    V = H ** 3
    if case["kind"] in ("solve", "adjoint"):
        gamma = t["gamma"].clone().requires_grad_(case["kind"] == "adjoint")
        with torch.no_grad():
            A = _Box(gamma)
            x = _solve_cg(A, -t["rhs"] * V)
        if case["kind"] == "solve":
            return {"x": x.reshape(-1)}
        with torch.no_grad():
            lam = _solve_cg(A, t["weight"])
        B = _Box(gamma)
        s = (B.out * _end(x, 2, True) * _end(lam, 2, True)).sum()  # lam . A(gamma) x
        for a in range(3):
            (xl, xh), (ll, lh) = _sides(x, a), _sides(lam, a)
            s = s + (B.k[a] * (xl - xh) * (ll - lh)).sum()
        (-s).backward()
        return {"x": x.reshape(-1), "grad": gamma.grad.reshape(-1)}
    U, p = t["U"], t["p"]
    if case["kind"] == "momentum":
        return _exact_momentum(case, U, V)
    # least-squares gradient on a uniform box: the mean of the two sides' slopes
    bU = _bc_velocity(U)
    gU, gp, Uf, snp, phi, end = [], [], [], [], [], {}
    div = torch.zeros_like(p)
    flux = _box_flux(U)
    for a in range(3):
        d = -1 - a

        def slopes(f, lo_s, hi_s):
            lo, hi = _sides(f, a)
            s = (hi - lo) / H
            return 0.5 * (torch.cat([lo_s, s], d) + torch.cat([s, hi_s], d))

        gU.append(slopes(U, (_end(U, a, False) - bU[a][0]) / (H / 2), (bU[a][1] - _end(U, a, True)) / (H / 2)))
        zero = torch.zeros_like(_end(p, a, False))
        sp_hi = -_end(p, a, True) / (H / 2) if a == 2 else zero
        gp.append(slopes(p, zero, sp_hi))
        fi, fl, fh = flux[a]
        lo, hi = _sides(div, a)
        lo += fi
        hi -= fi
        end_l, end_h = _end(div, a, False), _end(div, a, True)
        end_l -= fl
        end_h += fh
    grad_U = torch.stack([gU[j][k] for k in range(3) for j in range(3)]).reshape(9, -1)
    return {"grad_U": grad_U, "grad_p": torch.stack(gp).reshape(3, -1), "U_f": None, "sn_p": None, "phi": None,
            "div": (div / V).reshape(1, -1)}


def _exact_momentum(case, U, V):
    dt = 0.25 * H
    flux = _box_flux(U)
    D = torch.full_like(U[0], V / dt)
    g = NU * H
    up, low = [], []
    for a in range(3):
        fi, fl, fh = flux[a]
        w = (fi >= 0).to(fi.dtype) if case["div"] == "upwind" else 0.5
        lo, hi = _sides(D, a)
        lo += fi * w + g
        hi += -fi * (1 - w) + g
        up.append(fi * (1 - w) - g)
        low.append(-fi * w - g)
        e0, e1 = _end(D, a, False), _end(D, a, True)
        e0 += 2 * g  # boundary values zero: the flux through walls and inlet is zero too
        if a < 2:
            e1 += 2 * g
        else:
            e1 += fh  # outlet: the cell's own value leaves
    b = U * V / dt

    def off(x):
        y = torch.zeros_like(x)
        for a in range(3):
            lo, hi = _sides(x, a)
            ylo, yhi = _sides(y, a)
            ylo += up[a] * hi
            yhi += low[a] * lo
        return y

    u = U.clone()
    for _ in range(3000):
        new = (b - off(u)) / D
        far = (new - u).abs().max().item()
        u = new
        if far < 1e-16:
            break
    hbya = (b - off(u)) / D
    flat = lambda x: x.reshape(3, -1).t()  # noqa: E731
    return {"u": flat(u), "rAU": (V / D).reshape(-1), "HbyA": flat(hbya)}
