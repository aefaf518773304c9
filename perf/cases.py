"""The work that programs built on this package have it do, as timed cases.

A case is a dict of plain values.  `listed()` names twelve of them, `draw(rng)`
gives more of the same ranges, `prepare(case, seed)` builds what a program
holds before the call (a solver with its mesh, a heat problem, a batch),
`run(state)` is one pass through the public entry points and returns every
field they compute, `work(case)` counts what a pass cannot do without and
`exact(case, seed)` gives the solution of the equation where one is known in
closed form (a Monte Carlo mean differs from it by its sampling error).

Kinds of case:

* grid       one registry sweep, `Solver.solve_grid`, over the mesh's bounding
             box: the package's main use, in all three walk methods ("plain"
             is the default and follows the reference's random streams);
* points     `Solver.solve_points` at a handful of probe points, what an
             interactive program or an outer loop calls over and over;
* heat       probe values of the Gaussian heat source and the gradients of a
             loss with respect to the source and every boundary value, forward
             and backward through torch;
* transient  the welding plate's time loop, each step's source read from the
             previous step's field;
* batch      several solves of different meshes, grids and equations in one
             launch sequence;
* new_mesh   a program whose geometry changes between solves: upload a mesh,
             then sweep a grid over it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.batch import Batch
from walk_on_spheres_b200.heat import HeatProblem, heat_probe_values
from walk_on_spheres_b200.solver import Solver
from walk_on_spheres_b200.transient import solve_transient


def listed() -> list[dict]:
    return [
        # the smallest call: 48 probe points, where the launches and the copies count
        dict(name="probe_points_2d", kind="points", mesh="star", prims=256, points=48,
             equation="laplace", source="uniform", alpha=5.0, walks=256, eps=1e-2,
             method="fast"),
        # the annulus Laplace sweep of the workload table: few points, many walks
        dict(name="annulus_laplace", kind="grid", mesh="annulus", prims=256, nx=64, ny=64, nz=1,
             equation="laplace", source="uniform", alpha=5.0, walks=10000, eps=1e-2,
             method="fast"),
        # the disk Poisson sweep that bench.py measures (its Green half)
        dict(name="disk_poisson_green", kind="grid", mesh="circle", prims=1024, nx=256, ny=256,
             nz=1, equation="poisson", source="green", alpha=5.0, walks=4096, eps=1e-2,
             method="fast"),
        # an ordinary 2D sweep of odd sizes with screening, source and a finer shell
        dict(name="star_screened", kind="grid", mesh="star", prims=777, nx=93, ny=131, nz=1,
             equation="screened_poisson", source="green", alpha=3.7, walks=1000, eps=3e-3,
             method="fast"),
        # the largest: the screened sphere of the workload table
        dict(name="sphere_screened", kind="grid", mesh="sphere", prims=16128, nx=64, ny=64,
             nz=64, equation="screened_poisson", source="uniform", alpha=10.0, walks=1024,
             eps=1e-2, method="fast"),
        # the default method (the reference's own streams) at an ordinary 2D size
        dict(name="plain_annulus", kind="grid", mesh="annulus", prims=256, nx=48, ny=48, nz=1,
             equation="laplace", source="uniform", alpha=5.0, walks=1000, eps=1e-2,
             method="plain"),
        # the default method in 3D on an uneven surface, an odd grid
        dict(name="plain_blob", kind="grid", mesh="blob", prims=3968, nx=21, ny=23, nz=19,
             equation="poisson", source="green", alpha=5.0, walks=100, eps=1e-2,
             method="plain"),
        # FP64 arithmetic throughout
        dict(name="fp64_disk", kind="grid", mesh="circle", prims=1024, nx=100, ny=100, nz=1,
             equation="poisson", source="uniform", alpha=5.0, walks=512, eps=1e-2,
             method="fast64"),
        # forward and backward of the differentiable heat source: 20k-triangle slab
        dict(name="heat_gradient", kind="heat", mesh="slab", prims=20000, probes=4096,
             source="green", walks=2048, eps=1e-5, method="fast"),
        # a quarter of the transient welding baseline (49 x 33, 500 walks a step)
        dict(name="transient_weld", kind="transient", nx=49, ny=33, steps=25, walks=500,
             eps=8e-6, scenario=2, cubic=True, method="fast"),
        # twelve solves of the mixed batch's ranges in one graph
        dict(name="batch_mixed", kind="batch", solves=12, largest2d=128, largest3d=24,
             most_prims=8000, walks=512, eps=1e-2, method="fast"),
        # upload and solve of a surface that changes every time
        dict(name="new_mesh_blob", kind="new_mesh", mesh="blob", prims=60000, nx=24, ny=24,
             nz=24, equation="laplace", source="uniform", alpha=5.0, walks=128, eps=1e-2,
             method="fast"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sweep(rng, three, method):
    """Mesh, grid, equation and walks of a drawn sweep."""
    equation = rng.choice(("laplace", "poisson", "screened_poisson", "helmholtz"))
    if three:
        # helmholtz weights kR / sin(kR) need balls well below pi, as here
        mesh = rng.choice(("sphere", "blob"))
        prims = _log_int(rng, 200, 60000 if method == "fast" else 12000)
        nx, ny, nz = (_log_int(rng, 8, 56) for _ in range(3))
    else:
        mesh = rng.choice(("annulus", "circle", "star"))
        prims = _log_int(rng, 24, 4096)
        nx, ny = (_log_int(rng, 12, 230) for _ in range(2))
        nz = 1
    points = nx * ny * nz
    # the FP64 methods run for as long at far fewer walks, above all in 3D
    most = {"fast": 1.0e8, "fast64": 4.0e6, "plain": 2.0e6}[method] / (4 if three else 1)
    high = max(17, min(10000 if method == "fast" else 200 if three else 800,
                       int(most / points)))
    return dict(mesh=mesh, prims=prims, nx=nx, ny=ny, nz=nz, equation=equation,
                source=rng.choice(("uniform", "green")),
                alpha=round(math.exp(rng.uniform(0.0, 3.0)), 3), walks=_log_int(rng, 16, high),
                eps=round(math.exp(rng.uniform(math.log(2e-3), math.log(2e-2))), 5),
                method=method)


def draw(rng) -> dict:
    kind = rng.choice(("grid", "grid", "grid", "grid", "grid", "points", "heat", "transient",
                       "batch", "new_mesh"))
    if kind == "grid":
        method = rng.choice(("fast", "fast", "plain", "plain", "fast64"))
        return dict(kind="grid", **_sweep(rng, rng.random() < 0.45, method))
    if kind == "points":
        c = _sweep(rng, rng.random() < 0.5, "fast")
        for k in ("nx", "ny", "nz"):
            del c[k]
        return dict(kind="points", points=_log_int(rng, 1, 3000),
                    **{**c, "walks": _log_int(rng, 32, 4096)})
    if kind == "new_mesh":
        c = _sweep(rng, rng.random() < 0.6, "fast")
        return dict(kind="new_mesh", **{**c, "walks": min(c["walks"], 300)})
    if kind == "heat":
        return dict(kind="heat", mesh=rng.choice(("slab", "slab", "circle")),
                    prims=_log_int(rng, 300, 20000), probes=_log_int(rng, 16, 4096),
                    source=rng.choice(("green", "green", "mis", "uniform")),
                    walks=_log_int(rng, 64, 2048),
                    eps=round(math.exp(rng.uniform(math.log(1e-5), math.log(1e-4))), 7),
                    method="fast")
    if kind == "transient":
        return dict(kind="transient", nx=_log_int(rng, 9, 96) | 1, ny=_log_int(rng, 9, 64) | 1,
                    steps=_log_int(rng, 4, 25), walks=_log_int(rng, 50, 500), eps=8e-6,
                    scenario=rng.choice((2, 2, 3)), cubic=rng.random() < 0.7,
                    method="fast")
    return dict(kind="batch", solves=_log_int(rng, 2, 16), largest2d=_log_int(rng, 32, 160),
                largest3d=_log_int(rng, 12, 28), most_prims=_log_int(rng, 2200, 20000),
                walks=_log_int(rng, 64, 512), eps=1e-2, method="fast")


# ------------------------------------------------------------------- inputs

def _mesh(case, rng):
    kind, n = case["mesh"], case["prims"]
    if kind == "annulus":
        return meshes.annulus(segments=max(12, n // 2))
    if kind == "circle":
        return meshes.circle(radius=0.05 if case["kind"] == "heat" else 1.0,
                             segments=min(n, 4096))
    if kind == "star":
        return meshes.star_polygon(rng, n)
    if kind == "slab":
        return meshes.slab_box(target_triangles=n)
    # lon x lon/2 bands have about lon^2 triangles
    lon = max(8, int(round(math.sqrt(n))))
    if kind == "sphere":
        return meshes.uv_sphere(lon=lon + 1, lat=lon // 2 + 1) if n != 16128 else meshes.uv_sphere()
    return meshes.perturbed_sphere(rng, lon, max(4, lon // 2))


def _params(case, seed):
    return dict(N_walks=case["walks"], epsilon=case["eps"], seed=seed, alpha=case["alpha"],
                source_mode=case["source"], method=case["method"])


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    walk_seed = int(rng.integers(1, 1 << 62))
    state = dict(case=case)
    if case["kind"] == "transient":
        state["solver"] = Solver(0)
        dt = 0.1
        kw = dict(nx=case["nx"], ny=case["ny"], dt=dt, total_time=dt * case["steps"],
                  walks=case["walks"], epsilon=case["eps"], scenario=case["scenario"],
                  cubic=case["cubic"], method=case["method"], seed=walk_seed)
        kw["heat_on_time"] = 0.5 * dt * case["steps"]
        if case["scenario"] == 3:
            kw.update(source_start_x=-0.05, weld_y=0.0, weld_speed=0.02)
        state["kw"] = kw
        # a plate that still carries heat from an earlier pass
        hot = np.zeros((case["nx"], case["ny"]))
        hot[1:-1, 1:-1] = rng.uniform(0.0, 30.0, size=(case["nx"] - 2, case["ny"] - 2))
        state["initial"] = hot
        return state
    if case["kind"] == "batch":
        solver = Solver(0)
        batch = Batch(solver)
        ids = []
        for k in range(case["solves"]):
            # sizes in even steps of their logarithm over the batch's ranges, 2D and 3D in turn
            f = (k // 2 + 0.5) / ((case["solves"] + 1) // 2)
            if k % 2 == 0:
                m = meshes.star_polygon(rng, int(64 * (2048 / 64) ** f))
                side = int(round(24 * (case["largest2d"] / 24) ** f))
                grid = (side, side + k, 1)
            else:
                lon = int(round(math.sqrt(500 * (case["most_prims"] / 500) ** f)))
                m = meshes.perturbed_sphere(rng, lon, max(4, lon // 2))
                side = int(round(8 * (case["largest3d"] / 8) ** f))
                grid = (side, side, side + k % 3)
            equation = ("laplace", "poisson", "screened_poisson")[(k // 2) % 3]
            ids.append(batch.add_solve(
                batch.add_mesh(m), equation, *grid, N_walks=max(1, case["walks"] >> (k % 3)),
                epsilon=case["eps"], alpha=1.0 + 1.5 * k, seed=walk_seed + k,
                source_mode=("uniform", "green")[k % 4 // 2], method=case["method"]))
        batch.prepare()
        state.update(solver=solver, batch=batch, ids=ids)
        return state
    mesh = _mesh(case, rng)
    state["solver"] = solver = Solver(0)
    if case["kind"] == "new_mesh":
        state.update(mesh=mesh, kw=_params(case, walk_seed))
        return state
    solver.set_mesh(mesh)
    if case["kind"] == "heat":
        if mesh.dim == 3:
            hi = np.array([0.10, 0.05, 0.01])
            probes = hi * rng.uniform(0.001, 0.999, size=(case["probes"], 3))
            x0, sigma = np.array([0.05, 0.025, 0.01]), 2e-3
        else:
            r = 0.05 * np.sqrt(rng.uniform(0.0, 0.98, case["probes"]))
            t = rng.uniform(0.0, 2.0 * math.pi, case["probes"])
            probes = np.stack([r * np.cos(t), r * np.sin(t)], axis=1)
            x0, sigma = np.array([0.01, -0.005]), 8e-3
        x0 = x0 + 1e-3 * rng.standard_normal(mesh.dim)
        heat = HeatProblem(solver, probes, N_walks=case["walks"], epsilon=case["eps"],
                           seed=walk_seed, source_mode=case["source"], method=case["method"],
                           proposal=(x0, sigma))
        leaf = dict(dtype=torch.float64, device="cuda:0", requires_grad=True)
        state.update(heat=heat, theta=[
            torch.tensor(1e3 * rng.uniform(0.5, 2.0), **leaf), torch.tensor(x0, **leaf),
            torch.tensor(sigma, **leaf),
            torch.tensor(1e-3 * rng.standard_normal(heat.n_verts), **leaf)],
            target=torch.tensor(1e-3 * rng.standard_normal(heat.n), dtype=torch.float64,
                                device="cuda:0"))
        return state
    state["kw"] = _params(case, walk_seed)
    if case["kind"] == "points":
        # probes spread over the inner part of the domain
        d = rng.standard_normal((case["points"], mesh.dim))
        d /= np.linalg.norm(d, axis=1)[:, None]
        lo, hi = (0.55, 0.95) if case["mesh"] == "annulus" else (0.0, 0.7)
        state["probes"] = d * rng.uniform(lo, hi, size=(case["points"], 1))
    return state


# --------------------------------------------------------------------- pass

def _fields(r):
    return dict(mean=r.mean, variance=r.variance, standard_error=r.standard_error,
                mean_steps=r.mean_steps, location=r.location)


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "grid":
        return _fields(state["solver"].solve_grid(case["equation"], case["nx"], case["ny"],
                                                  case["nz"], **state["kw"]))
    if kind == "points":
        return _fields(state["solver"].solve_points(case["equation"], state["probes"],
                                                    **state["kw"]))
    if kind == "new_mesh":
        solver = state["solver"].set_mesh(state["mesh"])
        return _fields(solver.solve_grid(case["equation"], case["nx"], case["ny"], case["nz"],
                                         **state["kw"]))
    if kind == "heat":
        theta = state["theta"]
        for t in theta:
            t.grad = None
        u = heat_probe_values(state["heat"], *theta)
        ((u - state["target"]) ** 2).sum().backward()
        return dict(u=u.detach(), grads=[t.grad for t in theta])
    if kind == "transient":
        r = solve_transient(state["solver"], initial=state["initial"], **state["kw"])
        return dict(fields=r.fields, standard_error=r.standard_error)
    state["batch"].run(use_graph=True)
    return [_fields(state["batch"].result(i)) for i in state["ids"]]


# --------------------------------------------------------------------- work

def work(case: dict) -> dict:
    """Bytes: the mesh (or initial field), the points and the result fields
    once each.  Flops: walks x steps x the arithmetic of one step (a direction,
    a move and one distance to the nearest primitive: about 35 in 2D and 80 in
    3D; random draws, searches and special functions are not counted), with a
    walk of about 1.2 ln(size / eps) steps in 2D and 2.1 ln(size / eps) in 3D."""
    kind = case["kind"]

    def cost(dim, walks, size_over_eps):
        steps = (1.2 if dim == 2 else 2.1) * math.log(size_over_eps)
        return walks * steps * (35.0 if dim == 2 else 80.0)

    if kind == "transient":
        n = case["nx"] * case["ny"]
        return {"bytes": 16.0 * n * (case["steps"] + 1) + 8.0 * n,
                "flops": case["steps"] * cost(2, float(n) * case["walks"], 0.05 / case["eps"])}
    if kind == "batch":
        b = f = 0.0
        for k in range(case["solves"]):
            s = (k // 2 + 0.5) / ((case["solves"] + 1) // 2)
            walks = max(1, case["walks"] >> (k % 3))
            if k % 2 == 0:
                n, dim = 0.7 * (24 * (case["largest2d"] / 24) ** s) ** 2, 2
                prims = 64 * (2048 / 64) ** s
            else:
                n, dim = 0.5 * (8 * (case["largest3d"] / 8) ** s) ** 3, 3
                prims = 500 * (case["most_prims"] / 500) ** s
            b += 33.0 * n + 24.0 * prims
            f += cost(dim, n * walks, 1.0 / case["eps"])
        return {"bytes": b, "flops": f}
    dim = 2 if case["mesh"] in ("annulus", "circle", "star") else 3
    mesh_bytes = case["prims"] * (28.0 if dim == 2 else 24.0)
    if kind == "heat":
        n = case["probes"]
        # forward walks and their replay
        return {"bytes": mesh_bytes + 8.0 * case["prims"] + n * (8.0 * dim + 16.0),
                "flops": 2.0 * cost(dim, float(n) * case["walks"], 0.01 / case["eps"])}
    if kind == "points":
        n, inside = case["points"], case["points"]
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        inside = n * {"annulus": 0.59, "circle": 0.78, "star": 0.7}.get(case["mesh"], 0.5)
    return {"bytes": mesh_bytes + 33.0 * n,
            "flops": cost(dim, inside * case["walks"], 1.0 / case["eps"])}


# -------------------------------------------------------------------- exact

def exact(case: dict, seed: int):
    """The equation's solution in the place of the mean, at the points that lie
    inside (NaN outside, as the sweep gives it): `laplace` with g = x^2 - y^2
    on one loop is x^2 - y^2, on the annulus (inner value 0) it is
    (16/15 r^2 - 1/(15 r^2)) cos 2 theta, and 2D `poisson` on the unit disk has
    the log profile of its uniform load.  None elsewhere, and where the walks
    are so few that the sampling error hides the value."""
    if case["kind"] != "grid" or case["nz"] != 1 or case["walks"] < 400:
        return None
    eq, mesh_kind = case["equation"], case["mesh"]
    if not (eq == "laplace" or (eq == "poisson" and mesh_kind == "circle" and
                                case["source"] == "green" and case["walks"] >= 2000)):
        return None
    rng = np.random.default_rng(seed)
    rng.integers(1, 1 << 62)
    mesh = _mesh(case, rng)
    b = mesh.bbox()
    ax = [lo + (hi - lo) * np.arange(n) / (n - 1)
          for lo, hi, n in ((b[0], b[1], case["nx"]), (b[2], b[3], case["ny"]))]
    X, Y = np.meshgrid(*ax, indexing="ij")
    wn = np.zeros(X.shape, dtype=np.int64)
    for (p, q) in mesh.prims:
        (x0, y0), (x1, y1) = mesh.verts[p], mesh.verts[q]
        area = (x1 - x0) * (Y - y0) - (X - x0) * (y1 - y0)
        wn += (y0 <= Y) & (y1 > Y) & (area > 0)
        wn -= (y0 > Y) & (y1 <= Y) & (area < 0)
    r2 = np.maximum(X * X + Y * Y, 1e-300)
    if eq == "poisson":
        f, a = 0.1, 0.15
        u = np.where(r2 <= a * a, f / 4 * (a * a - r2) + f * a * a / 2 * math.log(1 / a),
                     -f * a * a / 4 * np.log(r2))
    elif mesh_kind == "annulus":
        u = (16.0 / 15.0 * r2 - 1.0 / (15.0 * r2)) * (X * X - Y * Y) / r2
    else:
        u = X * X - Y * Y
    mean = np.where(wn != 0, u, np.nan)[:, :, None]
    return dict(mean=mean, variance=None, standard_error=None, mean_steps=None, location=None)
