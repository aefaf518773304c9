"""FAST_FP32 and heat walks that wait in a warp's pool.

A walk's path depends on its own index alone, so however a solve is cut into
tasks (one walk, one short of a warp, a warp, one more, several pools' worth),
the total steps and closest-point queries are equal, and the fields agree to
the order of their FP64 sums: 1e-12 of the largest value.  The scenes cover
lists in 2D and 3D, trees without lists, lane scans, the rejection sampler and
a step cap that ends walks outside the shell.
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.heat import HeatProblem

pytestmark = pytest.mark.gpu

CHUNKS = (1, 31, 32, 33, 95, 200)


def _star(n):
    return meshes.star_polygon(np.random.default_rng(n), n)


CASES = {
    "lists2d": (lambda: _star(300), "poisson", (9, 8, 1), dict(source_mode="green")),
    "sampler2d": (lambda: _star(300), "screened_poisson", (9, 8, 1),
                  dict(source_mode="green", alpha=9.0)),
    "sampler_lane_scan": (lambda: _star(40), "screened_poisson", (9, 8, 1),
                          dict(source_mode="green", alpha=2.0)),
    "lane_scan_cap": (lambda: _star(40), "laplace", (9, 8, 1), dict(max_steps=3)),
    "cap2d": (lambda: _star(300), "laplace", (9, 8, 1), dict(max_steps=2)),
    "lists3d": (lambda: meshes.uv_sphere(lon=40, lat=21), "laplace", (6, 5, 6), dict()),
    "dense3d": (lambda: meshes.uv_sphere(lon=250, lat=120), "screened_poisson", (5, 5, 5),
                dict(alpha=4.0)),
    "cap3d": (lambda: meshes.uv_sphere(lon=40, lat=21), "poisson", (6, 5, 6),
              dict(max_steps=4)),
}


def _close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(a)
    scale = max(1.0, np.abs(a[ok]).max()) if ok.any() else 1.0
    assert np.all(np.abs(a - b)[ok] <= 1e-12 * scale)


@pytest.mark.parametrize("lists", [True, False], ids=["lists", "no_lists"])
@pytest.mark.parametrize("name", CASES)
def test_walks_do_not_depend_on_the_tasks(solver, monkeypatch, name, lists):
    make, eq, (nx, ny, nz), kw = CASES[name]
    if not lists:
        monkeypatch.setenv("WOS_NEAR_LISTS", "0")
    solver.set_mesh(make())
    runs = []
    try:
        for chunk in CHUNKS:
            solver.set_tuning(chunk, 0)
            runs.append(solver.solve_grid(eq, nx, ny, nz, N_walks=200, seed=17, method="fast",
                                          **kw))
    finally:
        solver.set_tuning(0, 0)
    ref = runs[0]
    assert ref.counters["inside_points"] > 0
    for r in runs[1:]:
        for k in ("total_steps", "exact_queries", "max_steps_hits", "total_walks"):
            assert r.counters[k] == ref.counters[k], k
        for f in ("mean", "variance", "mean_steps"):
            _close(getattr(r, f), getattr(ref, f))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("cap", [100000, 6], ids=["free", "cap"])
def test_heat_walks_do_not_depend_on_the_tasks(solver, dim, cap):
    if dim == 3:
        solver.set_mesh(meshes.slab_box(target_triangles=2000))
        probes = np.array([0.1, 0.05, 0.01]) * np.random.default_rng(2).uniform(
            0.05, 0.95, size=(9, 3))
        theta = (1e3, (0.05, 0.025, 0.01), 4e-3)
    else:
        solver.set_mesh(meshes.circle(radius=0.05, segments=300))
        probes = 0.03 * np.random.default_rng(2).uniform(-1.0, 1.0, size=(9, 2))
        theta = (1e3, (0.01, -0.005), 8e-3)
    h = HeatProblem(solver, probes, N_walks=200, epsilon=2e-5, max_steps=cap, seed=4)
    g = np.linspace(-1.0, 1.0, h.n_verts)
    runs = []
    try:
        for chunk in CHUNKS:
            solver.set_tuning(chunk, 0)
            f, a = h.forward(*theta, g), h.adjoint(*theta, g)
            assert np.array_equal(a.replayed_mean, f.mean)
            runs.append((f, a))
    finally:
        solver.set_tuning(0, 0)
    f0, a0 = runs[0]
    for f, a in runs[1:]:
        for k in ("total_steps", "exact_queries", "max_steps_hits"):
            assert f.counters[k] == f0.counters[k] == a.counters[k], k
        _close(f.mean, f0.mean)
        _close(a.jacobian, a0.jacobian)
        _close(a.grad_vertex_values, a0.grad_vertex_values)


def test_points_beyond_any_distance_are_outside(solver):
    """A finite point whose squared distance overflows has no nearest primitive:
    it is classified, not read through slot -1."""
    solver.set_mesh(meshes.circle(segments=300))
    pts = np.array([[1e200, 0.0], [-1e300, 1e300], [0.1, 0.2]])
    for method in ("fast", "plain", "fast64"):
        r = solver.solve_points("laplace", pts, N_walks=8, seed=1, method=method)
        assert r.location.tolist() == [0, 0, 1]
