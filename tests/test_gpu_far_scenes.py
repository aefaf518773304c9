"""Scenes so far from the origin that FP32 bounds cannot steer FP64 queries:
classification, FAST_FP32 and FAST_FP64 solves, heat walks and batches keep the
per-thread queries there (PLAIN_FP64: test_gpu_plain_warp).

Locations equal PLAIN's, means lie within 4.5 standard errors of its at 99% of
the points (test_gpu_plain_warp's rule; FP32 positions are rounded to 6e-5
there, far below the sampling error), the heat replay repeats its forward pass
bit for bit, and a batch reproduces its solves as in test_gpu_batch.
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.batch import Batch
from walk_on_spheres_b200.heat import HeatProblem
from walk_on_spheres_b200.meshes import Mesh

pytestmark = pytest.mark.gpu

SHIFT = 1000.0


def _far(dim):
    m = meshes.annulus(segments=100) if dim == 2 else meshes.uv_sphere(lon=20, lat=11)
    return Mesh(dim, m.verts + SHIFT, m.prims, m.boundary_ids)


def _agree(a, b):
    both = np.sqrt(a.standard_error ** 2 + b.standard_error ** 2)
    ok = both > 0.0
    z = np.abs(a.mean - b.mean)[ok] / both[ok]
    assert ok.any() and (z <= 4.5).mean() >= 0.99, z.max()


@pytest.mark.parametrize("method", ["fast", "fast64"])
@pytest.mark.parametrize("dim", [2, 3])
def test_far_solves(solver, dim, method):
    solver.set_mesh(_far(dim))
    n = (15, 13, 1) if dim == 2 else (7, 6, 5)
    want = solver.solve_grid("laplace", *n, N_walks=400, seed=5, method="plain")
    r = solver.solve_grid("laplace", *n, N_walks=400, seed=5, method=method)
    assert set(want.location.ravel().tolist()) >= {0, 1}
    assert np.array_equal(r.location, want.location)
    _agree(r, want)


@pytest.mark.parametrize("dim", [2, 3])
def test_far_heat(solver, dim):
    solver.set_mesh(_far(dim))
    rng = np.random.default_rng(4)
    d = rng.standard_normal((40, dim))
    probes = SHIFT + 0.75 * d / np.linalg.norm(d, axis=1)[:, None]
    theta = (3.0, (SHIFT + 0.4,) * dim, 0.5)
    g = rng.standard_normal(len(_far(dim).verts))
    runs = {}
    for method in ("fast", "fast64"):
        h = HeatProblem(solver, probes, N_walks=600, epsilon=1e-2, seed=6, method=method)
        runs[method] = h.forward(*theta, g)
        assert np.array_equal(h.adjoint(*theta, g).replayed_mean, runs[method].mean)
        assert np.all(runs[method].location == 1)
    _agree(runs["fast"], runs["fast64"])


def test_far_batches(solver):
    specs = [(dim, method) for dim in (2, 3) for method in ("fast", "fast64")]
    alone = []
    for dim, method in specs:
        solver.set_mesh(_far(dim))
        n = (15, 13, 1) if dim == 2 else (7, 6, 5)
        alone.append((n, solver.solve_grid("laplace", *n, N_walks=100, seed=5, method=method)))
    batch = Batch(solver)
    ids = [batch.add_solve(batch.add_mesh(_far(dim)), "laplace", *n, N_walks=100, seed=5,
                           method=method) for (dim, method), (n, _) in zip(specs, alone)]
    batch.prepare()
    batch.run()
    for i, (_, want) in zip(ids, alone):
        r = batch.result(i)
        assert np.array_equal(r.location, want.location)
        assert np.array_equal(r.mean_steps, want.mean_steps, equal_nan=True)
        for k in ("mean", "variance", "standard_error"):
            x, y = getattr(r, k), getattr(want, k)
            assert np.array_equal(np.isnan(x), np.isnan(y)), k
            both = ~np.isnan(x)
            assert np.allclose(x[both], y[both], rtol=1e-12, atol=1e-15), k
