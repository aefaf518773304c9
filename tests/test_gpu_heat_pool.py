"""Heat walks that return from the pool in large numbers.

The FP32 shell is 2^-16 of the mesh's size wide; with a far smaller epsilon
nearly every walk that comes within it is re-projected and resumed, several
times over, so full warps of walks are read from the pool and written back to
slots that overlap those just read.  How a solve is cut into tasks decides how
many walks wait together (one walk a task: never two), and must not change a
walk: the counters are equal, the sums agree to 1e-12 of the largest value.
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.heat import HeatProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_resumed_heat_walks_do_not_depend_on_the_tasks(solver, dim):
    if dim == 3:
        solver.set_mesh(meshes.slab_box(target_triangles=2000))
        probes = np.array([0.1, 0.05, 0.01]) * np.random.default_rng(2).uniform(
            0.05, 0.95, size=(9, 3))
        theta = (1e3, (0.05, 0.025, 0.01), 4e-3)
    else:
        solver.set_mesh(meshes.circle(radius=0.05, segments=300))
        probes = 0.03 * np.random.default_rng(2).uniform(-1.0, 1.0, size=(9, 2))
        theta = (1e3, (0.01, -0.005), 8e-3)
    h = HeatProblem(solver, probes, N_walks=640, epsilon=1e-7, seed=4)
    g = np.linspace(-1.0, 1.0, h.n_verts)
    runs = []
    try:
        for chunk in (1, 63, 64, 95, 128, 640):
            solver.set_tuning(chunk, 0)
            f, a = h.forward(*theta, g), h.adjoint(*theta, g)
            assert np.array_equal(a.replayed_mean, f.mean)
            runs.append((f, a))
    finally:
        solver.set_tuning(0, 0)
    f0, a0 = runs[0]
    pairs = [(f0.mean, f.mean) for f, _ in runs[1:]]
    for _, a in runs[1:]:
        pairs += [(a0.jacobian, a.jacobian), (a0.grad_vertex_values, a.grad_vertex_values)]
    for want, got in pairs:
        assert np.all(np.abs(got - want) <= 1e-12 * max(1.0, np.abs(want).max()))
    for f, a in runs[1:]:
        for k in ("total_steps", "exact_queries", "max_steps_hits"):
            assert f.counters[k] == f0.counters[k] == a.counters[k], k
