"""Probe means of FAST_FP32 heat walks on a circle, to the order of their FP64
sums.  A walk's path depends on every FP32 rounding on its way, so a list scan
or a query that the compiler contracts otherwise shows here as a difference of
1e-8 and more; the recorded values are those of the walks since the list scans
were introduced."""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.heat import HeatProblem

pytestmark = pytest.mark.gpu

VALUES = {
    (300, "green"): ([0.00596249506996063, 0.049864516341243115, 0.06830503932924539,
                      0.05578700904429228], 80376, 16435),
    (300, "uniform"): ([0.019093411862093634, 0.02488869385158203, 0.0691796317398885,
                        0.06926906117084823], 80551, 16155),
    (1575, "green"): ([0.006437343879836967, 0.021721634769689357, 0.03606188534317825,
                       0.03968485751145549], 80561, 16580),
    (1575, "uniform"): ([-0.0014416119325713712, 0.037260698667236414, 0.04726180658162678,
                         0.05830258762595192], 80768, 16388),
}


@pytest.mark.parametrize("segments, mode", VALUES)
def test_recorded_heat_walks(solver, segments, mode):
    solver.set_mesh(meshes.circle(radius=0.05, segments=segments))
    probes = 0.03 * np.array([[-0.9, 0.1], [0.2, 0.7], [0.6, -0.5], [0.0, 0.0]])
    h = HeatProblem(solver, probes, N_walks=2000, epsilon=2e-5, seed=4, source_mode=mode)
    r = h.forward(1e3, (0.01, -0.005), 8e-3, np.sin(np.arange(h.n_verts)))
    mean, steps, queries = VALUES[segments, mode]
    assert r.counters["total_steps"] == steps and r.counters["exact_queries"] == queries
    assert np.all(np.abs(r.mean - mean) <= 1e-12)
