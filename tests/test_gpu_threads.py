"""Contexts on eight host threads, whose launches of one kernel ask for
different amounts of shared memory: the heat pass and its adjoint (with a scene
staged beside their pools, 46 and 68 KB), and sweeps of two scenes that are
staged whole when there are no near-boundary lists.  Every call succeeds and
repeats its first result.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

from walk_on_spheres_b200 import Solver, meshes
from walk_on_spheres_b200.heat import HeatProblem

pytestmark = pytest.mark.gpu


def _heat(adjoint):
    s = Solver(0).set_mesh(meshes.circle(radius=0.05, segments=1000))
    probes = 0.03 * np.random.default_rng(2).uniform(-1.0, 1.0, size=(9, 2))
    h = HeatProblem(s, probes, N_walks=64, epsilon=2e-5, seed=4)
    g = np.linspace(-1.0, 1.0, h.n_verts)
    theta = (1e3, (0.01, -0.005), 8e-3)
    if adjoint:
        return s, lambda: h.adjoint(*theta, g).replayed_mean
    return s, lambda: h.forward(*theta, g).mean


def _sweep(segments):
    s = Solver(0).set_mesh(meshes.circle(segments=segments))
    pts = np.random.default_rng(2).uniform(-0.5, 0.5, (40, 2))
    return s, lambda: s.solve_points("laplace", pts, N_walks=64, method="fast").mean


@pytest.mark.parametrize("make, a, b, lists", [(_heat, False, True, True),
                                               (_sweep, 150, 4000, False)],
                         ids=["heat", "sweep"])
def test_threads_launch_one_kernel(monkeypatch, make, a, b, lists):
    if not lists:
        monkeypatch.setenv("WOS_NEAR_LISTS", "0")
    failed = []
    gate = threading.Barrier(8)

    def work(arg):
        try:
            s, call = make(arg)
            first = call()
            gate.wait(60)
            for _ in range(1500):
                assert np.array_equal(call(), first)
            s.close()
        except Exception as e:  # reported by the main thread
            failed.append(f"{make.__name__}({arg}): {e}")
            gate.abort()

    threads = [threading.Thread(target=work, args=(x,)) for x in (a, b) * 4]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
