"""Results that come back in one copy (up to 512 KB with the counters: 15 879
points) and in one copy per field, on both sides of the line, in growing and
shrinking solves of one context: a point's values do not depend on it."""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import Solver, meshes

pytestmark = pytest.mark.gpu


def test_values_on_both_sides_of_the_line():
    s = Solver(0).set_mesh(meshes.circle(segments=100))
    pts = np.random.default_rng(1).uniform(-1.1, 1.1, (16000, 2))
    kw = dict(N_walks=2, seed=9, method="fast")
    want = s.solve_points("laplace", pts, **kw)
    assert set(want.location.tolist()) == {0, 1}
    for n in (1, 31, 2000, 15879, 15880, 300, 15879, 16000):
        r = s.solve_points("laplace", pts[:n], **kw)
        for f in ("mean", "variance", "standard_error", "mean_steps", "location"):
            assert np.array_equal(getattr(r, f), getattr(want, f)[:n], equal_nan=True), (n, f)
    s.close()
