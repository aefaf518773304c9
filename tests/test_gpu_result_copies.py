"""Results that come back through the staging block (below 2048 points, or up to
15 879 in separate arrays), straight into arrays that lie end to end, and in
one copy per field, on both sides of each line, in growing and shrinking solves
of one context: a point's values do not depend on it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from walk_on_spheres_b200 import Solver, _lib, meshes

pytestmark = pytest.mark.gpu


def test_values_on_both_sides_of_the_line():
    s = Solver(0).set_mesh(meshes.circle(segments=100))
    pts = np.random.default_rng(1).uniform(-1.1, 1.1, (16000, 2))
    kw = dict(N_walks=2, seed=9, method="fast")
    want = s.solve_points("laplace", pts, **kw)
    assert set(want.location.tolist()) == {0, 1}
    fields = ("mean", "variance", "standard_error", "mean_steps", "location")
    for n in (1, 31, 2047, 2048, 15879, 15880, 300, 15879, 16000):
        r = s.solve_points("laplace", pts[:n], **kw)
        for f in fields:
            assert np.array_equal(getattr(r, f), getattr(want, f)[:n], equal_nan=True), (n, f)
        # separate arrays, as a program with the C interface may pass them
        out = [np.empty(n) for _ in range(4)] + [np.empty(n, dtype=np.uint8)]
        p = s.params("laplace", **kw)
        c = _lib.Counters()
        some = np.ascontiguousarray(pts[:n])
        rc = s._L.wos_solve_points(s._ctx, C.byref(p), some.ctypes.data_as(C.c_void_p), None, n,
                                   *(a.ctypes.data_as(C.c_void_p) for a in out), C.byref(c))
        assert rc == 0
        for f, a in zip(fields, out):
            assert np.array_equal(a, getattr(want, f)[:n], equal_nan=True), (n, f)
    s.close()
