"""Results by every way back to the host: through the process's page-locked block
(up to 31 767 points, once there have been many), through a context's own
staging memory before that and where another thread's solve holds the block (up
to 15 879), and in one copy per field; on both sides of each line, in growing
and shrinking solves.  A point's values do not depend on it."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest
import torch

from walk_on_spheres_b200 import Solver, _lib, meshes

pytestmark = pytest.mark.gpu

FIELDS = ("mean", "variance", "standard_error", "mean_steps", "location")
SIZES = (1, 31, 2048, 15879, 15880, 300, 31767, 31768, 15879, 32000)


def _solve_all(pts, want, kw, rounds):
    s = Solver(0).set_mesh(meshes.circle(segments=100))
    for n in SIZES * rounds:
        some = np.ascontiguousarray(pts[:n])
        r = s.solve_points("laplace", some, **kw)
        for f in FIELDS:
            assert np.array_equal(getattr(r, f), getattr(want, f)[:n], equal_nan=True), (n, f)
    s.close()


@pytest.mark.parametrize("threads", [1, 6])  # some 2 ms of copies make the block
def test_values_do_not_depend_on_the_way_back(threads):
    pts = np.random.default_rng(1).uniform(-1.1, 1.1, (32000, 2))
    kw = dict(N_walks=2, seed=9, method="fast")
    with Solver(0).set_mesh(meshes.circle(segments=100)) as s:
        want = s.solve_points("laplace", pts, **kw)
    assert set(want.location.tolist()) == {0, 1}
    failed = []

    def work():
        try:
            _solve_all(pts, want, kw, 6 if threads == 1 else 4)
        except BaseException as e:  # reported by the main thread
            failed.append(repr(e))

    running = [threading.Thread(target=work) for _ in range(threads)]
    for t in running:
        t.start()
    for t in running:
        t.join()
    assert not failed


def test_page_locked_fields_that_lie_end_to_end():
    """Fields in page-locked arrays of their own, which the allocator lays next to
    one another: adjacent addresses, but not one allocation."""
    n = 65536
    pts = np.random.default_rng(2).uniform(-0.7, 0.7, (n, 2))
    kw = dict(N_walks=1, seed=9, method="fast")
    with Solver(0).set_mesh(meshes.circle(segments=100)) as s:
        want = s.solve_points("laplace", pts, **kw)
        out = [torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
        out.append(torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy())
        p, c = s.params("laplace", **kw), _lib.Counters()
        rc = s._L.wos_solve_points(s._ctx, C.byref(p), pts.ctypes.data_as(C.c_void_p), None, n,
                                   *(a.ctypes.data_as(C.c_void_p) for a in out), C.byref(c))
        assert rc == 0
    for f, a in zip(FIELDS, out):
        assert np.array_equal(a, getattr(want, f), equal_nan=True), f
