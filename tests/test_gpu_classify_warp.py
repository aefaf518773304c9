"""Warp-cooperative classification: location codes and ray counters equal the
oracle's, start points the per-thread query's.

With epsilon above the domain's half-width every walk ends at its start point,
so PLAIN_FP64's mean is g at the start's nearest boundary point: it shows the
start query's winner, also where two primitives are equally near (grid points
on the symmetry planes of a box), which the traversal order of the per-thread
query decides (the oracle's own tree may decide otherwise).  No walk takes a
step, so the means must equal g at closest_points' nearest points to 1e-12
relative everywhere (closest points found through either side of a shared edge
differ by ulps).  Grids have remainders of the eight points a warp takes
together in 2D, and trees have one to four heights.
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes

pytestmark = pytest.mark.gpu


def _star(n):
    return meshes.star_polygon(np.random.default_rng(n), n)


CASES = {
    "star20": (lambda: _star(20), (7, 9, 1)),
    "square_ties": (lambda: meshes.annulus(segments=4), (33, 33, 1)),
    "star2000": (lambda: _star(2000), (141, 139, 1)),
    "slab_ties": (lambda: meshes.slab_box(target_triangles=2000), (13, 9, 5)),
    "sphere_small": (lambda: meshes.uv_sphere(lon=4, lat=4), (9, 9, 9)),
    "sphere": (lambda: meshes.uv_sphere(lon=40, lat=21), (17, 15, 13)),
    "sphere_height4": (lambda: meshes.uv_sphere(lon=180, lat=95), (6, 7, 8)),
}


@pytest.mark.parametrize("name", CASES)
def test_starts_and_locations_match_the_oracle(solver, oracle, name):
    from oracle.oracle import Solve
    make, (nx, ny, nz) = CASES[name]
    m = make()
    solver.set_mesh(m)
    ref = oracle.solve_grid("laplace", Solve(m, nx, ny, nz, N_walks=1, seed=11, epsilon=10.0))
    r = solver.solve_grid("laplace", nx, ny, nz, N_walks=1, seed=11, epsilon=10.0, method="plain")
    loc = ref.location.reshape(r.location.shape)
    assert np.array_equal(r.location, loc)
    for k in ("ambiguous_ray_retries", "indeterminate_points"):
        assert r.counters[k] == ref.counters[k]
    known = ((loc == 1) | (loc == 2)).ravel()
    b = solver.bbox
    axes = [np.array([lo + (hi - lo) * float(i) / float(n - 1) if n > 1 else lo
                      for i in range(n)])
            for lo, hi, n in ((b[0], b[1], nx), (b[2], b[3], ny), (b[4], b[5], nz))]
    pts = np.stack([c.ravel() for c in np.meshgrid(*axes, indexing="ij")], axis=1)[:, :m.dim]
    _, near, bid = solver.closest_points(pts, precision=64)
    if m.dim == 2:
        want = np.where(bid == 0, near[:, 0] ** 2 - near[:, 1] ** 2, 0.0)
    else:
        x, y, z = near.T
        q = x * x + y * y
        want = (z * (8 * z ** 4 - 40 * z * z * q + 15 * q * q)
                + 4 * (8 * z * z - q) * y * (3 * x * x - y * y))
    got = r.mean.ravel()
    assert np.all(np.abs(got - want)[known] <= 1e-12 * np.maximum(1.0, np.abs(want[known])))
    # FAST radii take other (lower) bounds, never other locations
    f = solver.solve_grid("laplace", nx, ny, nz, N_walks=1, seed=11, method="fast")
    assert np.array_equal(f.location, loc)
