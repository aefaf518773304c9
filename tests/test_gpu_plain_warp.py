"""PLAIN_FP64 walks with warp-cooperative queries, against the oracle.

The walks follow the reference's streams, so PLAIN's rule applies (as in
test_gpu_parity): at least 98% of the inside points to 1e-9 relative, every
point within 4 standard errors, equal step counts where the means agree, equal
location codes.  The meshes cover wide trees of one to four heights, a corner
where two boundaries meet (ties between primitives of different boundary
values) and a scene far from the origin, whose queries stay per thread; the
grids give 1, 2 and 8 points per warp with a remainder.
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200.meshes import Mesh

pytestmark = pytest.mark.gpu


def _star(n):
    return meshes.star_polygon(np.random.default_rng(n), n)


def _two_boundary_corner():
    # an L whose re-entrant corner joins a segment of boundary 0 and one of 1
    v = np.array([[0, 0], [2, 0], [2, 1], [1, 1], [1, 2], [0, 2]], dtype=np.float64) - 0.3
    p = np.array([[i, (i + 1) % 6] for i in range(6)], dtype=np.int32)
    return Mesh(2, v, p, np.array([0, 1, 0, 1, 0, 1], dtype=np.int32))


def _far_annulus():
    m = meshes.annulus(segments=64)
    return Mesh(2, m.verts + 1e6, m.prims, m.boundary_ids)


CASES = {
    "height1": (lambda: _star(20), "laplace", (17, 15, 1), 40),
    "height2": (lambda: _star(777), "screened_poisson", (31, 29, 1), 20),
    "height2_full": (lambda: _star(1024), "poisson", (67, 63, 1), 6),
    "height3": (lambda: _star(1025), "helmholtz", (131, 127, 1), 2),
    "corner": (_two_boundary_corner, "laplace", (33, 35, 1), 60),
    "far": (_far_annulus, "laplace", (13, 13, 1), 30),
    "sphere_height2": (lambda: meshes.uv_sphere(lon=12, lat=6), "laplace", (9, 8, 7), 40),
    "sphere_height3": (lambda: meshes.uv_sphere(lon=60, lat=31), "poisson", (33, 33, 31), 1),
    "sphere_height4": (lambda: meshes.uv_sphere(lon=180, lat=95), "screened_poisson",
                       (7, 7, 7), 6),
}


@pytest.mark.parametrize("name", CASES)
def test_plain_walks_match_the_oracle(solver, oracle, name):
    from oracle.oracle import Solve
    make, eq, (nx, ny, nz), walks = CASES[name]
    m = make()
    solver.set_mesh(m)
    r = solver.solve_grid(eq, nx, ny, nz, N_walks=walks, seed=91, method="plain",
                          source_mode="green", alpha=3.0)
    ref = oracle.solve_grid(eq, Solve(m, nx, ny, nz, N_walks=walks, seed=91, source_mode=1,
                                      alpha=3.0))
    loc = ref.location.reshape(r.location.shape)
    assert np.array_equal(r.location, loc)
    ins = loc == 1
    assert ins.any()
    want, got = ref.mean.reshape(loc.shape)[ins], r.mean[ins]
    close = np.abs(got - want) <= 1e-9 * np.maximum(1.0, np.abs(want))
    assert close.mean() >= 0.98, close.mean()
    se = ref.standard_error.reshape(loc.shape)[ins]
    if walks > 1:
        assert np.all(np.abs(got - want)[~close] <= 4.0 * se[~close])
    steps = ref.mean_steps.reshape(loc.shape)[ins]
    assert np.array_equal(r.mean_steps[ins][close], steps[close])


def _sliver_fan():
    # a closed fan whose side triangles are up to 1e4 times longer than wide:
    # their FP32 distances say little, so the queries must compare them in FP64
    rng = np.random.default_rng(3)
    n = 400
    t = np.sort(rng.uniform(0.0, 2.0 * np.pi, n))
    t[1::4] = t[::4] + 1e-4
    ring = np.stack([np.cos(t), np.sin(t), np.zeros(n)], axis=1)
    v = np.concatenate([ring, [[0.0, 0.0, 0.9], [0.0, 0.0, -0.9]]])
    i = np.arange(n, dtype=np.int32)
    j = np.roll(i, -1).astype(np.int32)
    top = np.stack([i, j, np.full(n, n, np.int32)], axis=1)
    bottom = np.stack([j, i, np.full(n, n + 1, np.int32)], axis=1)
    p = np.concatenate([top, bottom]).astype(np.int32)
    return Mesh(3, v, p, np.zeros(len(p), dtype=np.int32))


@pytest.mark.parametrize("make", [_two_boundary_corner, _sliver_fan, lambda: _star(161),
                                  lambda: meshes.uv_sphere(lon=40, lat=21)],
                         ids=["corner", "slivers", "star161", "sphere"])
def test_fp64_walks_take_exact_radii(solver, oracle, make):
    """FAST_FP64 and PLAIN_FP64 with one step per walk: the walk ends at the
    nearest boundary point of its first step, so a wrong nearest primitive
    shows in the boundary value (PLAIN, point by point against the oracle) or
    in the mean (FAST_FP64, within 4.5 standard errors at 99% of the points).
    Where two boundaries meet in a corner, FAST_FP64 may take either one's
    value (its distances round otherwise than the reference's, so equal ones
    need not tie), and only PLAIN_FP64 is compared."""
    from oracle.oracle import Solve
    m = make()
    solver.set_mesh(m)
    n = (15, 13, 1) if m.dim == 2 else (9, 9, 9)
    walks = 400
    ref = oracle.solve_grid("laplace", Solve(m, *n, N_walks=walks, seed=5, max_steps=1))
    r = solver.solve_grid("laplace", *n, N_walks=walks, seed=5, max_steps=1, method="plain")
    ins = ref.location.reshape(r.location.shape) == 1
    want, se = ref.mean.reshape(ins.shape)[ins], ref.standard_error.reshape(ins.shape)[ins]
    close = np.abs(r.mean[ins] - want) <= 1e-9 * np.maximum(1.0, np.abs(want))
    assert close.mean() >= 0.98, close.mean()
    if len(set(m.boundary_ids.tolist())) > 1:
        return
    f = solver.solve_grid("laplace", *n, N_walks=walks, seed=5, max_steps=1, method="fast64")
    assert np.array_equal(f.location, r.location)
    both = np.sqrt(se ** 2 + f.standard_error[ins] ** 2)
    live = both > 0
    z = (f.mean[ins] - want)[live] / both[live]
    assert (np.abs(z) <= 4.5).mean() >= 0.99, np.abs(z).max()
