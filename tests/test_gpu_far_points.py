"""Points so far away that FP32 distances to the mesh overflow, or nearly do.

Their queries stay on the per-thread FP64 tree.  The meshes have wide trees of
one to four heights, because a node's padding children (at distance infinity)
are what a query without any finite FP32 distance must not enter.  Far points
lie outside; the points beside them keep the values of a solve without them,
bit for bit (a point's streams depend on its own index).  Walks that leave an
open surface take the same queries; their number that reaches the step cap is
the oracle's to 5 binomial standard deviations (single walks are not compared:
900 steps amplify rounding until they part).
"""
from __future__ import annotations

import numpy as np
import pytest

from walk_on_spheres_b200 import meshes
from walk_on_spheres_b200._lib import Grid, WosError
from walk_on_spheres_b200.heat import HeatProblem
from walk_on_spheres_b200.meshes import Mesh

pytestmark = pytest.mark.gpu

MESHES = {
    "height1_2d": lambda: meshes.circle(segments=30),
    "height2_2d": lambda: meshes.circle(segments=300),
    "height3_2d": lambda: meshes.circle(segments=1100),
    "height4_2d": lambda: meshes.circle(segments=33000),
    "height1_3d": lambda: meshes.uv_sphere(lon=5, lat=4),
    "height2_3d": lambda: meshes.uv_sphere(lon=20, lat=11),
    "height3_3d": lambda: meshes.uv_sphere(lon=40, lat=21),
    "height4_3d": lambda: meshes.uv_sphere(lon=180, lat=95),
}
FAR = (1e8, 9.9e8, 1.01e9, 1e13, 1.8e19, 2e19, 1e20, 3e38, 4e38, 1e77, 1e155, 1e300)


def _points(dim):
    rng = np.random.default_rng(8)
    near = rng.uniform(-0.3, 0.3, size=(9, dim))
    far = [s * v * np.eye(dim)[k] for v in FAR for k in range(dim) for s in (1.0, -1.0)]
    far += [np.full(dim, -v) for v in FAR]
    return near, np.array(far)


@pytest.mark.parametrize("method", ["fast", "fast64", "plain"])
@pytest.mark.parametrize("name", MESHES)
def test_far_points_are_outside(solver, name, method):
    m = MESHES[name]()
    solver.set_mesh(m)
    near, far = _points(m.dim)
    kw = dict(N_walks=16, seed=3, method=method)
    alone = solver.solve_points("laplace", near, **kw)
    both = solver.solve_points("laplace", np.concatenate([near, far]), **kw)
    n = len(near)
    assert alone.location.tolist() == [1] * n
    assert both.location.tolist() == [1] * n + [0] * len(far)
    assert np.isnan(both.mean[n:]).all()
    assert np.array_equal(both.mean[:n], alone.mean)
    assert np.array_equal(both.mean_steps[:n], alone.mean_steps)


@pytest.mark.parametrize("method", ["fast", "fast64"])
@pytest.mark.parametrize("name", ["height3_2d", "height4_3d"])
def test_far_heat_probes_are_outside(solver, name, method):
    m = MESHES[name]()
    solver.set_mesh(m)
    near, far = _points(m.dim)
    theta = (1.0, (0.1,) * m.dim, 0.2)
    g = np.linspace(-1.0, 1.0, len(m.verts))
    kw = dict(N_walks=16, epsilon=1e-3, seed=3, method=method)
    alone = HeatProblem(solver, near, **kw).forward(*theta, g)
    both = HeatProblem(solver, np.concatenate([near, far]), **kw).forward(*theta, g)
    n = len(near)
    assert both.location.tolist() == [1] * n + [0] * len(far)
    assert np.array_equal(both.mean[:n], alone.mean)


def _open_sphere():
    m = meshes.uv_sphere(lon=60, lat=31)
    p = m.prims[m.verts[m.prims].mean(axis=1)[:, 2] > -0.1]
    return Mesh(3, m.verts, p, np.zeros(len(p), dtype=np.int32))


def test_walks_that_leave_an_open_surface(solver, oracle):
    from oracle.oracle import Solve
    m = _open_sphere()
    assert len(m.prims) > 1024
    solver.set_mesh(m)
    kw = dict(N_walks=12, seed=7, max_steps=900)
    ref = oracle.solve_grid("laplace", Solve(m, 7, 7, 7, **kw))
    n = 12 * int((ref.location == 1).sum())
    hits = ref.counters["max_steps_hits"]
    assert 0.05 * n < hits < 0.95 * n
    q = hits / n
    for method in ("plain", "fast64"):
        r = solver.solve_grid("laplace", 7, 7, 7, method=method, **kw)
        assert np.array_equal(r.location, ref.location.reshape(r.location.shape))
        assert np.isfinite(r.mean[r.location == 1]).all()
        assert abs(r.counters["max_steps_hits"] - hits) <= 5.0 * np.sqrt(2.0 * n * q * (1.0 - q))


@pytest.mark.parametrize("dim", [2, 3])
def test_grids_whose_spacing_overflows(solver, dim):
    """Their first coordinates are NaN, the others infinite.  In 2D all are
    outside; a 3D ray from such a point may cross anything, but the call returns
    (walks from there find no primitive, which is an error) and the context
    stays usable."""
    m = MESHES["height3_2d" if dim == 2 else "height4_3d"]()
    solver.set_mesh(m)
    near, _ = _points(dim)
    want = solver.solve_points("laplace", near, N_walks=16, seed=3, method="fast")
    for lim in (1e19, 1e21, 1e300, 1.7e308):
        for yz in (lim, 0.5):
            grid = Grid(3, 3, 3 if dim == 3 else 1, -lim, lim, -yz, yz, -yz, yz)
            expected = np.zeros((3, 3, 3 if dim == 3 else 1), dtype=np.uint8)
            if lim < 1.7e308:  # the middle of each axis is 0
                if yz == 0.5:
                    expected[1] = 1
                else:
                    expected[(1,) * dim] = 1
            for method in ("fast", "fast64", "plain"):
                kw = dict(N_walks=2, seed=1, method=method, max_steps=50)
                try:
                    r = solver.solve_grid("laplace", grid=grid, **kw)
                except WosError:
                    assert dim == 3 and lim == 1.7e308
                    continue
                if dim == 2 or lim < 1.7e308:
                    assert np.array_equal(r.location, expected)
    again = solver.solve_points("laplace", near, N_walks=16, seed=3, method="fast")
    assert np.array_equal(again.mean, want.mean)


def test_fp32_walks_that_leave_an_open_surface(solver, oracle):
    """Counts at a step cap that they reach within FP32's range, as above; with
    a higher cap their distances overflow, which is an error."""
    from oracle.oracle import Solve
    m = _open_sphere()
    solver.set_mesh(m)
    kw = dict(N_walks=12, seed=7, max_steps=60)
    ref = oracle.solve_grid("laplace", Solve(m, 7, 7, 7, **kw))
    n = 12 * int((ref.location == 1).sum())
    hits = ref.counters["max_steps_hits"]
    q = hits / n
    assert 0.05 < q < 0.95
    r = solver.solve_grid("laplace", 7, 7, 7, method="fast", **kw)
    assert abs(r.counters["max_steps_hits"] - hits) <= 5.0 * np.sqrt(2.0 * n * q * (1.0 - q))
    with pytest.raises(WosError):
        solver.solve_grid("laplace", 7, 7, 7, method="fast", N_walks=12, seed=7, max_steps=900)
    again = solver.solve_grid("laplace", 7, 7, 7, method="fast", **kw)
    assert np.array_equal(again.mean, r.mean, equal_nan=True)


@pytest.mark.parametrize("name", MESHES)
def test_closest_points_of_far_points(solver, name):
    """FP64 distances up to the largest whose square is finite, FP32 ones to a
    relative 1e-5 (the coordinates' and squares' rounding) up to FP32's range;
    beyond it, and for NaN, no primitive: infinity and boundary id -1."""
    m = MESHES[name]()
    solver.set_mesh(m)
    x = np.array([1e3, 1e10, 1e18, 3e19, 1e30, 1e150, 1e160, np.nan])
    pts = np.zeros((len(x), m.dim))
    pts[:, 0] = x
    pts[-1] = np.nan
    reach = np.max(m.verts[:, 0])
    for precision, last in ((64, 5), (32, 2)):
        dist, near, bid = solver.closest_points(pts, precision=precision)
        want = np.where(np.arange(len(x)) <= last, x - reach, np.inf)
        ok = np.isfinite(want)
        assert np.all(np.abs(dist[ok] - want[ok]) <= 1e-5 * want[ok])
        assert np.array_equal(np.isinf(dist), ~ok)
        assert np.all(near[~ok] == 0.0)
        if bid is not None:
            assert np.all(bid[~ok] == -1)


@pytest.mark.parametrize("name", ["height2_2d", "height3_2d", "height3_3d", "height4_3d"])
def test_scenes_whose_fp32_distances_overflow(solver, name):
    """A mesh 2^66 times as large: its lattice and lists hold no finite distance,
    so FAST_FP32 walks find no primitive (an error) and read nothing.  FP64
    walks are those of the unit mesh, scaled: equal steps, and g = x^2 - y^2 (2D)
    and a degree-5 harmonic (3D) scale exactly."""
    m = MESHES[name]()
    f = 2.0 ** 66
    near, _ = _points(m.dim)
    kw = dict(N_walks=8, seed=3, max_steps=100)
    solver.set_mesh(m)
    want = solver.solve_points("laplace", near, method="plain", epsilon=1e-2, **kw)
    solver.set_mesh(Mesh(m.dim, m.verts * f, m.prims, m.boundary_ids))
    with pytest.raises(WosError):
        solver.solve_points("laplace", near * f, method="fast", epsilon=1e-2 * f, **kw)
    r = solver.solve_points("laplace", near * f, method="plain", epsilon=1e-2 * f, **kw)
    assert np.array_equal(r.location, want.location)
    assert np.array_equal(r.mean_steps, want.mean_steps)
    g = f ** 2 if m.dim == 2 else f ** 5
    assert np.all(np.abs(r.mean / g - want.mean) <= 1e-9 * np.maximum(1.0, np.abs(want.mean)))


@pytest.mark.parametrize("power", [133, 533])
@pytest.mark.parametrize("name", ["height1_2d", "height3_2d", "height4_3d"])
def test_scenes_beyond_fp32(solver, name, power):
    """Coordinates that FP32 cannot hold (2^133), or whose FP64 squares overflow
    too (2^533): no lattice; FAST_FP32 fails as above.  FP64 walks at 2^133 are
    the unit mesh's, scaled; at 2^533 no distance is finite, and 2D calls only
    have to return (3D meshes are refused: no triangle has a finite area).  The
    solver stays usable."""
    m = MESHES[name]()
    f = 2.0 ** power
    near, _ = _points(m.dim)
    kw = dict(N_walks=8, seed=3, max_steps=100)
    solver.set_mesh(m)
    want = solver.solve_points("laplace", near, method="plain", epsilon=1e-2, **kw)
    scaled = Mesh(m.dim, m.verts * f, m.prims, m.boundary_ids)
    if m.dim == 3 and power == 533:
        with pytest.raises(WosError):
            solver.set_mesh(scaled)
        return
    solver.set_mesh(scaled)
    results = {}
    for method in ("fast", "fast64", "plain"):
        try:
            results[method] = solver.solve_points("laplace", near * f, method=method,
                                                  epsilon=1e-2 * f, **kw)
        except WosError:
            assert method == "fast"
    if power == 133:
        assert "fast" not in results
        r = results["plain"]
        assert np.array_equal(r.location, want.location)
        assert np.array_equal(r.mean_steps, want.mean_steps)
        g = f ** 2 if m.dim == 2 else f ** 5
        assert np.all(np.abs(r.mean / g - want.mean)
                      <= 1e-9 * np.maximum(1.0, np.abs(want.mean)))
    solver.set_mesh(m)
    again = solver.solve_points("laplace", near, method="plain", epsilon=1e-2, **kw)
    assert np.array_equal(again.mean, want.mean)
