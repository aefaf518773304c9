"""The FP32 slab tests that choose the boxes of a ray (device/wide64.cuh),
compiled for the host and compared with the same tests in FP64: a box that the
ray meets is never lost, also where a component of the ray is zero or vanishes
in FP32 and the origin lies exactly on a padded face; and a box whose slab the
origin is off by a thousandth is not met by a ray along it."""
from __future__ import annotations

import subprocess

import numpy as np
import pytest

from walk_on_spheres_b200.build import ARCH, CSRC, INCLUDE, NVCC

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "device/common.cuh"
int main() {
    float lo[3], hi[3];
    double ray[3];
    while (std::scanf("%f %f %f %f %f %f %lf %lf %lf", lo, lo + 1, lo + 2, hi, hi + 1, hi + 2, ray,
                      ray + 1, ray + 2) == 9) {
        float t0 = 0.0f, t1 = INFINITY;
        for (int k = 0; k < 3; ++k) {
            wosb::clip_to_slab(lo[k], hi[k], wosb::ray_reciprocal(ray[k]), t0, t1);
        }
        std::printf("%d\n", t0 <= t1 * (1.0f + 0x1p-20f) ? 1 : 0);
    }
}
"""


@pytest.fixture(scope="module")
def meets(tmp_path_factory):
    d = tmp_path_factory.mktemp("slabs")
    (d / "slabs.cu").write_text(PROGRAM)
    subprocess.run([NVCC, *ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(INCLUDE),
                    "-I", str(CSRC), "-o", str(d / "slabs"), str(d / "slabs.cu")], check=True,
                   capture_output=True)

    def run(rows):
        text = "\n".join(" ".join(f"{x:.17g}" for x in row) for row in rows) + "\n"
        r = subprocess.run([str(d / "slabs")], input=text, capture_output=True, text=True,
                           check=True)
        return np.array(r.stdout.split(), dtype=int)
    return run


def _expected(lo, hi, ray):
    t0, t1 = 0.0, np.inf
    for a, b, r in zip(lo, hi, ray):
        if r == 0.0:
            if not a <= 0.0 <= b:
                return 0
            continue
        u, v = sorted((a / r, b / r))
        t0, t1 = max(t0, u), min(t1, v)
    return int(t0 <= t1)


def test_rays_along_a_face_meet_the_box(meets):
    rows = []
    for small in (0.0, -0.0, 1e-300, -1e-300, 1e-42, -1e-42, 1e-39, 1e-35, -1e-35):
        for lo, hi in ((0.0, 0.25), (-0.25, 0.0), (0.0, 0.0), (-0.5, 0.5), (-1e9, 0.0)):
            for axis in range(3):
                for sign in (1.0, -1.0):
                    box_lo, box_hi = [-1.0] * 3, [1.0] * 3
                    box_lo[axis], box_hi[axis] = lo, hi
                    ray = [0.6 * sign, 0.8, 0.8]
                    ray[axis] = small
                    rows.append((*box_lo, *box_hi, *ray))
    assert meets(rows).all()


def test_rays_along_a_slab_miss_the_boxes_beside_it(meets):
    rows = []
    for small in (0.0, -0.0, 1e-300, -1e-42, 1e-35):
        for lo, hi in ((1e-3, 0.25), (-0.25, -1e-3), (1e6, 1e9)):
            rows.append((lo, -1.0, -1.0, hi, 1.0, 1.0, small, 0.6, -0.8))
    assert not meets(rows).any()


def test_no_box_is_lost(meets):
    rng = np.random.default_rng(6)
    n = 20000
    lo = rng.uniform(-2.0, 1.5, (n, 3)).astype(np.float32)
    hi = lo + rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    ray = rng.standard_normal((n, 3))
    ray /= np.linalg.norm(ray, axis=1)[:, None]
    ray[rng.random((n, 3)) < 0.1] = 0.0
    want = np.array([_expected(a, b, r) for a, b, r in zip(lo.astype(float), hi.astype(float),
                                                           ray)])
    # a padding above FP32 rounding, as the traversal has one
    got = meets(np.concatenate([lo - 1e-5, hi + 1e-5, ray], axis=1))
    assert (got >= want).all()
    assert 0 < want.sum() and got.sum() <= want.sum() + 0.001 * n
