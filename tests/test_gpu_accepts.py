"""The quick accept test of the FP32 screened sampler (sc_accepts_2d) against the
exact form, u < clamp_probability(sc_acceptance_2d), in a kernel compiled from
the same headers: for balls alpha R from 1e-6 to 6e4, radii over all of the
ball, and thirteen u next to each threshold (steps of 2^-26 to 2^-8 on either
side, and one anywhere) no decision differs, and the two forms of the
probability differ by at most a fifth of the tolerance that the test allows
for."""
from __future__ import annotations

import subprocess

import pytest

from walk_on_spheres_b200.build import NVCC, NVCC_FLAGS

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "device/common.cuh"
using namespace wosb;
constexpr int kBlocks = 148, kThreads = 256, kEach = 2000;
__global__ void sweep(float lo, float hi, double *worst, unsigned long long *wrong) {
    const unsigned long long t = blockIdx.x * 1ull * blockDim.x + threadIdx.x;
    PhiloxStream s(point_seed(11, t), 0u);
    double w = 0.0;
    unsigned long long bad = 0;
    for (int i = 0; i < kEach; ++i) {
        s.begin_step(static_cast<unsigned>(i));
        const float alpha = expf(-3.0f + 7.0f * s.uniform_f());
        const float R = lo * expf(logf(hi / lo) * s.uniform_f()) / alpha;
        const ScreenedBall<float> b = sc_ball_2d(alpha, R);
        const float v = s.uniform_f(), c = s.uniform_f();
        float r = R * v;                                    // anywhere,
        if (c > 0.4f) r = R * expf(-18.0f * v);             // near the centre,
        if (c > 0.7f) r = R * (1.0f - expf(-16.0f * v));    // near the sphere
        if (c > 0.85f) r = fminf(R, 4.0f * v / alpha);      // within the kernel's reach
        if (!(r > 0.0f) || (b.X >= 2.0f && r >= R)) continue;
        const float p = clamp_probability(sc_acceptance_2d(alpha, b, r));
        // the two forms (sc_accepts_2d's expressions)
        const float x = alpha * r;
        float quick, exact, tol;
        if (b.X < 2.0f) {
            const float i0 = as_i0_small(x), k0 = quick_k0_small(x, i0);
            const float l = __logf(__fdividef(b.R, r));
            quick = k0 - i0 * b.k;
            exact = p * l;
            tol = b.X < 1e-5f ? INFINITY : 1e-5f * (1.0f + k0 + l);
        } else {
            const float e = __expf(quick_log_i0(x) - quick_log_k0(x) + b.k);
            quick = 1.0f - e;
            exact = p;
            tol = e * (1e-5f + 4e-6f * b.X) + 1e-6f;
        }
        if (p > 0.0f && p < 1.0f && tol < INFINITY) w = fmax(w, fabsf(quick - exact) / tol);
        for (int j = -6; j <= 6; ++j) {
            const float step = j == 0 ? 0.0f : copysignf(exp2f(3.0f * abs(j) - 26.0f), j);
            const float u = j == 6 ? s.uniform_f() : p + step;
            if (u >= 0.0f && u < 1.0f) bad += sc_accepts_2d(alpha, b, r, u) != (u < p);
        }
    }
    if (bad) atomicAdd(wrong, bad);
    worst[t] = w;
}
int main() {
    double *worst;
    unsigned long long *wrong;
    cudaMallocManaged(&worst, sizeof(double) * kBlocks * kThreads);
    cudaMallocManaged(&wrong, sizeof(*wrong));
    const float edges[] = {1e-6f, 1e-4f, 0.1f, 2.0f, 4.0f, 20.0f, 200.0f, 2000.0f, 60000.0f};
    for (int k = 0; k < 8; ++k) {
        *wrong = 0;
        sweep<<<kBlocks, kThreads>>>(edges[k], edges[k + 1], worst, wrong);
        const cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
            return 1;
        }
        double w = 0.0;
        for (int i = 0; i < kBlocks * kThreads; ++i) w = std::fmax(w, worst[i]);
        std::printf("%g %llu %.6f\n", edges[k], *wrong, w);
    }
}
"""


def test_every_decision_is_the_exact_forms(tmp_path):
    (tmp_path / "accepts.cu").write_text(PROGRAM)
    subprocess.run([NVCC, *NVCC_FLAGS, "-o", str(tmp_path / "accepts"),
                    str(tmp_path / "accepts.cu")], check=True, capture_output=True)
    r = subprocess.run([str(tmp_path / "accepts")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 8
    for lo, wrong, worst in rows:
        assert int(wrong) == 0, f"alpha R from {lo}: {wrong} decisions differ"
        assert float(worst) <= 0.2, f"alpha R from {lo}: the forms differ by {worst} tol"
