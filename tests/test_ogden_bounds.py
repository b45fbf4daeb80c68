"""A part's Ogden series bounds (make_matp in ft_materials.cuh), compiled for the
host: the radii against the definition they stand for, a bisection of the whole
truncation bound, and what forming them costs.  The allocation-free entry point
does so on every call: 60 us at most (half a millisecond with the bisections
themselves, a few microseconds with Newton's steps; the least of many calls).

The radii are FP32 values of a root found to 1e-10: 2.5e-7."""
import json
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

ALPHAS = [5.0, -5.0, 0.5, 25.0, 2.0, 8.0, 1.0, -1.0, 3.7, -40.0, 120.0, -0.01, 1e4]
PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include "ft_materials.cuh"
using namespace ftgpu;
template <class R> void one(double alpha, bool last) {
  const double p[9] = {1040.0, 1.5e3, 2.0e7, alpha, 0, 0, 0, 0, 0};
  double best = 1e9;
  MatP<R> m;
  for (int k = 0; k < 50; ++k) {
    const auto t = std::chrono::steady_clock::now();
    m = make_matp<R>(6, p);
    best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count());
  }
  printf("{\"alpha\": %.17g, \"bytes\": %d, \"us\": %g, \"r\": [", alpha, (int)sizeof(R), 1e6 * best);
  for (int k = 0; k < OgdenSeries<R>::kSteps; ++k) printf("%s%.9g", k ? ", " : "", (double)m.ser_r[k]);
  printf("]}%s\n", last ? "" : ",");
}
int main(int n, char **v) {
  printf("[");
  for (int k = 1; k < n; ++k) {
    one<float>(atof(v[k]), false);
    one<double>(atof(v[k]), k == n - 1);
  }
  printf("]");
}
"""


def radius(alpha, n, eps):
    k = np.arange(n + 400)
    with np.errstate(divide="ignore"):  # (an even alpha: a factor zero, the coefficients behind it too)
        size = np.cumsum(np.log(np.abs(alpha / 2 - 1 - k) / (k + 1)))[n:]  # ln |b_j|, j = n + 1 ..
    j = np.arange(n + 1, n + 401)

    def within(r):
        return np.exp(np.minimum(size + (j - 1) * np.log(r), 700.0)).sum() * (3 + 2 * r) <= eps

    lo, hi = 0.0, 0.5
    if within(hi):
        return hi
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if within(mid) else (lo, mid)
    return lo


def test_series_bounds_and_their_cost(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "bounds.cu", tmp_path / "bounds"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                    "-I" + os.path.join(ROOT, "femtech_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    got = json.loads(subprocess.run([str(exe)] + [repr(a) for a in ALPHAS], check=True, capture_output=True,
                                    text=True).stdout)
    assert len(got) == 2 * len(ALPHAS)
    for g in got:
        a = g["alpha"]
        counts, eps = ((9, 20), 1e-7) if g["bytes"] == 4 else ((8, 12, 16, 24, 32), 5e-17)
        want = np.array([radius(a, n, eps) for n in counts]) * (1 - 1e-6)
        if g["bytes"] == 4 and abs(a) < 2:
            want[1] = want[0]  # (the longer FP32 series only where it is as exact)
        if a == 1e4:
            want[:] = 0.0  # (the bound at 0.5 is beyond FP64: the eigen-decomposition alone)
        np.testing.assert_allclose(g["r"], want, rtol=2.5e-7, err_msg=str(g))
        assert g["us"] < 60.0, g
