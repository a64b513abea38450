"""The FP64 reciprocal, square root, sine, cosine and angle of the edge kernels
(dtrt_gb300/csrc/dt_common.cuh), compiled for the host with nvcc, against numpy: a few
roundings of 1.1e-16 each, whatever the size of the argument."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "dt_common.cuh"
int main(int, char **a) {
    FILE *f = fopen(a[1], "rb"), *g = fopen(a[2], "wb");
    double x[2];
    while (fread(x, 8, 2, f) == 2) {
        double o[6];
        o[0] = dt::rcp_d(x[0]);
        o[1] = dt::rsqrt_d(fabs(x[0]), o[2]);
        dt::sincos_d(x[1], o[3], o[4]);
        o[5] = dt::angle_d(sin(x[1]), cos(x[1]));
        fwrite(o, 8, 6, g);
    }
    fclose(g);
    return 0;
}
"""


def test_fp64_math(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc is missing")
    (tmp_path / "m.cu").write_text(DRIVER)
    exe = str(tmp_path / "m")
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"),
                    str(tmp_path / "m.cu"), "-o", exe], check=True)
    rng = np.random.default_rng(3)
    n = 20000
    x = np.exp(rng.uniform(-300, 300, n)) * rng.choice([-1.0, 1.0], n)  # past the FP32 range on both sides
    x[: n // 2] = rng.uniform(-4, 4, n // 2)
    x[:4] = [1.0, -1.0, 2.0 ** -126, 2.0 ** 127]
    t = rng.uniform(0, np.pi, n)
    t[:7] = [0.0, np.pi, np.pi / 2, np.pi / 4, 3 * np.pi / 4, 1e-7, np.pi - 1e-7]
    np.stack([x, t], 1).tofile(tmp_path / "i.bin")
    subprocess.run([exe, str(tmp_path / "i.bin"), str(tmp_path / "o.bin")], check=True)
    o = np.fromfile(tmp_path / "o.bin").reshape(n, 6)
    eps = 2.0 ** -53
    assert np.abs(o[:, 0] * x - 1).max() <= 5 * eps
    assert np.abs(o[:, 1] * np.sqrt(np.abs(x)) - 1).max() <= 6 * eps
    assert np.abs(o[:, 2] / np.sqrt(np.abs(x)) - 1).max() <= 6 * eps
    assert np.abs(o[:, 3] - np.sin(t)).max() <= 4 * eps and np.abs(o[:, 4] - np.cos(t)).max() <= 4 * eps
    # absolute: the inputs sin(t), cos(t) are rounded, and t itself is up to pi
    assert np.abs(o[:, 5] - t).max() <= 8 * eps
