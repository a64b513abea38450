"""The sum of an edge sample's two sub-path values (dtrt_gb300/csrc/dt_common.cuh), compiled for
the host with nvcc: exactly the FP64 sum of the two FP32 values, as when each is added to the FP64
accumulator by itself."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

DRIVER = r"""
#include <cstdio>
#include "dt_common.cuh"
int main(int, char **a) {
    FILE *f = fopen(a[1], "rb"), *g = fopen(a[2], "wb");
    float x[3];
    while (fread(x, 4, 3, f) == 3) {
        const double v = dt::pair_value(x[0], x[1], x[2]);
        fwrite(&v, 8, 1, g);
    }
    fclose(g);
    return 0;
}
"""


def test_pair_value_is_the_fp64_sum(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc is missing")
    (tmp_path / "m.cu").write_text(DRIVER)
    exe = str(tmp_path / "m")
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"),
                    str(tmp_path / "m.cu"), "-o", exe], check=True)
    rng = np.random.default_rng(1)
    n = 20000
    a = np.exp(rng.uniform(-20, 20, n)).astype(np.float32)
    b = (-a * np.exp(rng.uniform(-12, 12, n))).astype(np.float32)
    b[: n // 2] = -a[: n // 2] * (1 + rng.normal(0, 1e-3, n // 2)).astype(np.float32)  # nearly cancelling pairs
    s = rng.normal(size=n).astype(np.float32)
    np.stack([a, b, s], 1).tofile(tmp_path / "i.bin")
    subprocess.run([exe, str(tmp_path / "i.bin"), str(tmp_path / "o.bin")], check=True)
    got = np.fromfile(tmp_path / "o.bin")
    want = (a * s).astype(np.float64) + (b * s).astype(np.float64)
    assert np.array_equal(got, want)
    assert np.mean(want != ((a + b) * s).astype(np.float64)) > 0.3  # an FP32 sum would not do
