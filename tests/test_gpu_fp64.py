"""FP64 arithmetic of the edge kernels as the device runs it, in a small program of its own: the reuse
of a CDF's random number is the correctly rounded quotient; reciprocal, square root, sine,
cosine and angle, whose seeds are the device's FP32 approximations, keep the bounds that the
host build of the same code has (test_fp64_math.py), also at the ends of the seeds' range."""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

DRIVER = r"""
#include <cstdio>
#include <vector>
#include "dt_kernels.cuh"
using namespace dt;
static __global__ void k_reuse(const double *cdf, int n, const double *u, int m, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    double x = u[i], pdf;
    out[3 * i] = sample_reuse(cdf, n, x, pdf);
    out[3 * i + 1] = x;
    out[3 * i + 2] = pdf;
}
static __global__ void k_math(const double *in, int m, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double x = in[4 * i], t = in[4 * i + 1];
    double *o = out + 6 * i;
    o[0] = rcp_d(x);
    o[1] = rsqrt_d(fabs(x), o[2]);
    sincos_d(t, o[3], o[4]);
    o[5] = angle_d(in[4 * i + 2], in[4 * i + 3]);
}
static std::vector<double> read(const char *p) {
    std::vector<double> v;
    FILE *f = fopen(p, "rb");
    double x;
    while (f && fread(&x, 8, 1, f) == 1) v.push_back(x);
    if (f) fclose(f);
    return v;
}
static double *upload(const std::vector<double> &v) {
    double *p = nullptr;
    if (cudaMalloc(&p, v.size() * 8) != cudaSuccess ||
        cudaMemcpy(p, v.data(), v.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
    return p;
}
int main(int, char **a) {
    const std::vector<double> cdf = read(a[1]), in = read(a[2]);
    const bool math = cdf.size() < 2;  // no CDF: the functions
    const int m = (int)in.size() / (math ? 4 : 1);
    std::vector<double> out((math ? 6 : 3) * (size_t)m);
    double *dc = upload(cdf), *di = upload(in), *dout = upload(out);
    if (!dc || !di || !dout) return 2;
    if (math) k_math<<<(m + 127) / 128, 128>>>(di, m, dout);
    else k_reuse<<<(m + 127) / 128, 128>>>(dc, (int)cdf.size() - 1, di, m, dout);
    if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    FILE *g = fopen(a[3], "wb");
    const bool ok = g && fwrite(out.data(), 8, out.size(), g) == out.size();
    if (g) fclose(g);
    return ok ? 0 : 4;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    (d / "m.cu").write_text(DRIVER)
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"), str(d / "m.cu"), "-o", str(d / "m")], check=True)

    def run(a, b, width):
        np.asarray(a, np.float64).tofile(d / "a.bin")
        np.asarray(b, np.float64).tofile(d / "b.bin")
        subprocess.run([str(d / "m"), str(d / "a.bin"), str(d / "b.bin"), str(d / "o.bin")], check=True)
        return np.fromfile(d / "o.bin").reshape(-1, width)

    return run


@pytest.mark.parametrize("n", [1, 2, 3, 1000])
def test_cdf_reuse_rounds_once(program, n):
    rng = np.random.default_rng(n)
    w = np.exp(rng.uniform(-8, 0, n))
    cdf = np.concatenate([[0.0], np.cumsum(w) / w.sum()])
    cdf[-1] = 1.0
    u = rng.uniform(0, 1, 20001)
    u[:2] = [0.0, np.nextafter(1.0, 0.0)]
    o = program(cdf, u, 3)
    idx = np.clip(np.searchsorted(cdf, u, side="left") - 1, 0, n - 1)
    pdf = cdf[idx + 1] - cdf[idx]
    assert np.array_equal(o[:, 0].astype(int), idx)
    assert np.array_equal(o[:, 2], pdf)
    assert np.array_equal(o[:, 1], (u - cdf[idx]) / pdf)


def test_math_keeps_the_bounds_of_the_host_build(program):
    rng = np.random.default_rng(3)
    n = 20000
    x = np.exp(rng.uniform(-300, 300, n)) * rng.choice([-1.0, 1.0], n)
    x[: n // 2] = rng.uniform(-4, 4, n // 2)
    # the ends of the FP32 seeds' range, 2^-125 to 2^125, and the powers beside them
    ends = [s * 2.0 ** e * m for e in (-127, -126, -125, -124, 124, 125, 126, 127) for s in (1, -1)
            for m in (1.0, np.nextafter(1.0, 2.0), 1.5, np.nextafter(2.0, 1.0))]
    x[: len(ends)] = ends
    t = rng.uniform(0, np.pi, n)
    t[:11] = [0.0, np.pi, np.pi / 2, np.pi / 4, 3 * np.pi / 4, 1e-7, np.pi - 1e-7, 1e-12, 1e-300, 0.78539816, 2.35619449]
    o = program([0.0], np.stack([x, t, np.sin(t), np.cos(t)], 1), 6)
    eps = 2.0 ** -53
    # a seed off by 2^-21 at most leaves 2^-63 after the third-order step: the roundings remain, as on the host
    assert np.abs(o[:, 0] * x - 1).max() <= 5 * eps
    assert np.abs(o[:, 1] * np.sqrt(np.abs(x)) - 1).max() <= 6 * eps
    assert np.abs(o[:, 2] / np.sqrt(np.abs(x)) - 1).max() <= 6 * eps
    assert np.abs(o[:, 3] - np.sin(t)).max() <= 4 * eps and np.abs(o[:, 4] - np.cos(t)).max() <= 4 * eps
    assert np.abs(o[:, 5] - t).max() <= 8 * eps


def test_math_of_zero_and_not_finite(program):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7e308])
    o = program([0.0], np.stack([x, 0 * np.ones(7), np.zeros(7), np.ones(7)], 1), 6)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(o[:, 0], 1 / x)
        np.testing.assert_array_equal(o[:, 2], np.sqrt(np.abs(x)))
        np.testing.assert_array_equal(o[:, 1], 1 / np.sqrt(np.abs(x)))
    assert (o[:, 5] == 0).all()
