"""FP64 arithmetic of the edge kernels as the device runs it, in a small program of its own: the reuse
of a CDF's random number is the correctly rounded quotient."""
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
    const int m = (int)in.size();
    std::vector<double> out(3 * (size_t)m);
    double *dc = upload(cdf), *di = upload(in), *dout = upload(out);
    if (!dc || !di || !dout) return 2;
    k_reuse<<<(m + 127) / 128, 128>>>(dc, (int)cdf.size() - 1, di, m, dout);
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
