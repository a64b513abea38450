"""Device buffers of a render when the device is full (dtrt_gb300/csrc/dt_buffers.h), compiled for
the host against a fake allocator of a fixed size: density cells, which a render can do
without, give way to what it needs, and a wavefront that does not fit in all its lanes runs in
one before it is given up."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"

DRIVER = r"""
#include "dt_buffers.h"
#include <cstdio>
#include <cstdlib>
#include <map>
using namespace dt;
static std::map<void *, size_t> live;
static size_t room = 0, used = 0;
static bool error = false;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (used + n > room) { error = true; return cudaErrorMemoryAllocation; }
    *p = malloc(1);
    live[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (!live.count(p)) abort();
    used -= live[p];
    live.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { error = false; return cudaSuccess; }
}
struct Buf { void *p = nullptr; size_t n = 0; };
static Buf cells, state, queue;
static bool ensure(Buf &b, size_t n) { return grow_buffer(&b.p, &b.n, n, &cells.p, &cells.n) == cudaSuccess; }
static int wave(int lanes, size_t per_state, size_t per_queue) {
    return fit_lanes(lanes, [&](int k) { return ensure(state, k * per_state) && ensure(queue, k * per_queue); },
                     [&] {
                         for (Buf *b : {&state, &queue}) { if (b->p) cudaFree(b->p); *b = Buf(); }
                     });
}
int main() {
    room = 100000;
    if (!ensure(cells, 60000) || !ensure(state, 10) || state.n != 256 || used != 60256) return 1;
    if (!ensure(state, 200) || used != 60256) return 2;                    // large enough already
    if (!ensure(state, 50000) || cells.p || cells.n || used != 50000) return 3;  // the cells gave way
    if (ensure(cells, 60000) || cells.p || used != 50000) return 4;        // cells that do not fit free nothing else
    cudaGetLastError();
    if (wave(8, 10000, 2000) != 8 || used != 96000) return 5;
    if (wave(8, 11000, 2000) != 1 || used != 13000 || error) return 6;     // states of 8 lanes fit, their queues do not
    if (!ensure(cells, 80000) || wave(8, 11000, 1000) != 8 || cells.p) return 7;  // lanes before cells
    if (wave(8, 99000, 2000) != 0 || used != 0 || error) return 8;         // not even one: all given back
    if (wave(1, 99000, 2000) != 0 || wave(1, 90000, 2000) != 1) return 9;
    puts("ok");
    return 0;
}
"""


def test_a_full_device(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    (tmp_path / "d.cpp").write_text(DRIVER)
    exe = str(tmp_path / "d")
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"),
                    str(tmp_path / "d.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)
