"""Side streams of a render (dtrt_gb300/csrc/dt_lanes.h), compiled for the host against a fake of
the runtime that logs its calls and can fail one of them: every stream that was forked joins
the main stream again, also when a launch in between fails or a render gives up."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"

DRIVER = r"""
#include "dt_lanes.h"
#include <cstdio>
#include <set>
#include <string>
#include <vector>
using namespace dt;
static std::vector<std::string> calls;
static int fail_at = -1, made = 0;
static cudaError_t note(const std::string &s) {
    calls.push_back(s);
    return (int)calls.size() - 1 == fail_at ? cudaErrorUnknown : cudaSuccess;
}
static std::string id(const void *p) { return std::to_string((size_t)p); }
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)(size_t)(100 + made++); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)(size_t)(200 + made++); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { --made; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { --made; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return note("rec " + id(e) + " " + id(s)); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return note("wait " + id(s) + " " + id(e)); }
}
// the main stream (1) waits for an event recorded on side stream k after its last work
static bool joined(const Lanes &sb, int k) {
    size_t last = 0;
    for (size_t i = 0; i < calls.size(); ++i)
        if (calls[i] == "work " + id(sb.side[k])) last = i + 1;
    for (size_t i = last; i < calls.size(); ++i)
        if (calls[i] == "rec " + id(sb.side_ev[k]) + " " + id(sb.side[k]))
            for (size_t j = i; j < calls.size(); ++j)
                if (calls[j] == "wait 1 " + id(sb.side_ev[k])) return true;
    return false;
}
static int render(Lanes &sb, bool give_up) {
    SideWork w(sb, (cudaStream_t)1);
    if (w.fork() != cudaSuccess) return 1;
    note("work " + id(w.stream()));
    if (give_up) return 2;
    return w.join() == cudaSuccess && !w.open() ? 0 : 3;
}
int main() {
    Lanes sb;
    if (!ensure_lanes(sb, kLanes)) return 1;
    // a render that ends, one that gives up, one that never forks
    calls.clear();
    if (render(sb, false) || calls.size() != 5 || !joined(sb, 0)) return 2;
    calls.clear();
    if (render(sb, true) != 2 || !joined(sb, 0)) return 3;
    calls.clear();
    { SideWork w(sb, (cudaStream_t)1); }
    if (!calls.empty()) return 4;
    // batches over the lanes: each in turn, and all joined when one fails
    for (int bad = -1; bad < 5; ++bad) {
        calls.clear();
        std::vector<int> seen;
        cudaError_t e = in_lanes(sb, (cudaStream_t)1, 4, 5, [&](long long k, int lane, cudaStream_t q) {
            if (lane != k % 4 || q != (lane ? sb.side[lane - 1] : (cudaStream_t)1)) return cudaErrorInvalidValue;
            seen.push_back((int)k);
            note("work " + id(q));
            return (int)k == bad ? cudaErrorUnknown : cudaSuccess;
        });
        if ((e != cudaSuccess) != (bad >= 0) || (int)seen.size() != (bad >= 0 ? bad + 1 : 5)) return 5;
        for (int k = 0; k < 3; ++k)
            if (!joined(sb, k)) return 6;
    }
    free_lanes(sb);
    if (made != 0 || sb.fork_ev || sb.side[0]) return 7;
    puts("ok");
    return 0;
}
"""


def test_forked_streams_join(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    (tmp_path / "d.cpp").write_text(DRIVER)
    exe = str(tmp_path / "d")
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"),
                    str(tmp_path / "d.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)


LANES = r"""
#include "dt_lanes.h"
#include <cstdio>
using dt::lanes_for;
int main() {
    const long long P = 1ll << 20;
    // as planned: up to 8 batches of 2^20 paths
    if (lanes_for(1, P, 8, 8 * P) != 1 || lanes_for(3, P, 8, 8 * P) != 3 || lanes_for(99, P, 8, 8 * P) != 8) return 1;
    if (lanes_for(0, 1, 8, 8 * P) != 1) return 2;  // nothing to render
    // one pixel with more samples than a batch was meant to hold
    if (lanes_for(4, 1ll << 24, 8, 8 * P) != 1 || lanes_for(4, 1ll << 22, 8, 8 * P) != 2) return 3;
    for (long long b = 1; b < (1ll << 26); b = b * 3 + 1)
        for (long long n : {0ll, 1ll, 2ll, 7ll, 8ll, 1000ll}) {
            const int k = lanes_for(n, b, 8, 8 * P);
            if (k < 1 || k > 8 || (k > 1 && (k * b > 8 * P || k > n))) return 4;
        }
    puts("ok");
    return 0;
}
"""


def test_lanes_are_bounded_by_their_paths(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    # the functions that call the runtime are linked against nothing: only lanes_for is used
    (tmp_path / "d.cpp").write_text(LANES)
    exe = str(tmp_path / "d")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CUDA_INC, "-I", os.path.join(ROOT, "dtrt_gb300", "csrc"),
                    str(tmp_path / "d.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)
