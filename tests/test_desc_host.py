"""Checks of scene descriptions that need no device (dtrt_gb300/csrc/dt_desc.h), compiled for the
host with checks of ranges and accesses: velocities that are all zero
move nothing, and a shape whose vertex count scene creation refuses is not read at all."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <climits>
#include <cstdio>
#include <vector>
#include "dt_desc.h"
int main() {
    for (int nder : {1, 3, 8})
        for (int nv : {1, 5}) {
            std::vector<float> vel((size_t)nv * 3 * (nder + 1), 0.f), nrm((size_t)nv * 3, 0.f);
            dtrt_shape_desc s{};
            s.num_vertices = nv;
            if (dt::shape_moves(s, nder)) return 1;  // no velocities
            s.velocities = vel.data();
            vel.back() = 1.f;  // the last normal velocity: read with normals only
            if (dt::shape_moves(s, nder)) return 2;
            s.normals = nrm.data();
            if (!dt::shape_moves(s, nder)) return 3;
            vel.back() = -0.f;
            if (dt::shape_moves(s, nder)) return 4;
            vel[(size_t)nv * 3 * nder - 1] = 1e-30f;
            if (!dt::shape_moves(s, nder)) return 5;
            for (int bad : {0, -1, -7, INT_MIN}) {
                s.num_vertices = bad;
                if (dt::shape_moves(s, nder)) return 6;
            }
        }
    puts("ok");
    return 0;
}
"""


def test_shape_moves(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is missing")
    (tmp_path / "d.cpp").write_text(DRIVER)
    exe = str(tmp_path / "d")
    subprocess.run(["g++", "-std=c++17", "-D_GLIBCXX_DEBUG", "-fsanitize=address", "-I",
                    os.path.join(ROOT, "dtrt_gb300", "csrc"), str(tmp_path / "d.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
