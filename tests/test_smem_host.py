"""Shared-memory opt-ins of the walk kernels, on the host: one per kernel and
device, made again after a failure; block widths that fit."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <vector>
#include "sph3_smem.h"
int main() {
    using namespace sph3;
    SmemOptIn s;
    int a, b, fail = 1;
    std::vector<std::pair<const void *, int>> calls;
    auto ok = [&](const void *k, int bytes) { calls.push_back({k, bytes}); return 0; };
    if (s.once(0, &a, ok) || s.once(0, &a, ok) || calls.size() != 1) return 1;
    if (s.once(1, &a, ok) || calls.size() != 2) return 2;  // the same kernel on a second device
    if (s.once(1, &b, ok) || s.once(0, &b, ok) || calls.size() != 4) return 3;
    for (auto &c : calls) if (c.second != (int)kMaxBlockSmem) return 4;
    auto bad = [&](const void *, int) { return fail; };
    int c;
    if (s.once(0, &c, bad) != 1 || s.once(0, &c, bad) != 1) return 5;  // a failure is reported and not remembered
    fail = 0;
    if (s.once(0, &c, bad) != 0) return 6;
    for (size_t bytes : {size_t(1), size_t(25600), size_t(25601), size_t(51201), size_t(204800)})
        for (int w = 8; w >= 1; w /= 2) {
            const int f = warps_that_fit(w, bytes);
            if (f > w || f * bytes > kMaxBlockSmem || (f < w && 2 * f * bytes <= kMaxBlockSmem)) return 7;
        }
    return 0;
}
"""


def test_opt_ins(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "sph_3_b200", "csrc"), "-o", str(exe), str(src),
                    "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.parametrize("name", ["sph3_walk_sph.cu", "sph3_walk_grav.cu"])
def test_launchers_use_it(name):
    with open(os.path.join(ROOT, "sph_3_b200", "csrc", name)) as f:
        text = f.read()
    assert "cudaFuncSetAttribute" not in text and "allow_smem(" in text
