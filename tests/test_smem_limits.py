"""The table of raised shared-memory limits: one entry per device and kernel,
only ever raised, and only remembered when the call that raises it succeeded.
"""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fortran_airtools_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "smem_limits.h"
int main() {
    fair::SmemLimits t;
    int k1 = 0, k2 = 0, calls = 0, status = 0;
    auto raise = [&] { ++calls; return status; };
    auto step = [&](int dev, const int *k, size_t bytes, int want_calls, int want_status) {
        calls = 0;
        const int got = t.allow(dev, k, bytes, raise);
        if (calls != want_calls || got != want_status) {
            printf("device %d, %zu bytes: %d calls, status %d\n", dev, bytes, calls, got);
            return 1;
        }
        return 0;
    };
    int bad = 0;
    bad += step(0, &k1, 100, 1, 0);
    bad += step(0, &k1, 100, 0, 0);
    bad += step(0, &k1, 50, 0, 0);   // not lowered
    bad += step(1, &k1, 50, 1, 0);   // another device's limit is its own
    bad += step(0, &k2, 50, 1, 0);
    status = 1;
    bad += step(0, &k1, 200, 1, 1);  // refused: the old limit stands
    status = 0;
    bad += step(0, &k1, 200, 1, 0);
    bad += step(0, &k1, 100, 0, 0);
    bad += step(1, &k1, 100, 1, 0);
    return bad;
}
"""


def test_limits_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
