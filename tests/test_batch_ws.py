"""The workspace of a batch on two kernels (assist_gb300/csrc/batch_ws.h, plain
C++): both kernels' slots fit, apart from each other, also when all groups are
deep and the other kernel has none."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "batch_ws.h"
#include <cstdio>
int main() {
    int bad = 0;
    const size_t per[2] = {40 * 3, 40 * 21};
    const int slots[5] = {0, 32, 224, 9728, 14592};
    for (size_t p : per) for (int a : slots) for (int d : slots) {
        const AgBatchWs w = ag_batch_ws(p, a, d);
        if (w.deep_at < p * a || w.total < w.deep_at + p * d) bad++;
    }
    std::printf("bad %d\n", bad);
    return bad != 0;
}
"""


def test_both_kernels_slots_fit(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "ws.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "ws"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "assist_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
