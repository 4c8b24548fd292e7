"""How the blocks of a shared-step run kernel report a launch
(assist_gb300/csrc/run_ctl.h, plain C++): whatever the order in which the
blocks' last words arrive, a block that stopped waiting is seen by the host
and block 0's state is what the host reads."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "run_ctl.h"
#include <algorithm>
#include <cstdio>
int main() {
    int bad = 0, order[3] = {0, 1, 2};
    do for (int who = -1; who < 3; who++) {
        ShRunMem m = {};
        for (int b : order) {
            ShCtl K = {};
            K.t = 100.0 + b;
            sh_run_report(K, b == who, b, &m.ctl[1], &m.gave_up);
        }
        if (m.ctl[1].t != 100.0 || (m.gave_up != 0) != (who >= 0)) bad++;
    } while (std::next_permutation(order, order + 3));
    std::printf("bad %d\n", bad);
    return bad != 0;
}
"""


def test_a_block_that_gave_up_is_reported(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "run.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "run"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "assist_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
