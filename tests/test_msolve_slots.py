"""The residual ring of the multi-shift solver on the CPU: from every position of a window, including
the first one, the kernels continue from a slot inside the ring."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rhmc-on-gpu_b200", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_previous_slot_stays_in_the_ring(tmp_path):
    src = tmp_path / "slots.cu"
    src.write_text('#include <cstdio>\n#include "solver.h"\n'
                   "int main() { for (int win = 8; win <= 16; win += 8) for (int m = 0; m <= win; m++)\n"
                   '  printf("%d %d %d\\n", win, m, rhmc::ms_prev_slot(m, win)); }\n')
    exe = tmp_path / "slots"
    subprocess.check_call(["nvcc", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)])
    rows = [tuple(map(int, line.split())) for line in subprocess.check_output([str(exe)], text=True).splitlines()]
    assert len(rows) == 9 + 17
    for win, m, slot in rows:
        assert slot == (m + win - 1) % win
