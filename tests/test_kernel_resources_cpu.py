"""What ptxas reports of kernels whose speed on small grids hangs on it (no GPU)."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not shutil.which(NVCC), reason="no nvcc")
def test_row_pass_without_run_time_radix_has_no_stack():
    """The run-time radix keeps a local array of 31 elements; only the instance of the lengths that
    need it may have one."""
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xptxas", "-v",
                        "-c", os.path.join(CSRC, "mixed.cu"), "-o", os.devnull], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = re.findall(r"Function properties for \S*mr_rows_kernel\S*\s+(\d+) bytes stack frame, (\d+) bytes spill",
                        r.stdout + r.stderr)
    assert sorted(int(a) == 0 for a, _ in frames) == [False, True], frames
    assert all(int(b) == 0 for _, b in frames)
