"""The prefix sum's kernels take their parameters from constant memory: compiled
for sm_100a they need no stack (a parameter block indexed at run time would be
copied to every thread's)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include "scan.cuh"
void both(int *a, long long *b, int n, cudaStream_t st)
{
    mps::scan_exclusive2<int>(a, a, n, a, a, n, a, st);
    mps::scan_exclusive<long long>(b, b, n, b, st);
}
'''


def test_kernels_need_no_stack(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "scan.cu"
    src.write_text(SOURCE)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xptxas", "-v",
                        "-I" + os.path.join(ROOT, "mps_b200", "csrc"), "-c", "-o", str(tmp_path / "scan.o"), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = [int(x) for x in re.findall(r"(\d+) bytes stack frame", r.stderr)]
    assert len(frames) >= 4 and not any(frames), r.stderr
