"""The list of row exchanges that wait for the next launch: a job beyond its places
is counted, so that the launch refuses the list, and writes nothing past them."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lu2_b200", "csrc")
NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)

PROGRAM = r"""
#include "lu2gpu_internal.cuh"
using namespace lu2gpu;
int main()
{
    struct {
        SwapJobs jobs;
        int after = 1234567;
    } s;
    for (int i = 0; i < SWAP_JOBS; i++) s.jobs.add(i, i + 1, i, i + 1);
    if (s.jobs.n != SWAP_JOBS) return 1;
    for (int i = 0; i < 3; i++) s.jobs.add(70, 80, 70, 80);
    return !(s.jobs.n == SWAP_JOBS + 1 && s.after == 1234567 && s.jobs.j[SWAP_JOBS - 1].k0 == SWAP_JOBS - 1);
}
"""


@pytest.mark.skipif(NVCC is None, reason="no nvcc")
def test_a_job_beyond_the_last_place(tmp_path):
    src = tmp_path / "jobs.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "jobs"
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, "-o", str(exe),
                    str(src)], check=True, capture_output=True, text=True)
    assert subprocess.run([str(exe)]).returncode == 0
