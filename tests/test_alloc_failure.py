"""Allocations that fail half-way, on the host: csrc/k_pme.cu and csrc/k_list.cu
compiled with fakes of the runtime's calls (tests/alloc_*.cu).  What is half
built is not taken for complete by the next call."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc is needed to compile the sources")
@pytest.mark.parametrize("what", ["plan", "list"])
def test_half_built_is_built_again(what, tmp_path):
    src = os.path.join(os.path.dirname(HERE), "orac-porting_b200", "csrc")
    exe = str(tmp_path / what)
    subprocess.run([NVCC, "-std=c++17", "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", src, "-I", HERE, "-I",
                    os.path.join(src, "..", "..", "include"), "-o", exe, os.path.join(HERE, f"alloc_{what}.cu")],
                   check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
