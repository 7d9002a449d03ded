"""A plan of the reciprocal sum whose allocation fails half-way is not taken for
complete by the next call (tests/plan_alloc.cu, on the host with a fake of the
allocation call)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc is needed to compile the plan's source")
def test_half_built_plan_is_laid_out_again(tmp_path):
    src = os.path.join(os.path.dirname(HERE), "orac-porting_b200", "csrc")
    exe = str(tmp_path / "plan_alloc")
    subprocess.run([NVCC, "-std=c++17", "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", src, "-I", os.path.join(src, "..", "..", "include"), "-o",
                    exe, os.path.join(HERE, "plan_alloc.cu")], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
