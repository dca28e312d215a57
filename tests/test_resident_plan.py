"""The resident CG's plans on the host: which CTA holds which rows, and the split of a share's slots over
its warps (tests/support/resident_plan.cpp restates the kernel's index arithmetic)."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opensurgsim_gb300", "csrc")


def test_plans_and_slot_splits(tmp_path):
    from opensurgsim_gb300 import build

    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "resident_plan")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-I" + CSRC, "-I" + cuda, "-o", exe,
                    os.path.join(ROOT, "tests", "support", "resident_plan.cpp"), os.path.join(CSRC, "gbfem_plan.cpp")],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "plan ok", out.stdout + out.stderr
