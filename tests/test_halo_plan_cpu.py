"""What the direct convolution's kernel takes for granted, over some ten thousand plans, on the CPU (halo_plan() is host code)."""
import importlib
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_plans_hold_what_the_kernel_assumes(tmp_path):
    pkg = Path(importlib.import_module("deep-learning-math-kernel-research_b200").__file__).parent
    objects = sorted((pkg / "build").glob("*.o"))
    if not objects or not shutil.which("nvcc"):
        pytest.skip("needs nvcc and the library's objects")
    exe = tmp_path / "halo_plan_check"
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", f"-I{pkg / 'csrc'}", "-o", str(exe),
                           str(ROOT / "tests" / "native" / "halo_plan_check.cu")] + [str(o) for o in objects])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]
