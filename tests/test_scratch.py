"""The scratch that grows with the calls (fjg_scratch.cu), on a device of limited
memory that a host program (tests/scratch_check.cu) plays (CPU only; needs nvcc)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    return None


def test_workspace_of_the_rounds_is_optional(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "scratch_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "fastjet_gpu_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "scratch_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True, timeout=600)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.startswith("ok"), res.stdout + res.stderr
