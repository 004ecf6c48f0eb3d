"""Launch grids of the elastic-wave stages on domains of many blocks, compiled with
nvcc and run on the host (stage_grid_check.cu)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_stage_grids_can_be_launched(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "stage_grid_check")
    cmd = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
           os.path.join(ROOT, "b2r_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(HERE, "stage_grid_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
