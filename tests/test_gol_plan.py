"""The search for a Game-of-Life pass's tile, compiled with nvcc and run on the host:
it finds the best by its own model (gol_plan_check.cu); and the first run of a new
domain does not wait for it where that size is known."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_plan_is_the_best_tile(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "gol_plan_check")
    cmd = [nvcc, "-std=c++17", "-O3", "-I", os.path.join(ROOT, "b2r_gb300", "csrc"),
           os.path.join(HERE, "gol_plan_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
def test_first_run_of_a_known_size_is_no_slower(b2r):
    """Host time of a first and a second run of 17 generations on fresh domains: the
    search (0.3 ms through every tile) is done once per size."""
    import time
    firsts, seconds = [], []
    for _ in range(12):
        with b2r.Domain(b2r.MODEL_GOL, (256, 256, 256), blocks=(2, 2, 2), R=4, boundary=b2r.BC_PERIODIC) as d:
            d.upload(np.zeros(d.domain_shape, np.uint8))
            d.synchronize()
            for ts in (firsts, seconds):
                t = time.perf_counter()
                d.step(17)
                ts.append(time.perf_counter() - t)
                d.synchronize()
    assert min(firsts[1:]) <= min(seconds) + 50e-6, (min(firsts[1:]), min(seconds))
