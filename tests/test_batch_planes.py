"""The batches' own rule for planes per unit: it picks no length whose work queue
is too long where a longer unit's is not (batch_planes.h, compiled with nvcc and
run on the host), and such batches are accepted on the GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_planes_rule(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "batch_planes_check")
    cmd = [nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "b2r_gb300", "csrc"),
           os.path.join(HERE, "batch_planes_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
def test_long_heat_batch_is_accepted(b2r):
    # 12 x 2000000 rounds: 12 units of two planes each, 2 of 16
    with b2r.Batch([dict(env=(24, 24, 24), D=1, nsteps=2000000)] * 12) as bt:
        assert bt.lups == 12 * 24 ** 3 * 2000000


@pytest.mark.gpu
def test_long_elastic_batch_is_accepted(b2r):
    # 4000 planes and 840000 rounds: 334 units of 12 planes a round, 125 of 32
    with b2r.Domain(b2r.MODEL_EQWP_STAG, (8, 8, 4000), D=2, dt=2e-4, h=1.0, src=(3, 4, 5)) as d:
        with b2r.EqwpBatch([d], [420000]) as bt:
            assert bt.lups == 8 * 8 * 4000 * 420000
