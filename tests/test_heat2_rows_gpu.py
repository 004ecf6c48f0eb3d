"""Radius-1 heat, two steps per pass in two-row tiles, where its units have
edges: rows of 120 cells, 121 to 128 (one tile column without halo lanes when
both faces are fixed) and 129, z chunks of one plane, tile rows with one cell
in the last: the same bits as one step per pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [120, 121, 124, 127, 128, 129])
@pytest.mark.parametrize("ny,nz,blocks,R,periodic", [
    (14, 5, (1, 1, 1), 1, False), (29, 33, (1, 1, 1), 2, False), (58, 22, (1, 2, 2), 2, False), (30, 26, (1, 1, 2), 4, True)])
def test_two_steps_equal_one_step_per_pass(b2r, nx, ny, nz, blocks, R, periodic):
    rng = np.random.default_rng(17)
    env = (nx, ny, nz)
    dom = rng.random(env[::-1] if periodic else tuple(e + 2 for e in env[::-1]), dtype=np.float32)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    outs = []
    for knobs in ({}, dict(tblock=2, zchunk2=3), dict(tblock=1)):
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=1, alpha_dt=0.1, dy=1.1, boundary=bc) as d:
            if knobs:
                d.set_tuning(**knobs)
            d.upload(dom)
            for n in (1, 4, 13):    # pieces that leave and meet a period in its middle
                d.step(n)
            outs.append(d.download())
            d.synchronize()
    assert np.array_equal(outs[0], outs[2]) and np.array_equal(outs[1], outs[2])
