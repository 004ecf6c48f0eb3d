"""Which kernels the default schedule takes, by the launches it counts: tests that
compare the default with the blocks would pass as well if both ran the blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def launches(b2r, d, n):
    d.synchronize()
    before = b2r.kernel_launches()
    d.step(n)
    return b2r.kernel_launches() - before


def heat(b2r, env, blocks, R, D, periodic):
    d = b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02,
                   boundary=b2r.BC_PERIODIC if periodic else b2r.BC_SHELL)
    d.upload(np.random.default_rng(1).random(d.domain_shape, dtype=np.float32))
    return d


# the sizes of test_heat_small_gpu.py that gain by it
@pytest.mark.parametrize("env,blocks,R,D,periodic", [
    ((48, 40, 32), (2, 2, 1), 2, 1, False), ((30, 45, 51), (3, 1, 3), 2, 1, False), ((16, 20, 18), (2, 2, 1), 1, 2, False),
    ((40, 33, 32), (2, 1, 1), 1, 1, True), ((35, 2, 2), (1, 1, 1), 1, 1, True), ((4, 4, 18), (1, 1, 1), 1, 2, True),
    ((2, 21, 41), (1, 3, 1), 1, 1, True), ((37, 13, 21), (1, 1, 1), 1, 2, True), ((18, 12, 48), (1, 2, 3), 1, 2, True),
    ((48, 40, 32), (1, 1, 1), 1, 1, False), ((47, 40, 32), (1, 1, 1), 1, 2, False)])
def test_cluster(b2r, env, blocks, R, D, periodic):
    with heat(b2r, env, blocks, R, D, periodic) as d:
        assert launches(b2r, d, 40) == 1


# steps per pass of the one-block form, and between its exchanges
@pytest.mark.parametrize("env,blocks,R,D,periodic,per_pass,period", [
    ((130, 63, 70), (2, 3, 1), 1, 1, False, 2, 0), ((100, 62, 81), (1, 2, 3), 2, 2, False, 1, 0),
    ((66, 30, 46), (2, 3, 1), 1, 4, False, 1, 0), ((90, 75, 64), (2, 1, 1), 2, 1, True, 2, 4),
    ((77, 83, 65), (1, 1, 1), 1, 2, True, 1, 3), ((35, 36, 37), (1, 1, 1), 1, 4, True, 1, 2),
    ((256, 200, 180), (2, 2, 2), 4, 1, False, 3, 0), ((300, 160, 170), (2, 1, 1), 1, 1, True, 3, 3)])
def test_one_block(b2r, env, blocks, R, D, periodic, per_pass, period):
    with heat(b2r, env, blocks, R, D, periodic) as d:
        n = 24
        assert launches(b2r, d, n) == 2 + n // per_pass + (n // period if period else 0)   # join, split; passes; exchanges


def test_several_steps_per_pass(b2r):
    with heat(b2r, (256, 200, 180), (1, 1, 1), 1, 1, False) as d:
        assert launches(b2r, d, 24) == 8
    with heat(b2r, (128, 128, 128), (1, 1, 1), 1, 1, False) as d:
        assert launches(b2r, d, 24) == 12


@pytest.mark.parametrize("model,R", [("EQWP_STAG", 2), ("EQWP_REF", 1)])
def test_wave_as_one_block(b2r, model, R):
    with b2r.Domain(getattr(b2r, "MODEL_" + model), (48, 40, 32), blocks=(2, 2, 1), R=R, D=2, dt=2e-4, h=1.0,
                    src=(3, 4, 5)) as d:
        assert launches(b2r, d, 24) == 2 + 2 * 24


def test_life_on_the_bit_grid(b2r):
    with b2r.Domain(b2r.MODEL_GOL, (64, 64, 64), blocks=(2, 2, 2), R=4, boundary=b2r.BC_PERIODIC) as d:
        assert launches(b2r, d, 24) == 2 + 24 // 8
