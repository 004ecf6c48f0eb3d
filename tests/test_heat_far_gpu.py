"""One heat step per pass with a producer warp (the default of radius 2..4, and
of radius 1 where a pass takes one step): the same bits as the sweep that the
launch-schedule knobs select, where its tiles (128 x 30, 22 or 14 cells), z
chunks and ring have edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a domain smaller than a tile and than the ring's planes; one column and row
# more than a tile of each height; many tiles of the smallest height (two CTAs
# per SM), and the largest of the three heights; subdomains with deep halos;
# tori
@pytest.mark.parametrize("env,blocks,R,periodic", [
    ((9, 8, 10), (1, 1, 1), 1, False), ((129, 31, 5), (1, 1, 1), 1, False), ((128, 23, 67), (1, 1, 1), 2, False),
    ((257, 15, 40), (1, 1, 1), 1, False), ((200, 190, 96), (1, 1, 1), 1, False), ((96, 66, 48), (2, 2, 1), 2, False),
    ((66, 58, 34), (2, 1, 2), 2, True), ((131, 30, 33), (1, 1, 1), 3, True)])
@pytest.mark.parametrize("D", [1, 2, 3, 4])
def test_far_equals_sweep(b2r, env, blocks, R, periodic, D):
    if R * D > min(e // b for e, b in zip(env, blocks)) // 2:
        pytest.skip("R*D <= min(B)/2 (b2r.cpp:54)")
    rng = np.random.default_rng(53)
    dom = rng.random(env[::-1] if periodic else tuple(e + 2 * D for e in env[::-1]), dtype=np.float32)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    outs = []
    for knobs in (None, dict(tblock=1)):
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02, dz=0.9, boundary=bc) as d:
            if knobs:
                d.set_tuning(**knobs)
            d.upload(dom)
            for n in (1, 4, 2):      # pieces that start and end inside periods
                d.step(n)
            outs.append(d.download())
            d.synchronize()
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("D", [1, 2, 3, 4])
def test_far_matches_oracle(b2r, orc, D):
    env = (70, 45, 41)
    rng = np.random.default_rng(54)
    dom = rng.random(tuple(e + 2 * D for e in env[::-1]), dtype=np.float32)
    with b2r.Domain(b2r.MODEL_HEAT, env, D=D, alpha_dt=0.02) as d:
        d.upload(dom)
        for _ in range(9):
            d.step(1)
        got = d.download()
        d.synchronize()
    ref = dom.copy()
    orc.heat_run(ref, D, D, 9, 0.02, 1.0, 1.0, 1.0)
    assert np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref) <= 1e-5
