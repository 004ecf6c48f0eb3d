"""Radius-1 heat on large blocks, several steps per pass with four rows per
thread: the same bits as one step per pass, where its tiles (120 x 44, 120 x
46 and 120 x 26 cells), z chunks and fixed faces have edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks on both sides of the line to two rows per thread; rows of one tile, one
# cell more, and ragged float4s at the high face; periods of 2 (two steps per
# pass), 3, 4 (four) and 5 (three and two); tori
@pytest.mark.parametrize("env,blocks,R,periodic", [
    ((120, 88, 100), (1, 1, 1), 1, False), ((121, 89, 97), (1, 1, 1), 1, False), ((126, 40, 199), (1, 1, 1), 4, False),
    ((246, 91, 93), (2, 1, 1), 2, False), ((97, 268, 202), (1, 2, 2), 3, False), ((242, 104, 167), (2, 1, 1), 4, True),
    ((122, 133, 64), (1, 1, 1), 5, True), ((240, 132, 150), (1, 1, 1), 1, False), ((245, 177, 198), (1, 1, 1), 4, False),
    ((482, 132, 190), (2, 1, 1), 2, False), ((241, 268, 302), (1, 2, 2), 3, False),
    ((480, 176, 167), (2, 1, 1), 4, True), ((242, 133, 264), (1, 1, 1), 5, True)])
def test_rows_equal_one_step_per_pass(b2r, env, blocks, R, periodic):
    rng = np.random.default_rng(51)
    shape = env[::-1] if periodic else tuple(e + 2 for e in env[::-1])
    dom = rng.random(shape, dtype=np.float32)      # a shell that is not zero
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    outs = []
    for tblock in (None, 1):
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=1, alpha_dt=0.1, dz=0.9, boundary=bc) as d:
            if tblock:
                d.set_tuning(tblock=tblock)
            d.upload(dom)
            for n in (1, 7, 12):
                d.step(n)
            outs.append(d.download())
            d.synchronize()
    assert np.array_equal(outs[0], outs[1])


def test_rows_match_oracle(b2r, orc):
    env = (123, 95, 90)
    rng = np.random.default_rng(52)
    dom = rng.random(tuple(e + 2 for e in env[::-1]), dtype=np.float32)
    with b2r.Domain(b2r.MODEL_HEAT, env, D=1, alpha_dt=0.1) as d:
        d.upload(dom)
        d.step(10)
        got = d.download()
        d.synchronize()
    ref = dom.copy()
    orc.heat_run(ref, 1, 1, 10, 0.1, 1.0, 1.0, 1.0)
    rel = np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref)
    assert rel <= 1e-5
