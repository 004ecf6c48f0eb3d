"""Many steps of a heat domain of several blocks, or on a torus, run on the
domain as one block: the same bits as the blocks with their exchanges, with
steps of the block kernels before, between and after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# three subdomains on an axis, rows that end inside a float4, an axis of the
# torus as short as its halo, one block on a torus, a live shell
@pytest.mark.parametrize("env,blocks,R,D,periodic", [
    ((48, 40, 32), (2, 2, 1), 2, 1, False), ((39, 34, 27), (3, 1, 3), 1, 2, False), ((66, 30, 46), (2, 3, 1), 1, 4, False),
    ((37, 31, 29), (1, 1, 1), 1, 1, True), ((50, 22, 26), (2, 1, 1), 2, 2, True), ((35, 16, 17), (1, 1, 1), 1, 4, True),
    ((33, 8, 90), (1, 1, 2), 1, 3, True), ((244, 104, 168), (2, 2, 2), 4, 1, False),
    ((130, 63, 70), (2, 3, 1), 1, 1, False), ((100, 62, 81), (1, 2, 3), 2, 2, False), ((90, 75, 64), (2, 1, 1), 2, 1, True),
    ((77, 83, 65), (1, 1, 1), 1, 2, True)])
def test_joined_equals_blocks(b2r, env, blocks, R, D, periodic):
    import torch
    rng = np.random.default_rng(71)
    dom = rng.random(env[::-1] if periodic else tuple(e + 2 * D for e in env[::-1]), dtype=np.float32)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    outs = []
    for knobs in (None, dict(tblock=1)):     # a knob keeps to the blocks
        s = torch.cuda.Stream()
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02, dz=0.9, boundary=bc, stream=s) as d:
            if knobs:
                d.set_tuning(**knobs)
            d.upload(dom)
            got = []
            for n in (3, 20, 1, 33, 2, 21):  # pieces that leave and meet a period in its middle
                d.step(n)
                got.append(d.download())
            d.upload(dom * np.float32(0.5))  # another shell too
            d.step(40)
            got.append(d.download())
            assert d.time_step == 40
            d.synchronize()
            outs.append(got)
    for k, (a, b) in enumerate(zip(*outs)):
        assert np.array_equal(a, b), k
