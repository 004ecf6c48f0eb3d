"""Heat on small domains, whole runs in the shared memory of one cluster: the
same bits as steps through the blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one CTA and sixteen, slabs of one plane more in some, rows that end inside a
# float4, one float4 per row, axes as short as the halo allows, one to four
# planes per thread, several blocks, tori (an axis that wraps both ways at once)
@pytest.mark.parametrize("env,blocks,R,D,periodic", [
    ((48, 40, 32), (2, 2, 1), 2, 1, False), ((33, 17, 2), (1, 1, 1), 1, 1, False), ((6, 5, 37), (1, 1, 1), 1, 1, False),
    ((129, 8, 31), (1, 1, 1), 1, 1, False), ((30, 45, 51), (3, 1, 3), 2, 1, False), ((47, 40, 32), (1, 1, 1), 1, 2, False),
    ((16, 20, 18), (2, 2, 1), 1, 2, False), ((40, 33, 32), (2, 1, 1), 1, 1, True), ((35, 2, 2), (1, 1, 1), 1, 1, True),
    ((4, 4, 18), (1, 1, 1), 1, 2, True), ((2, 21, 41), (1, 3, 1), 1, 1, True), ((37, 13, 21), (1, 1, 1), 1, 2, True), ((18, 12, 48), (1, 2, 3), 1, 2, True)])
def test_small_equals_blocks(b2r, env, blocks, R, D, periodic):
    import torch
    rng = np.random.default_rng(29)
    dom = rng.random(env[::-1] if periodic else tuple(e + 2 * D for e in env[::-1]), dtype=np.float32)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    outs = []
    for knobs in (None, dict(tblock=1)):     # a knob keeps to the blocks
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02, dz=0.9, boundary=bc,
                        stream=torch.cuda.Stream()) as d:
            if knobs:
                d.set_tuning(**knobs)
            d.upload(dom)
            got = []
            for n in (3, 20, 1, 33, 2, 21):  # pieces that leave and meet a period in its middle
                d.step(n)
                got.append(d.download())
            d.upload(dom * np.float32(0.5))  # another shell too
            d.step(2100)                     # more than a launch takes
            got.append(d.download())
            assert d.time_step == 2100
            d.synchronize()
            outs.append(got)
    for k, (a, b) in enumerate(zip(*outs)):
        assert np.isfinite(a).all() and np.array_equal(a, b), k
