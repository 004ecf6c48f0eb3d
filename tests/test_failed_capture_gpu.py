"""A capture of periods that fails (the stream is already being captured) leaves the
domain as it was: its step count, its fields, and that its halos are behind."""
import numpy as np
import pytest

from test_scatter_gather_gpu import padded

pytestmark = pytest.mark.gpu


def test_failed_capture_leaves_the_state(b2r):
    import torch
    env, blocks, R = (64, 64, 64), (2, 2, 2), 4
    rng = np.random.default_rng(5)
    dom = (rng.random(env[::-1]) < 0.3).astype(np.uint8)
    s = torch.cuda.Stream()
    kw = dict(blocks=blocks, R=R, boundary=b2r.BC_PERIODIC, stream=s)
    with b2r.Domain(b2r.MODEL_GOL, env, **kw) as d, b2r.Domain(b2r.MODEL_GOL, env, **kw) as ref:
        for x in (d, ref):
            x.upload(dom)
            x.step(200)                       # on the bit grid: the halos are left behind
            x.set_tuning(gol_push=1)          # block passes, whole periods from graphs
            x.synchronize()
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=s):
            with pytest.raises(b2r.B2RError):
                d.step(64)
        assert d.time_step == 200
        want = padded(d.download(), env, blocks, R, 0, True)
        for key, got in d.download_blocks().items():
            assert np.array_equal(got, want[key]), key
        for x in (d, ref):
            x.step(66)
        assert np.array_equal(d.download(), ref.download()) and d.time_step == 266
