"""The elastic-wave misfit gradient keeps the last segments of its forward and
replays the others: the same bits for every split of the steps into segments
(one, two, several with a remainder, one step each), the traces of a plain
record, the wavefield of plain steps, and receivers that share a cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env,n", [((21, 14, 9), 7), ((130, 16, 33), 11)])
def test_segments_change_nothing(b2r, env, n):
    import torch
    shape = tuple(e + 4 for e in env[::-1])
    rec = [(1, 2, 3), (env[0] - 1, 0, env[2] - 1), (1, 2, 3)]

    def domain(**kw):
        rng = np.random.default_rng(8)
        d = b2r.Domain(b2r.MODEL_EQWP_STAG, env, D=2, dt=2e-2, h=1.0, src=(4, 5, 6), stream=torch.cuda.Stream())
        for f, c in (("lambda", 3.0), ("mu", 2.0), ("buoy", 0.5)):
            d.upload(np.float32(c) + rng.random(shape, dtype=np.float32), field=f)
        d.set_source(rng.random(n, dtype=np.float32))
        f0 = [rng.random(shape, dtype=np.float32) - np.float32(0.5) for _ in range(9)]
        for k, f in enumerate(f0):
            d.upload(f, field=k)
        if kw:
            d.set_tuning(**kw)
        return d, f0

    d, _ = domain()
    with d:
        d.step(n)
        want = [d.download(field=f) for f in range(9)]
    d, _ = domain()
    with d:
        syn = d.eqwp_record(n, rec)
    obs = np.random.default_rng(1).random(syn.shape, dtype=np.float32)
    obs[:, 2] = obs[:, 0]   # equal residuals: their order of adding is free
    first = None
    for kw in ({}, dict(adj_fused=0), dict(eqwp_fused=1)):
        d, f0 = domain(**kw)
        with d:
            for K in (n, 0, n - 1, 4, 3, 2, 1):
                for k, f in enumerate(f0):
                    d.upload(f, field=k)
                J, g, s = d.eqwp_misfit_gradient(n, rec, obs, ckpt_every=K)
                assert np.array_equal(s, syn)
                for f in range(9):
                    assert np.array_equal(d.download(field=f), want[f]), (kw, K, f)
                if first is None:
                    first = (J, g)
                assert J == first[0] and all(np.array_equal(a, b) for a, b in zip(g, first[1])), (kw, K)
                assert all(np.isfinite(a).all() and np.abs(a).max() > 0 for a in g)
