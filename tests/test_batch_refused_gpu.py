"""Batches after a schedule that is refused: a queue of more than 2^28 work items
is turned down and the batch goes on with the one it had."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a thin tall instance: in units of one plane its queue is too long, while
# another radius's queue, built before it, is not
def test_heat_batch_keeps_its_schedule(b2r):
    import torch
    items = [dict(env=(8, 8, 4096), D=1, nsteps=70001), dict(env=(33, 20, 18), D=4, nsteps=25)]
    rng = np.random.default_rng(2)
    ins = [rng.random(tuple(e + 2 * it["D"] for e in it["env"][::-1]), dtype=np.float32) for it in items]
    s = torch.cuda.Stream()
    with b2r.Batch(items, stream=s) as bt:
        for graph in (False, True):
            for i, a in enumerate(ins):
                bt.upload(i, a)
            with pytest.raises(b2r.B2RError):
                bt.set_zchunk(1)
            bt.run(graph=graph)
            bt.synchronize()
            for i, it in enumerate(items):
                with b2r.Domain(b2r.MODEL_HEAT, it["env"], D=it["D"], stream=s) as d:
                    d.upload(ins[i])
                    d.step(it["nsteps"])
                    assert np.array_equal(bt.download(i), d.download()), (i, graph)


def test_elastic_batch_keeps_its_schedule(b2r):
    import torch
    env, n = (8, 8, 4000), 34000
    s = torch.cuda.Stream()
    rng = np.random.default_rng(3)
    shape = tuple(e + 4 for e in env[::-1])
    fields = [(rng.random(shape, dtype=np.float32) - 0.5) * np.float32(1e-2) for _ in range(9)]

    def make():
        d = b2r.Domain(b2r.MODEL_EQWP_STAG, env, D=2, dt=2e-4, h=1.0, src=(3, 4, 5), stream=s)
        for f, c in (("lambda", 3.0), ("mu", 2.0), ("buoy", 0.5)):
            d.upload(np.full(shape, c, np.float32), field=f)
        for f in range(9):
            d.upload(fields[f], field=f)
        return d

    with make() as d, make() as ref, b2r.EqwpBatch([d], [n], stream=s) as bt:
        with pytest.raises(b2r.B2RError):
            bt.set_zchunk(1)
        bt.run()
        bt.synchronize()
        ref.step(n)
        for f in range(9):
            a, b = d.download(field=f), ref.download(field=f)
            assert np.isfinite(a).all() and np.array_equal(a, b), f
