"""Batched heat on the launches with a producer warp: every instance equal to
its own plain run where units, z chunks and tiles are smallest and ragged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one tile and many, narrower than a float4, every radius, no steps at all and
# one step beside many
ITEMS = [((3, 5, 9), 1, 7), ((33, 17, 8), 4, 5), ((130, 29, 11), 2, 12), ((64, 57, 20), 3, 1), ((65, 15, 40), 4, 40),
         ((31, 60, 33), 1, 25), ((47, 14, 5), 2, 0), ((128, 28, 16), 3, 9), ((200, 100, 24), 1, 3)]


# z chunks shorter than the radius (a unit then waits for more chunks than its
# neighbours), of a few planes, and whole columns
@pytest.mark.parametrize("zchunk,tile", [(1, 0), (3, 128), (7, 32), (16, 64), (0, 0)])
def test_batch_units_equal_plain_runs(b2r, zchunk, tile):
    import torch
    rng = np.random.default_rng(61)
    items = [dict(env=e, D=D, nsteps=n, alpha_dt=0.02, dz=0.8) for e, D, n in ITEMS]
    ins = [rng.random(tuple(e + 2 * it["D"] for e in it["env"][::-1]), dtype=np.float32) for it in items]
    s = torch.cuda.Stream()
    with b2r.Batch(items, stream=s) as bt:
        bt.set_tile(tile)
        bt.set_zchunk(zchunk)
        for graph in (True, False):
            for i, a in enumerate(ins):
                bt.upload(i, a)
            bt.run(graph=graph)
            bt.synchronize()
            got = [bt.download(i) for i in range(len(items))]
            for i, it in enumerate(items):
                with b2r.Domain(b2r.MODEL_HEAT, it["env"], D=it["D"], alpha_dt=0.02, dz=0.8) as d:
                    d.upload(ins[i])
                    d.step(it["nsteps"])
                    assert np.array_equal(got[i], d.download()), (i, graph)
