"""Batched elastic-wave instances whose units wait per z chunk: the bits of the
handles stepped alone, with chunks shorter than the stages' reach, remainders
of one plane, one chunk, and instances of very different step counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [((40, 33, 9), 31), ((64, 20, 35), 3), ((13, 45, 22), 77), ((129, 18, 13), 20), ((16, 16, 5), 50)]


@pytest.mark.parametrize("zchunk", [None, 1, 2, 3, 4, 0])
def test_chunks_equal_plain_steps(b2r, zchunk):
    import torch
    s = torch.cuda.Stream()
    sets = []
    for _ in range(2):
        rng = np.random.default_rng(3)
        ds = []
        for env, n in SIZES:
            shape = tuple(e + 4 for e in env[::-1])
            d = b2r.Domain(b2r.MODEL_EQWP_STAG, env, D=2, dt=2e-4, h=1.0, src=tuple(e // 2 for e in env), stream=s)
            for f, c in (("lambda", 3.0), ("mu", 2.0), ("buoy", 0.5)):
                d.upload(np.float32(c) + rng.random(shape, dtype=np.float32), field=f)
            for f in range(9):
                d.upload((rng.random(shape, dtype=np.float32) - 0.5) * np.float32(1e-2), field=f)
            d.set_source(rng.random(2 * n, dtype=np.float32))
            ds.append(d)
        sets.append(ds)
    with b2r.EqwpBatch(sets[0], [n for _, n in SIZES], stream=s) as b:
        if zchunk is not None:
            b.set_zchunk(zchunk)
        for _ in range(2):
            b.run()
        b.synchronize()
        for d, (_, n) in zip(sets[1], SIZES):
            d.step(2 * n)
        for i, (x, y) in enumerate(zip(*sets)):
            for f in range(9):
                u, v = x.download(field=f), y.download(field=f)
                assert np.isfinite(u).all() and np.array_equal(u, v), (i, f)
    for ds in sets:
        for d in ds:
            d.close()
