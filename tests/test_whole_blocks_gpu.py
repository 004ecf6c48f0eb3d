"""Whole blocks read after a long run and an upload of one array: the halos of
the fields that were not uploaded are still brought up to date first, and those
of the uploaded one are its own."""
import numpy as np
import pytest

from test_scatter_gather_gpu import padded

pytestmark = pytest.mark.gpu

NAMES = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz")


@pytest.mark.parametrize("model,one", [("EQWP_STAG", "vy"), ("EQWP_STAG", "mu"), ("EQWP_REF", "szz")])
def test_whole_blocks_after_a_partial_upload(b2r, tmp_path, model, one):
    env, blocks, R = (48, 40, 36), (2, 2, 1), 1
    rng = np.random.default_rng(17)
    shape = tuple(e + 4 for e in env[::-1])
    names = NAMES + (("disp",) if model == "EQWP_REF" else ())
    with b2r.Domain(getattr(b2r, "MODEL_" + model), env, blocks=blocks, R=R, D=2, dt=2e-4, h=1.0, src=(3, 4, 5)) as d:
        for f in names:
            d.upload((rng.random(shape, dtype=np.float32) - 0.5) * np.float32(1e-2), field=f)
        if model == "EQWP_STAG":
            for f in ("lambda", "mu", "buoy"):
                d.upload(1 + rng.random(shape, dtype=np.float32), field=f)
        d.step(25)
        d.upload(rng.random(shape, dtype=np.float32), field=one)
        for f in names:
            want = padded(d.download(field=f), env, blocks, d.halo, 2, False)
            for key, got in d.download_blocks(field=f).items():
                assert np.array_equal(got, want[key]), (f, key)
        # the same through the block files, halos lost again
        d.step(25)
        d.upload(rng.random(shape, dtype=np.float32), field=one)
        want = padded(d.download(field="sxy"), env, blocks, d.halo, 2, False)
        got = b2r.read_block_data_bin(d.write_block_data(field="sxy", block=1, directory=str(tmp_path)))
        assert np.array_equal(got, want[(1, 0, 0)])
