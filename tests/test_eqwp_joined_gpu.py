"""Many steps of an elastic-wave domain of several blocks run on the domain as
one block: the same bits as the blocks with their exchanges (short runs), with
block steps before, between and after, and with the one-pass step, which needs
the shell in both field sets, after them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAG = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz")


def fill(d, model, env, seed, shell=2):
    rng = np.random.default_rng(seed)
    shape = tuple(e + 2 * shell for e in env[::-1])
    for f in STAG + (("disp",) if model == 0 else ()):
        d.upload((rng.random(shape, dtype=np.float32) - 0.5) * np.float32(1e-2), field=f)
    return rng, shape


# three subdomains on an axis, odd sizes, halos of two steps, an axis of one block
@pytest.mark.parametrize("env,blocks,R", [((48, 40, 32), (2, 2, 1), 2), ((39, 34, 27), (3, 2, 3), 1),
                                          ((70, 25, 66), (1, 1, 2), 3), ((132, 16, 35), (4, 1, 1), 1)])
@pytest.mark.parametrize("ref", [False, True])
def test_joined_equals_blocks(b2r, env, blocks, R, ref):
    import torch
    model = b2r.MODEL_EQWP_REF if ref else b2r.MODEL_EQWP_STAG
    names = STAG + (("disp",) if ref else ())
    runs = (1, 45, 3, 61, 2)
    outs = []
    for many in (True, False):
        with b2r.Domain(model, env, blocks=blocks, R=R, D=2, dt=2e-4, h=1.0, src=(env[0] // 2, 5, env[2] // 2 + 1),
                        stream=torch.cuda.Stream()) as d:
            rng, shape = fill(d, 0 if ref else 1, env, 5)
            if not ref:
                for f, c in (("lambda", 3.0), ("mu", 2.0), ("buoy", 0.5)):
                    d.upload(np.float32(c) + rng.random(shape, dtype=np.float32), field=f)
                d.set_source(rng.random(90, dtype=np.float32))
            got = []
            for n in runs:
                for k in ([n] if many else [1] * n):
                    d.step(k)
                got += [d.download(field=f) for f in names]
            d.upload(np.full(shape, 0.25, np.float32), field="vy")   # one field: the others' halos are still lost
            for k in ([40] if many else [1] * 40):
                d.step(k)
            got += [d.download(field=f) for f in names]
            if not ref:
                d.set_tuning(eqwp_fused=1)
                d.step(4)
                got += [d.download(field=f) for f in names]
            d.synchronize()
            outs.append(got)
    for k, (a, b) in enumerate(zip(*outs)):
        assert np.isfinite(a).all() and np.array_equal(a, b), (k // len(names), names[k % len(names)])
