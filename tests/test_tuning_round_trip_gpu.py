"""Heat knobs read from one domain and set on another give it the same kernels, and
knobs set back to their defaults the library's own choice again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def launches(b2r, d, n):
    before = b2r.kernel_launches()
    d.step(n)
    return b2r.kernel_launches() - before


# one launch in a cluster's shared memory, the one-block form, three steps per
# pass, one step per launch
@pytest.mark.parametrize("env,blocks,R,D", [((48, 40, 32), (2, 2, 1), 2, 1), ((130, 63, 70), (2, 3, 1), 1, 1),
                                            ((256, 200, 180), (1, 1, 1), 1, 1), ((100, 90, 80), (1, 1, 1), 1, 3)])
def test_round_trip(b2r, env, blocks, R, D):
    def domain():
        d = b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02)
        d.upload(np.random.default_rng(1).random(d.domain_shape, dtype=np.float32))
        return d

    with domain() as a, domain() as b:
        own = launches(b2r, a, 24)
        b.set_tuning(**a.get_tuning())
        assert launches(b2r, b, 24) == own
        b.set_tuning(tblock=1, zchunk=8)
        assert launches(b2r, b, 24) == 24 + (0 if blocks == (1, 1, 1) else 24 // R)   # sweeps, exchanges
        b.set_tuning(**a.get_tuning())
        assert launches(b2r, b, 24) == own
        a.set_tuning(tblock=1, ctas_per_sm=2, pdl=0)     # not the library's own
        b.set_tuning(**a.get_tuning())
        assert launches(b2r, b, 24) == launches(b2r, a, 24)
        x, y = a.download(), b.download()
        assert np.isfinite(x).all() and np.isfinite(y).all()
