"""The collocated model's own entry for a period (b2r_eqwp_gpu_main) between steps of
several blocks: the fields move on without an exchange, so the next step has to
start with one, whether the halos were fresh from an upload, from the caller's
exchange, or brought up to date after a long run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz", "disp")


def exchange(d):
    for f in NAMES:
        d.boundary_updating_direct(d.time_step, field=f)


# before: steps from the upload on (0, a short run, a long one); exchanged:
# whether the caller exchanges before the call
@pytest.mark.parametrize("env,blocks,R", [((48, 40, 36), (2, 2, 1), 1), ((80, 32, 80), (2, 1, 2), 2)])
@pytest.mark.parametrize("before,exchanged", [(0, False), (0, True), (4, True), (30, False), (30, True)])
def test_step_after_gpu_main_exchanges(b2r, env, blocks, R, before, exchanged):
    outs = []
    for long_runs in (True, False):
        with b2r.Domain(b2r.MODEL_EQWP_REF, env, blocks=blocks, R=R, D=2) as d:
            rng = np.random.default_rng(83)
            for f in NAMES:
                d.upload((rng.random(d.domain_shape, dtype=np.float32) - 0.5) * np.float32(1e-2), field=f)
            for n in ([before] if long_runs else [1] * before):
                d.step(n)
            if exchanged or not long_runs:
                exchange(d)
            d.eqwp_gpu_main(d.time_step, R)
            if not long_runs:
                exchange(d)
            d.step(R)
            outs.append([d.download(field=f) for f in NAMES])
            d.synchronize()
    for f, a, b in zip(NAMES, *outs):
        assert np.isfinite(a).all() and np.array_equal(a, b), f
