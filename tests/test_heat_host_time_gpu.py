"""Host time of heat steps that no graph replays: a launch's tiles are searched for
once per domain, however many blocks it has."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# radius 1 at two steps per pass and one, a higher radius; eight blocks and 4096
@pytest.mark.parametrize("R,D", [(2, 1), (1, 1), (1, 3)])
def test_step_time_does_not_grow_with_the_blocks(b2r, R, D):
    def per_step(blocks, env):
        with b2r.Domain(b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=D, alpha_dt=0.02) as d:
            d.upload(np.random.default_rng(1).random(d.domain_shape, dtype=np.float32))
            ts = []
            for _ in range(30):
                d.synchronize()
                t = time.perf_counter()
                d.step(R)                      # short: no graph, no one-block form, and the queue has room
                ts.append(time.perf_counter() - t)
            d.synchronize()
            return min(ts[2:]) * 1e6

    few, many = per_step((2, 2, 2), (128, 128, 128)), per_step((16, 16, 16), (128, 128, 128))
    assert many <= 2 * few + 5, (few, many)
