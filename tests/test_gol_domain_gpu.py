"""Game of Life over several generations on the domain's bit grid: bit-exact
against the oracle where its tiles, words and wraps have edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(orc, dom, steps, periodic):
    a = dom.copy()
    if periodic:
        orc.gol_run_periodic(a, steps)
        return a
    b = dom.copy()
    for _ in range(steps):
        orc.gol_substep(a, b, 0, 1, 63)
        a, b = b, a
    return a


# rows of one word, a word and a bit, exactly 32 words and cut into x tiles
# (33 words, and a ragged 35); axes smaller than a tile's halo; many tiles
@pytest.mark.parametrize("env,blocks,R,periodic", [
    ((5, 4, 3), (1, 1, 1), 1, True), ((32, 9, 7), (1, 1, 1), 3, True), ((33, 20, 40), (1, 2, 2), 2, True),
    ((1024, 12, 10), (2, 1, 1), 1, True), ((1056, 11, 9), (1, 1, 1), 4, True), ((1100, 10, 12), (2, 1, 2), 3, True),
    ((30, 30, 30), (1, 1, 1), 1, False), ((31, 6, 50), (1, 1, 2), 3, False), ((1100, 8, 9), (2, 1, 1), 2, False),
    ((96, 130, 70), (3, 2, 1), 4, False), ((160, 90, 110), (1, 1, 1), 1, True)])
def test_many_generations_match_oracle(b2r, orc, env, blocks, R, periodic):
    rng = np.random.default_rng(41)
    if periodic:
        dom = (rng.random(env[::-1]) < 0.3).astype(np.uint8)
    else:
        dom = (rng.random(tuple(e + 2 for e in env[::-1])) < 0.3).astype(np.uint8)   # a live shell too
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    for steps in (4, 9, 21):
        with b2r.Domain(b2r.MODEL_GOL, env, blocks=blocks, R=R, D=1, boundary=bc) as d:
            d.upload(dom)
            d.step(steps)
            got = d.download()
            d.synchronize()
        assert np.array_equal(got, _reference(orc, dom, steps, periodic)), steps


@pytest.mark.parametrize("periodic", [True, False])
def test_single_generations_after_many(b2r, orc, periodic):
    """The grid leaves the blocks' halos behind: the sub-steps of a period
    that follow, at its start or in its middle, fetch them again."""
    env, R = (64, 40, 24), 4
    rng = np.random.default_rng(42)
    dom = (rng.random(env[::-1] if periodic else tuple(e + 2 for e in env[::-1])) < 0.3).astype(np.uint8)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    with b2r.Domain(b2r.MODEL_GOL, env, blocks=(2, 2, 2), R=R, D=1, boundary=bc) as d:
        d.upload(dom)
        done = 0
        for n in (1, 6, 1, 2, 8, 1, 3, 5, 2):
            d.step(n)
            done += n
            assert np.array_equal(d.download(), _reference(orc, dom, done, periodic)), done
        d.boundary_updating_direct()
        d.step(2)
        assert np.array_equal(d.download(), _reference(orc, dom, done + 2, periodic))
        assert d.time_step == done + 2
        d.synchronize()
