"""The one-block form of a domain of several blocks, or of a heat torus: a large one
lives in the blocks' own buffers, so that a domain takes the memory of its
blocks; small ones have spare buffers out of a share of the process.  Both give the
bits of the blocks, and a captured run can be replayed."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
WAVE = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz")


def make(b2r, model, env, blocks, R, D, periodic, **kw):
    return b2r.Domain(getattr(b2r, "MODEL_" + model), env, blocks=blocks, R=R, D=D, dt=2e-4, h=1.0, alpha_dt=0.02,
                      src=(env[0] // 2, 5, env[2] // 2 + 1), boundary=b2r.BC_PERIODIC if periodic else b2r.BC_SHELL, **kw)


def one_buffer(d):
    nx, ny, nz = d.block_n
    return 4 * ((nx + 40 + 31) // 32 * 32) * ny * nz * int(np.prod(list(d.cfg.blocks)))   # a padded row at most


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def no_share(b2r):
    """Domains that take up the share: one-block forms made now are in the blocks' buffers."""
    with contextlib.ExitStack() as held:
        for _ in range(5):
            held.enter_context(make(b2r, "HEAT", (300, 300, 300), (2, 1, 1), 1, 1, False))
        yield


# buffers of the blocks that a large domain holds: the collocated wave's one more
@pytest.mark.parametrize("model,env,blocks,R,D,periodic,buffers", [
    ("HEAT", (384, 384, 256), (2, 2, 2), 2, 1, False, 2), ("HEAT", (400, 360, 300), (1, 2, 1), 3, 2, True, 2),
    ("HEAT", (400, 320, 320), (1, 1, 1), 1, 4, True, 2), ("EQWP_STAG", (384, 384, 256), (2, 1, 2), 1, 2, False, 21),
    ("EQWP_REF", (512, 384, 256), (2, 2, 1), 1, 2, False, 11)])
def test_memory_is_the_blocks(b2r, model, env, blocks, R, D, periodic, buffers):
    before = free()
    with make(b2r, model, env, blocks, R, D, periodic) as d:
        taken = before - free()
        # a torus of one block may need a quarter more for deeper halos; 48 MB for what an allocation rounds up to
        room = 1.25 if periodic and blocks == (1, 1, 1) else 1
        assert taken <= buffers * one_buffer(d) * room + 48 * MB, taken / one_buffer(d)


def test_small_domains_share_a_bounded_amount(b2r):
    before = free()
    with contextlib.ExitStack() as held:
        ds = [held.enter_context(make(b2r, "HEAT", (250, 250, 250), (2, 1, 1), 1, 1, False)) for _ in range(16)]
        taken = before - free()
        assert taken <= 16 * (2 * one_buffer(ds[0]) + 4 * MB) + 1024 * MB
    assert before - free() <= 16 * MB


CASES = [("HEAT", (130, 63, 70), (2, 3, 1), 1, 1, False), ("HEAT", (100, 62, 81), (1, 2, 3), 2, 2, False),
         ("HEAT", (66, 30, 46), (2, 3, 1), 1, 4, False), ("HEAT", (90, 75, 64), (2, 1, 1), 2, 1, True),
         ("HEAT", (77, 83, 65), (1, 1, 1), 1, 3, True), ("EQWP_STAG", (48, 40, 32), (2, 2, 1), 2, 2, False),
         ("EQWP_STAG", (39, 34, 27), (3, 2, 3), 1, 2, False), ("EQWP_REF", (48, 40, 32), (2, 2, 1), 1, 2, False),
         ("EQWP_REF", (132, 16, 35), (4, 1, 1), 1, 2, False), ("EQWP_REF", (70, 25, 66), (1, 1, 2), 1, 2, False)]


# single steps between and after: they read the shell of both buffers and the halos
@pytest.mark.parametrize("model,env,blocks,R,D,periodic", CASES)
@pytest.mark.parametrize("share", [True, False])
def test_equals_blocks(b2r, model, env, blocks, R, D, periodic, share):
    import torch
    names = {"HEAT": (0,), "EQWP_STAG": WAVE, "EQWP_REF": WAVE + ("disp",)}[model]
    outs = []
    with contextlib.nullcontext() if share else no_share(b2r):
        for many in (True, False):
            rng = np.random.default_rng(37)
            with make(b2r, model, env, blocks, R, D, periodic, stream=torch.cuda.Stream()) as d:
                def fill():
                    for f in names + (("lambda", "mu", "buoy") if model == "EQWP_STAG" else ()):
                        d.upload(rng.random(d.domain_shape, dtype=np.float32), field=f)
                fill()
                if model == "EQWP_STAG":
                    d.set_source(rng.random(60, dtype=np.float32))
                got = []
                for n in (3, 25, 1, 40, 5):
                    for k in ([n] if many else [1] * n):
                        d.step(k)
                    got += [d.download(field=f) for f in names]
                    got += [b for f in names[:1] for b in d.download_blocks(field=f).values()] if many else []
                fill()
                for k in ([27] if many else [1] * 27):
                    d.step(k)
                got += [d.download(field=f) for f in names]
                d.synchronize()
                outs.append(got if not many else [g for g in got if g.shape == d.domain_shape])
    for k, (a, b) in enumerate(zip(*outs)):
        assert np.isfinite(a).all() and np.array_equal(a, b), (k // len(names), names[k % len(names)])


# the wave's force is a matter of the step count, which a replay does not move:
# past its 50 steps there is none
@pytest.mark.parametrize("model,env,blocks,R,D,periodic", CASES)
@pytest.mark.parametrize("share,n", [(True, 25), (False, 25), (False, 28)])
def test_replayed_capture_equals_steps(b2r, model, env, blocks, R, D, periodic, share, n):
    import torch
    names = {"HEAT": (0,), "EQWP_STAG": WAVE, "EQWP_REF": WAVE + ("disp",)}[model]
    outs = []
    with contextlib.nullcontext() if share else no_share(b2r):
        for captured in (True, False):
            rng = np.random.default_rng(31)
            s = torch.cuda.Stream()
            with make(b2r, model, env, blocks, R, D, periodic, stream=s) as d:
                d.set_graphs(False)
                for f in names + (("lambda", "mu", "buoy") if model == "EQWP_STAG" else ()):
                    d.upload(rng.random(d.domain_shape, dtype=np.float32), field=f)
                for _ in range(1 if model == "HEAT" else 2):
                    d.step(n + 4)
                d.synchronize()
                if captured:
                    g = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g, stream=s):
                        d.step(n)
                    with torch.cuda.stream(s):
                        for _ in range(3):
                            g.replay()
                else:
                    for _ in range(3):
                        d.step(n)
                outs.append([d.download(field=f) for f in names])
                d.synchronize()
    for f, a, b in zip(names, *outs):
        assert np.isfinite(a).all() and np.array_equal(a, b), f
