"""Uploads into the blocks and downloads out of them, cell by cell: rows around
the width from which a warp has twice the loads in flight, several blocks, tori,
arrays of bytes that start anywhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def padded(dom, env, blocks, H, shell, periodic):
    """{block: its padded cells} by the definition of the layout."""
    B = [e // b for e, b in zip(env, blocks)]
    if periodic:
        big = np.pad(dom, H, mode="wrap")
    else:
        big = np.pad(dom, H - shell)
    return {(bx, by, bz): big[bz * B[2]:bz * B[2] + B[2] + 2 * H, by * B[1]:by * B[1] + B[1] + 2 * H,
                              bx * B[0]:bx * B[0] + B[0] + 2 * H]
            for bx in range(blocks[0]) for by in range(blocks[1]) for bz in range(blocks[2])}


@pytest.mark.parametrize("gol", [False, True])
@pytest.mark.parametrize("env,blocks,R,periodic", [
    ((62, 5, 6), (1, 1, 1), 1, False), ((64, 4, 5), (1, 1, 1), 1, False), ((126, 6, 7), (1, 1, 1), 2, False),
    ((130, 5, 4), (1, 1, 1), 1, True), ((513, 4, 4), (1, 1, 1), 1, False), ((33, 6, 8), (3, 1, 2), 2, True),
    ((10, 9, 8), (2, 3, 2), 1, False), ((251, 4, 5), (1, 1, 1), 2, True), ((1030, 3, 2), (2, 1, 1), 1, False),
    ((253, 7, 4), (1, 1, 2), 1, False), ((505, 2, 3), (1, 1, 1), 1, True)])
def test_every_cell(b2r, env, blocks, R, periodic, gol):
    import torch
    rng = np.random.default_rng(3)
    shell = 0 if periodic else 1
    shape = tuple(e + 2 * shell for e in env[::-1])
    dom = (rng.integers(0, 2, shape).astype(np.uint8) if gol else rng.random(shape, dtype=np.float32))
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    with b2r.Domain(b2r.MODEL_GOL if gol else b2r.MODEL_HEAT, env, blocks=blocks, R=R, D=1, boundary=bc) as d:
        want = padded(dom, env, blocks, R, shell, periodic)
        for start in (0, 1, 2, 3) if gol else (0,):
            raw = torch.zeros(dom.size + 8, dtype=torch.uint8 if gol else torch.float32, device="cuda")
            src = raw[start:start + dom.size].view(shape)
            src.copy_(torch.from_numpy(dom))
            d.upload(torch.zeros_like(raw[:dom.size].view(shape)))
            d.upload(src)
            for key, got in d.download_blocks().items():
                assert np.array_equal(got, want[key]), (start, key)
            out = torch.full_like(raw, 7)
            d.download(out[start:start + dom.size].view(shape))
            assert np.array_equal(out[start:start + dom.size].view(shape).cpu().numpy(), dom)
            assert (out[:start] == 7).all() and (out[start + dom.size:] == 7).all()


@pytest.mark.parametrize("model,env,blocks,R,periodic", [
    ("HEAT", (40, 33, 32), (2, 1, 2), 2, True), ("HEAT", (130, 63, 70), (2, 3, 1), 1, False),
    ("GOL", (36, 30, 24), (2, 2, 2), 3, True), ("EQWP_STAG", (48, 40, 32), (2, 1, 2), 2, False)])
def test_whole_blocks_after_long_runs(b2r, model, env, blocks, R, periodic):
    """Runs that leave the halos between blocks behind: blocks read whole afterwards
    hold their neighbours' current cells, and the next steps are none the worse."""
    rng = np.random.default_rng(9)
    wave = model == "EQWP_STAG"
    H, shell = R * (4 if wave else 1), 0 if periodic else (2 if wave else 1)
    shape = tuple(e + 2 * shell for e in env[::-1])
    dom = rng.integers(0, 2, shape).astype(np.uint8) if model == "GOL" else rng.random(shape, dtype=np.float32)
    bc = b2r.BC_PERIODIC if periodic else b2r.BC_SHELL
    ends = []
    for look in (True, False):
        with b2r.Domain(getattr(b2r, "MODEL_" + model), env, blocks=blocks, R=R, D=2 if wave else 1, boundary=bc,
                        **(dict(dt=2e-4, h=1.0, src=(3, 4, 5)) if wave else {})) as d:
            for f in (*range(9), "lambda", "mu", "buoy") if wave else (0,):
                d.upload(dom, field=f)
            d.step(25)
            if look:
                want = padded(d.download(), env, blocks, H, shell, periodic)
                for key, got in d.download_blocks().items():
                    assert np.array_equal(got, want[key]), key
            d.step(3)
            ends.append(d.download())
    assert np.array_equal(*ends)
