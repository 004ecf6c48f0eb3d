"""Misfit gradients and recordings with thousands of receivers, whose samples and
residuals are shared out over the launches' CTAs."""
import numpy as np
import pytest

from test_heat_adjoint_gpu import domain, observed, problem, rel_l2

pytestmark = pytest.mark.gpu


# receivers on a CTA's edge and beyond, several in one cell; the bounds of the
# test with 16 receivers
@pytest.mark.parametrize("nrec", [1024, 1025, 5000])
def test_heat_gradient_matches_fp64_oracle(b2r, orc, nrec):
    D = 2
    P = problem(D, env=(24, 20, 18), nsteps=20, nrec=nrec)
    d_obs = observed(b2r, P)
    with domain(b2r, P, P["kappa"]) as d:
        J, g, syn = d.heat_misfit_gradient(P["nsteps"], P["rec"], d_obs, ckpt_every=7)
    rec_blk = [(int(x) + D, int(y) + D, int(z) + D) for x, y, z in P["rec"]]
    J64, g64, syn64, _ = orc.heat_kappa_gradient(P["u0"].astype(np.float64), P["kappa"].astype(np.float64), D,
                                                 orc.heat_lap_weights(D, *P["coef"]), rec_blk, P["nsteps"],
                                                 d_obs.astype(np.float64))
    assert abs(J - J64) <= 1e-4 * abs(J64)
    assert rel_l2(syn, syn64) <= 1e-5
    assert rel_l2(g, g64[(slice(D, -D),) * 3]) <= 1e-5


# every cell of a few planes once: whatever their order, each is added to its own cell
@pytest.mark.parametrize("fused", [1, 0])
def test_elastic_gradient_in_any_order(b2r, fused):
    env, n = (40, 36, 20), 12
    rng = np.random.default_rng(6)
    rec = np.stack(np.meshgrid(np.arange(40), np.arange(36), [3, 9], indexing="ij"), -1).reshape(-1, 3)
    shape = tuple(e + 4 for e in env[::-1])
    obs = rng.random((n, len(rec)), dtype=np.float32)
    f0 = [rng.random(shape, dtype=np.float32) - np.float32(0.5) for _ in range(9)]
    got = []
    for order in (np.arange(len(rec)), rng.permutation(len(rec))):
        with b2r.Domain(b2r.MODEL_EQWP_STAG, env, D=2, dt=2e-2, h=1.0, src=(4, 5, 6)) as d:
            d.set_tuning(adj_fused=fused)
            for f, c in (("lambda", 3.0), ("mu", 2.0), ("buoy", 0.5)):
                d.upload(np.full(shape, c, np.float32), field=f)
            for k, f in enumerate(f0):
                d.upload(f, field=k)
            _, g, syn = d.eqwp_misfit_gradient(n, rec[order], obs[:, order], ckpt_every=5)
            got.append((*g, syn[:, np.argsort(order)]))
    assert all(np.array_equal(a, b) for a, b in zip(*got))


def test_recording_time_is_the_copy(b2r):
    """Every cell of 64^3 a receiver: a recording takes what a few receivers do and the
    copy out (one CTA alone takes 0.4 ms a step for the samples, 8 ms in all)."""
    import time

    import torch

    def best(f):
        ts = []
        for _ in range(6):
            t = time.perf_counter()
            f()
            ts.append(time.perf_counter() - t)
        return min(ts) * 1e3

    rec = np.stack(np.meshgrid(*[np.arange(64)] * 3, indexing="ij"), -1).reshape(-1, 3)
    with b2r.Domain(b2r.MODEL_HEAT, (64, 64, 64), D=1, alpha_dt=0.05, stream=torch.cuda.Stream()) as d:
        d.upload(np.random.default_rng(0).random(d.domain_shape, dtype=np.float32))
        every, few = best(lambda: d.heat_record(20, rec)), best(lambda: d.heat_record(20, rec[:64]))
    out = torch.zeros((20, len(rec)), device="cuda")
    copy = best(lambda: np.copyto(np.empty(out.shape, np.float32), out.cpu().numpy()))
    assert every <= few + 2 * copy + 2.0, (every, few, copy)
