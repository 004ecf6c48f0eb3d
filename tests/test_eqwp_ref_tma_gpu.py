"""The collocated elastic wave on large blocks, inputs streamed through TMA rings:
the rounding of the plain stages, which small blocks take, cell by cell; tiles,
rows and z chunks with remainders, the body force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz", "disp")


def plain_step(v, s, disp, ts, force):
    """One step in float32 numpy as the plain stages round it: increments from
    central differences with one product of each pair fused."""
    f = np.float32
    a, b = f((-1 / 12) / 10.0), f((2 / 3) / 10.0)
    l2m, lam, mu = f(0.5 * (32.0 + 2 * 174.87)), f(16.0), f(0.5 * 174.87)
    ir = 0.0005555555555555556
    c = slice(2, -2)

    def fma(x, y, z):
        return (np.asarray(x, np.float64) * y + np.asarray(z, np.float64)).astype(f)

    def diff(u, ax):
        def at(k):
            sl = [c, c, c]
            sl[ax] = slice(2 + k, u.shape[ax] - 2 + k)
            return u[tuple(sl)]
        far, near = at(2) - at(-2), at(1) - at(-1)
        return fma(b, near, a * far) if ax == 1 else fma(a, far, b * near)

    X, Y, Z = 2, 1, 0
    vx, vy, vz = v
    xx, yy, zz = diff(vx, X), diff(vy, Y), diff(vz, Z)
    inc = dict(sxx=fma(l2m, xx, lam * (yy + zz)), syy=fma(l2m, yy, lam * (xx + zz)), szz=fma(lam, xx + yy, l2m * zz),
               sxy=mu * (diff(vx, Y) + diff(vy, X)), sxz=mu * (diff(vx, Z) + diff(vz, X)),
               syz=mu * (diff(vy, Z) + diff(vz, Y)))
    for k in inc:
        s[k][c, c, c] += inc[k]
    dx = diff(s["sxx"], X) + diff(s["sxy"], Y) + diff(s["sxz"], Z)
    dy = diff(s["sxy"], X) + diff(s["syy"], Y) + diff(s["syz"], Z)
    dz = diff(s["sxz"], X) + diff(s["syz"], Y) + diff(s["szz"], Z)
    if ts < 50:
        dy[force] += f(-10000.0)
    for u, d in zip(v, (dx, dy, dz)):
        u[c, c, c] += f(0.5 * ir) * d
    disp[c, c, c] += f(0.25 * ir) * dy


# one z chunk and many, tiles of 128, 72 and 32 cells, rows that end inside a float4
@pytest.mark.parametrize("env", [(129, 90, 81), (70, 131, 99), (33, 95, 300), (300, 61, 50)])
def test_streamed_stages_round_as_the_plain_ones(b2r, env):
    rng = np.random.default_rng(4)
    shape = tuple(e + 4 for e in env[::-1])
    ini = [(rng.random(shape, dtype=np.float32) - np.float32(0.5)) for _ in NAMES]
    with b2r.Domain(b2r.MODEL_EQWP_REF, env, D=2) as d:
        for n, u in zip(NAMES, ini):
            d.upload(u, field=n)
        d.step(3)
        got = [d.download(field=n) for n in NAMES]
        d.synchronize()
    F = dict(zip(NAMES, [u.copy() for u in ini]))
    nx, nz = env[0] + 4, env[2] + 4
    force = (slice(nz // 2 - 2, nz // 2 + nz // 10 - 2), env[1] - 7, slice(nx // 2 - 2, nx // 2 + nx // 10 - 2))
    for ts in range(3):
        plain_step([F["vx"], F["vy"], F["vz"]], F, F["disp"], ts, force)
    for n, u in zip(NAMES, got):
        same = np.mean(u == F[n])
        # numpy's doubles round an FMA twice: a last bit in a few cells
        assert same > 0.999 and np.abs(u - F[n]).max() <= 4e-7 * max(1.0, np.abs(F[n]).max()), (n, same)


@pytest.mark.parametrize("env,blocks,R", [((120, 96, 100), (1, 2, 2), 1), ((144, 104, 80), (2, 1, 1), 2)])
def test_streamed_equals_plain(b2r, env, blocks, R):
    """A run as one block against steps in several, both streamed; and two steps of
    the domain against its lower half alone, which is small enough for the plain
    stages: the same away from the cut and from the body force."""
    rng = np.random.default_rng(6)
    shape = tuple(e + 4 for e in env[::-1])
    ini = [(rng.random(shape, dtype=np.float32) - np.float32(0.5)) for _ in NAMES]
    got = []
    for many in (True, False):
        with b2r.Domain(b2r.MODEL_EQWP_REF, env, blocks=blocks, R=R, D=2) as d:
            for n, u in zip(NAMES, ini):
                d.upload(u, field=n)
            for k in ([30] if many else [1] * 30):
                d.step(k)
            got.append([d.download(field=n) for n in NAMES])
            d.synchronize()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    cut = env[2] // 2
    with b2r.Domain(b2r.MODEL_EQWP_REF, env, D=2) as d, \
            b2r.Domain(b2r.MODEL_EQWP_REF, (env[0], env[1], cut), D=2) as e:
        for n, u in zip(NAMES, ini):
            d.upload(u, field=n)
            e.upload(np.ascontiguousarray(u[:cut + 4]), field=n)
        d.step(2)
        e.step(2)
        for n in NAMES:
            part = (slice(0, 12), slice(0, env[1] - 20), slice(None))
            assert np.array_equal(d.download(field=n)[part], e.download(field=n)[part]), n
