"""The work whose speed is tracked: what programs have this library do, through its Python face.

Eight kinds of call.  A pass starts from the input that the program holds on
the GPU and ends with the whole result there (the misfit gradients give theirs
on the host, as the library does):

  heat, gol, wave, wave_ref   Domain: upload the initial fields, step, download the fields
  heat_batch, wave_batch      Batch / EqwpBatch: many uneven instances in one launch
  heat_grad, wave_grad        Domain.heat_misfit_gradient / eqwp_misfit_gradient

Schedules are the library's defaults.  All work goes to one non-default stream,
so that whole periods are replayed from CUDA graphs.
"""
import math
import random

import numpy as np
import torch

import b2r_gb300 as b2r

_WAVE = ("vx", "vy", "vz", "sxx", "sxy", "sxz", "syy", "syz", "szz")
_stream = None


def _the_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, env, steps, blocks=(1, 1, 1), R=1, D=1, periodic=False, **more):
    return dict(kind=kind, nx=env[0], ny=env[1], nz=env[2], bx=blocks[0], by=blocks[1], bz=blocks[2], R=R, D=D,
                periodic=periodic, steps=steps, **more)


def listed():
    return [
        # the smallest call: a few thousand cells in four subdomains, the
        # halo exchanged every second step; launches are everything
        dict(_case("heat", (48, 40, 32), 20, (2, 2, 1), R=2, alpha=0.1, dz=1.0), name="heat_small"),
        # the reference's CPU-runnable case with its own constants: fits in L2
        dict(_case("heat", (128, 128, 128), 100, alpha=0.01, dz=0.5), name="heat_128"),
        # the headline: a field larger than L2, second order in space
        dict(_case("heat", (512, 512, 512), 100, alpha=0.1, dz=1.0), name="heat_512"),
        # the high-order stencil on the same domain
        dict(_case("heat", (512, 512, 512), 50, D=4, alpha=0.02, dz=1.0), name="heat4_512"),
        # a torus of odd-sized subdomains with a deep halo, fourth order
        dict(_case("heat", (250, 186, 132), 48, (2, 2, 2), R=3, D=2, periodic=True, alpha=0.02, dz=1.0),
             name="heat_torus"),
        # Game of Life on a torus of eight subdomains, halo depth 4
        dict(_case("gol", (256, 256, 256), 400, (2, 2, 2), R=4, periodic=True), name="gol_256"),
        # the staggered elastic wave in layered rock, four subdomains
        dict(_case("wave", (512, 512, 256), 100, (2, 2, 1), R=2, D=2), name="wave_512"),
        # the reference's own elastic-wave model as its main program runs it
        dict(_case("wave_ref", (512, 256, 512), 50, (2, 1, 2), R=2, D=2), name="wave_ref"),
        # 64 heat instances of uneven sizes, orders and step counts
        dict(kind="heat_batch", n=64, lo=32, hi=192, grid=16, steps_lo=50, steps_hi=500, mix=4, name="heat_batch"),
        # 16 small elastic-wave instances (a survey's shots)
        dict(kind="wave_batch", n=16, lo=32, hi=128, grid=16, steps_lo=50, steps_hi=150, mix=6, name="wave_batch"),
        # inversion: the gradient of a receiver misfit, elastic wave
        dict(_case("wave_grad", (128, 128, 128), 200, D=2, ckpt=50, nrec=64), name="wave_gradient"),
        # the same for the conductivity of the heat model
        dict(_case("heat_grad", (160, 144, 128), 200, D=2, ckpt=50, nrec=64), name="heat_gradient"),
    ]


def _size(rng, lo, hi):
    """A size spread over its logarithm; odd ones as often as even ones."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _split(rng, lo, hi, R, D, depth):
    """(env, blocks, R): axes of one or two subdomains, the halo no deeper than a subdomain allows."""
    blocks = tuple(rng.choice((1, 1, 2)) for _ in range(3))
    env = tuple(_size(rng, max(lo, 16 * b) // b, hi // b) * b for b in blocks)
    smallest = min(e // b for e, b in zip(env, blocks))
    while R > 1 and (R * D > smallest // 2 or R * depth > smallest):
        R -= 1
    return env, blocks, R


def draw(rng):
    kind = rng.choice(("heat", "heat", "heat", "gol", "wave", "wave_ref", "heat_batch", "wave_batch", "wave_grad",
                       "heat_grad"))
    if kind == "heat":
        D = rng.choice((1, 1, 2, 3, 4))
        env, blocks, R = _split(rng, 32, 512, rng.randint(1, 4), D, D)
        lups = 4.0e9 if D == 1 else 2.0e9
        steps = max(8, min(rng.randint(20, 100), int(lups / (env[0] * env[1] * env[2]))))
        return _case(kind, env, steps, blocks, R, D, rng.random() < 0.3, alpha=0.1 if D == 1 else 0.02,
                     dz=rng.choice((1.0, 1.0, 0.8)))
    if kind == "gol":
        env, blocks, R = _split(rng, 48, 384, rng.randint(1, 4), 1, 1)
        steps = max(16, min(rng.randint(50, 400), int(8.0e9 / (env[0] * env[1] * env[2]))))
        return _case(kind, env, steps, blocks, R, 1, rng.random() < 0.6)
    if kind in ("wave", "wave_ref"):
        env, blocks, R = _split(rng, 48, 320, rng.randint(1, 2), 2, 4)
        return _case(kind, env, rng.randint(10, 50), blocks, R, 2, kind == "wave" and rng.random() < 0.2)
    if kind == "heat_batch":
        return dict(kind=kind, n=rng.randint(8, 48), lo=rng.choice((24, 32)), hi=_size(rng, 64, 192),
                    grid=rng.choice((1, 8, 16)), steps_lo=rng.randint(20, 60), steps_hi=rng.randint(100, 300),
                    mix=rng.randrange(1 << 30))
    if kind == "wave_batch":
        return dict(kind=kind, n=rng.randint(4, 16), lo=rng.choice((24, 32)), hi=_size(rng, 48, 128),
                    grid=rng.choice((1, 8, 16)), steps_lo=rng.randint(20, 50), steps_hi=rng.randint(60, 150),
                    mix=rng.randrange(1 << 30))
    env = tuple(_size(rng, 40, 144) for _ in range(3))
    D = 2 if kind == "wave_grad" else rng.randint(1, 4)
    return _case(kind, env, rng.randint(40, 160), D=D, ckpt=rng.choice((20, 32, 50)), nrec=rng.choice((16, 64)))


def _env(c):
    return c["nx"], c["ny"], c["nz"]


def _shape(c, shell):
    return c["nz"] + 2 * shell, c["ny"] + 2 * shell, c["nx"] + 2 * shell


def _items(c):
    """The instances of a batch: edges, radius (heat) and step counts drawn from the case's mix."""
    rng = random.Random(c["mix"])
    edges = range(c["lo"], c["hi"] + 1, c["grid"])
    got = []
    for _ in range(c["n"]):
        env = tuple(rng.choice(edges) for _ in range(3))
        D = rng.randint(1, 4) if c["kind"] == "heat_batch" else 2
        got.append((env, D, rng.randint(c["steps_lo"], c["steps_hi"])))
    return got


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _heat_field(shape, D, g):
    """U[0, 1) inside a cold fixed shell of D cells (no shell: D = 0)."""
    u = torch.rand(shape, generator=g, device="cuda")
    if D:
        inner = torch.zeros(shape, device="cuda")
        s = slice(D, -D)
        inner[s, s, s] = u[s, s, s]
        u = inner
    return u


def _layered(shape, g):
    """lambda, mu, 1/rho of eight horizontal layers: vp U[2000, 4000] m/s, vs = vp / sqrt(3), rho U[2000, 2600]."""
    n = 8
    vp = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2000 + 2000
    rho = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 600 + 2000
    at = torch.clamp(torch.arange(shape[1], device="cuda") * n // shape[1], max=n - 1)
    vp, rho = vp[at][None, :, None], rho[at][None, :, None]
    mu = rho * vp ** 2 / 3
    return [t.expand(shape).to(torch.float32).contiguous() for t in (rho * vp ** 2 - 2 * mu, mu, 1 / rho)]


_H, _F0 = 10.0, 10.0
_DT = 0.5 * _H / (4000 * 3 ** 0.5 * (9 / 8 + 1 / 24))


def _ricker(steps):
    t = np.arange(steps) * _DT - 0.3 / _F0
    a = (np.pi * _F0 * t) ** 2
    return (1e6 * _DT * (1 - 2 * a) * np.exp(-a)).astype(np.float32)


def _wavefield(shape, shell, g):
    """A wavefield in motion (a run that goes on from a saved state): velocities of 0.01 m/s and the stresses that
    belong to them in rock, at rest in the fixed shell."""
    got = []
    for k in range(9):
        f = (torch.rand(shape, generator=g, device="cuda") - 0.5) * (0.02 if k < 3 else 1.2e5)
        if shell:
            inner = torch.zeros(shape, device="cuda")
            s = slice(shell, -shell)
            inner[s, s, s] = f[s, s, s]
            f = inner
        got.append(f)
    return got


def _ref_wavefield(shape, g):
    """As _wavefield, in the reference model's units, with the displacement."""
    f = _wavefield(shape, 2, g)
    f = [a * 50 if k < 3 else a * (1 / 2400) for k, a in enumerate(f)]
    return f + [f[1] * 0.5]


def _receivers(c):
    """nrec receivers on a plane near the low y face."""
    k = int(math.sqrt(c["nrec"]))
    xs = np.linspace(4, c["nx"] - 5, k).astype(np.int32)
    zs = np.linspace(4, c["nz"] - 5, k).astype(np.int32)
    return np.array([(x, 2, z) for x in xs for z in zs], np.int32)


def _observed(c, seed, size):
    """Measured traces: a few tones per receiver."""
    rng = np.random.default_rng(seed)
    t = np.arange(c["steps"])[:, None]
    n = c["nrec"]
    d = sum(rng.uniform(0.2, 1, n) * np.sin(t * rng.uniform(0.02, 0.2, n) + rng.uniform(0, 6.28, n)) for _ in range(3))
    return (size * d).astype(np.float32)


def _inputs(c, seed):
    """What the seed makes: the same for the library's pass and for exact()."""
    g = _gen(seed)
    kind = c["kind"]
    if kind == "heat":
        return dict(u=_heat_field(_shape(c, 0 if c["periodic"] else c["D"]), 0 if c["periodic"] else c["D"], g))
    if kind == "gol":
        shell = 0 if c["periodic"] else 1
        u = (torch.rand(_shape(c, shell), generator=g, device="cuda") < 0.3).to(torch.uint8)
        return dict(u=u)
    if kind in ("wave", "wave_grad"):
        shell = 0 if c["periodic"] else 2
        shape = _shape(c, shell)
        return dict(f=_wavefield(shape, shell, g), mat=_layered(shape, g), amps=_ricker(c["steps"]),
                    src=tuple(e // 2 for e in _env(c)))
    if kind == "wave_ref":
        return dict(f=_ref_wavefield(_shape(c, 2), g))
    if kind == "heat_batch":
        return dict(us=[_heat_field(tuple(e + 2 * D for e in env[::-1]), D, g) for env, D, _ in _items(c)])
    if kind == "wave_batch":
        got = []
        for env, _, steps in _items(c):
            shape = tuple(e + 4 for e in env[::-1])
            got.append(dict(f=_wavefield(shape, 2, g), mat=_layered(shape, g), amps=_ricker(steps),
                            src=tuple(e // 2 for e in env)))
        return dict(shots=got)
    if kind == "heat_grad":
        shape = _shape(c, c["D"])
        return dict(u=_heat_field(shape, c["D"], g), kappa=0.5 + torch.rand(shape, generator=g, device="cuda"))
    raise ValueError(kind)


def _wave_domain(env, inp, **kw):
    d = b2r.Domain(b2r.MODEL_EQWP_STAG, env, D=2, dt=_DT, h=_H, src=inp["src"], stream=_the_stream(), **kw)
    for name, m in zip(("lambda", "mu", "buoy"), inp["mat"]):
        d.upload(m, field=name)
    d.set_source(inp["amps"])
    return d


def prepare(case, seed):
    c = case
    s = dict(case=c, **_inputs(c, seed))
    torch.cuda.current_stream().synchronize()   # the library's stream is another one
    kind = c["kind"]
    if kind.endswith("_batch"):
        items = _items(c)
        if kind == "heat_batch":
            s["b"] = b2r.Batch([dict(env=env, D=D, nsteps=n, alpha_dt=0.02) for env, D, n in items],
                               stream=_the_stream())
            s["out"] = [torch.empty_like(u) for u in s["us"]]
        else:
            s["ds"] = [_wave_domain(env, shot) for (env, _, _), shot in zip(items, s["shots"])]
            s["b"] = b2r.EqwpBatch(s["ds"], [n for _, _, n in items], stream=_the_stream())
            # one tensor per component, the shots one after another: a survey's whole result
            sizes = [shot["f"][0].numel() for shot in s["shots"]]
            s["out"] = [torch.empty(sum(sizes), device="cuda") for _ in range(9)]
            s["parts"] = [torch.split(o, sizes) for o in s["out"]]
        return s
    kw = dict(blocks=(c["bx"], c["by"], c["bz"]), R=c["R"],
              boundary=b2r.BC_PERIODIC if c["periodic"] else b2r.BC_SHELL)
    if kind == "heat":
        s["d"] = b2r.Domain(b2r.MODEL_HEAT, _env(c), D=c["D"], alpha_dt=c["alpha"], dz=c["dz"], stream=_the_stream(),
                            **kw)
    elif kind == "gol":
        s["d"] = b2r.Domain(b2r.MODEL_GOL, _env(c), stream=_the_stream(), **kw)
    elif kind == "wave_ref":
        s["d"] = b2r.Domain(b2r.MODEL_EQWP_REF, _env(c), D=2, stream=_the_stream(), **kw)
    elif kind in ("wave", "wave_grad"):
        s["d"] = _wave_domain(_env(c), s, **kw)
    elif kind == "heat_grad":
        s["d"] = b2r.Domain(b2r.MODEL_HEAT, _env(c), D=c["D"], alpha_dt=0.05, stream=_the_stream(), **kw)
        s["d"].upload(s["kappa"], field="kappa")
    if kind in ("heat", "gol"):
        s["out"] = torch.empty_like(s["u"])
    elif kind in ("wave", "wave_ref"):
        s["out"] = [torch.empty_like(f) for f in s["f"]]
    else:
        s["rec"] = _receivers(c)
        s["obs"] = _observed(c, seed, 0.3 if kind == "heat_grad" else 0.003)
    return s


def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind in ("heat", "gol"):
        s["d"].upload(s["u"])
        s["d"].step(c["steps"])
        return s["d"].download(s["out"])
    if kind in ("wave", "wave_ref"):
        for k, f in enumerate(s["f"]):
            s["d"].upload(f, field=k)
        s["d"].step(c["steps"])
        for k, f in enumerate(s["out"]):
            s["d"].download(f, field=k)
        return s["out"]
    if kind == "heat_batch":
        for i, u in enumerate(s["us"]):
            s["b"].upload(i, u)
        s["b"].run()
        for i, o in enumerate(s["out"]):
            s["b"].download(i, o)
        return s["out"]
    if kind == "wave_batch":
        for d, shot in zip(s["ds"], s["shots"]):
            for k, f in enumerate(shot["f"]):
                d.upload(f, field=k)
        s["b"].run()
        for i, d in enumerate(s["ds"]):
            for k in range(9):
                d.download(s["parts"][k][i], field=k)
        return s["out"]
    if kind == "heat_grad":
        s["d"].upload(s["u"])
        J, g, syn = s["d"].heat_misfit_gradient(c["steps"], s["rec"], s["obs"], ckpt_every=c["ckpt"])
        return J, g, syn
    for k, f in enumerate(s["f"]):
        s["d"].upload(f, field=k)
    J, g, syn = s["d"].eqwp_misfit_gradient(c["steps"], s["rec"], s["obs"], ckpt_every=c["ckpt"])
    return J, g, syn


def work(case):
    """Each input field read once and each result written once; the scheme's arithmetic."""
    c = case
    kind = c["kind"]
    heat = lambda D: 3 * (3 * D + 1) + 4           # noqa: E731  sums and weights of three axes, the update
    wave = 130                                     # two stages: 18 four-point differences and the updates
    if kind == "heat_batch":
        cells = [(math.prod(env), D, n) for env, D, n in _items(c)]
        return {"bytes": sum(8 * m for m, _, _ in cells), "flops": sum(m * n * heat(D) for m, D, n in cells)}
    if kind == "wave_batch":
        cells = [(math.prod(env), n) for env, _, n in _items(c)]
        return {"bytes": sum(84 * m for m, _ in cells), "flops": sum(m * n * wave for m, n in cells)}
    m, n = math.prod(_env(c)), c["steps"]
    if kind == "heat":
        return {"bytes": 8 * m, "flops": m * n * heat(c["D"])}
    if kind == "gol":
        return {"bytes": 2 * m, "flops": 27 * m * n}
    if kind == "wave":
        return {"bytes": 84 * m, "flops": m * n * wave}
    if kind == "wave_ref":
        return {"bytes": 80 * m, "flops": m * n * wave}
    if kind == "heat_grad":      # forward once, and the reverse step's two stencils
        return {"bytes": (4 + 4 + 8) * m, "flops": 3 * m * n * heat(c["D"])}
    return {"bytes": (48 + 24) * m, "flops": 3 * m * n * wave}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
_LAP = {1: (-2.0, (1.0,)), 2: (-5 / 2, (4 / 3, -1 / 12)), 3: (-49 / 18, (3 / 2, -3 / 20, 1 / 90)),
        4: (-205 / 72, (8 / 5, -1 / 5, 8 / 315, -1 / 560))}


def _inside(u, shell, dx=0, dy=0, dz=0):
    """The cells of u's interior moved by an offset of at most the shell's depth."""
    n = u.shape
    return u[shell + dz:n[0] - shell + dz, shell + dy:n[1] - shell + dy, shell + dx:n[2] - shell + dx]


def _laplacian(u, D, w):
    """On the interior of u (a shell of D cells); w: the weights of x, y and z."""
    c0, ck = _LAP[D]
    out = _inside(u, D) * (c0 * sum(w))
    for k, c in enumerate(ck, 1):
        for a in range(3):
            hi = [0, 0, 0]
            hi[a] = k
            out += (c * w[a]) * (_inside(u, D, *hi) + _inside(u, D, *[-v for v in hi]))
    return out


def _wrapped(u, D):
    for ax in range(3):
        n = u.shape[ax]
        u = torch.cat([u.narrow(ax, n - D, D), u, u.narrow(ax, 0, D)], ax)
    return u


def _exact_heat(u, D, steps, alpha, dz=1.0, periodic=False):
    u = u.double()
    w = (alpha, alpha, alpha / (dz * dz))
    for _ in range(steps):
        if periodic:
            u = u + _laplacian(_wrapped(u, D), D, w)
        else:
            _inside(u, D).add_(_laplacian(u, D, w))
    return u


_AX = {"x": (1, 0, 0), "y": (0, 1, 0), "z": (0, 0, 1)}


def _diff(f, ax, forward):
    """Staggered fourth-order difference on the interior of f (a shell of 2 cells)."""
    o = _AX[ax]
    at = lambda k: _inside(f, 2, *[k * v for v in o])   # noqa: E731
    if forward:
        return 9 / 8 * (at(1) - at(0)) - 1 / 24 * (at(2) - at(-1))
    return 9 / 8 * (at(0) - at(-1)) - 1 / 24 * (at(1) - at(-2))


def _wave_velocity(f, b, k):
    """The three velocity increments; f: nine fields with a shell of 2, b: buoyancy inside, k = dt / h."""
    P, M = (lambda i, a: _diff(f[i], a, True)), (lambda i, a: _diff(f[i], a, False))
    return (k * b * (P(3, "x") + M(4, "y") + M(5, "z")), k * b * (M(4, "x") + P(6, "y") + M(7, "z")),
            k * b * (M(5, "x") + M(7, "y") + P(8, "z")))


def _wave_stress(f, lam, mu, k):
    P, M = (lambda i, a: _diff(f[i], a, True)), (lambda i, a: _diff(f[i], a, False))
    exx, eyy, ezz = M(0, "x"), M(1, "y"), M(2, "z")
    tr = lam * (exx + eyy + ezz)
    return (k * (tr + 2 * mu * exx), k * mu * (P(0, "y") + P(1, "x")), k * mu * (P(0, "z") + P(2, "x")),
            k * (tr + 2 * mu * eyy), k * mu * (P(1, "z") + P(2, "y")), k * (tr + 2 * mu * ezz))


def _exact_wave(f, mat, amps, src, steps, periodic=False):
    f = [a.double() for a in f]
    lam, mu, b = (a.double() if periodic else _inside(a.double(), 2) for a in mat)
    k = _DT / _H
    x, y, z = src
    for n in range(steps):
        g = [_wrapped(a, 2) for a in f] if periodic else f
        inner = (lambda a: a) if periodic else (lambda a: _inside(a, 2))
        for i, d in enumerate(_wave_velocity(g, b, k)):
            inner(f[i]).add_(d)
        g = [_wrapped(a, 2) for a in f[:3]] if periodic else f
        for i, d in enumerate(_wave_stress(g, lam, mu, k)):
            inner(f[3 + i]).add_(d)
        for i in (3, 6, 8):
            inner(f[i])[z, y, x] += float(amps[n])
    return f


def _exact_ref(f, c):
    """The reference's collocated model (its constants, its force patch in every subdomain)."""
    f = [a.double() for a in f]
    dt, dx, inv_rho, l1, l2 = 0.5, 10.0, 0.0005555555555555556, 32.00, 174.87
    env, blocks = _env(c), (c["bx"], c["by"], c["bz"])
    B = [e // k for e, k in zip(env, blocks)]
    force = torch.zeros(_shape(c, 0), dtype=torch.float64, device="cuda")
    first = [(B[a] + 4) // 2 - 2 for a in range(3)]
    last = [(B[a] + 4) // 2 + (B[a] + 4) // 10 - 2 for a in range(3)]
    for k in range(blocks[2]):
        for j in range(blocks[1]):
            for i in range(blocks[0]):
                force[k * B[2] + first[2]:k * B[2] + last[2], j * B[1] + B[1] - 7,
                      i * B[0] + first[0]:i * B[0] + last[0]] = -10000.0

    def d(i, ax):
        o = _AX[ax]
        at = lambda k: _inside(f[i], 2, *[k * v for v in o])   # noqa: E731
        return (-1 / 12 * (at(2) - at(-2)) + 2 / 3 * (at(1) - at(-1))) / dx

    for n in range(c["steps"]):
        xx, yy, zz = d(0, "x"), d(1, "y"), d(2, "z")
        tr = l1 * (xx + yy + zz)
        new = (tr + 2 * l2 * xx, l2 * (d(0, "y") + d(1, "x")), l2 * (d(0, "z") + d(2, "x")), tr + 2 * l2 * yy,
               l2 * (d(1, "z") + d(2, "y")), tr + 2 * l2 * zz)
        for i, v in enumerate(new):
            _inside(f[3 + i], 2).add_(v, alpha=dt)
        ay = d(4, "x") + d(6, "y") + d(7, "z")
        if (n // c["R"]) * c["R"] < 50:    # the force acts in the periods that start before step 50
            ay += force
        _inside(f[0], 2).add_(d(3, "x") + d(4, "y") + d(5, "z"), alpha=dt * inv_rho)
        _inside(f[1], 2).add_(ay, alpha=dt * inv_rho)
        _inside(f[9], 2).add_(ay, alpha=dt * dt * inv_rho)
        _inside(f[2], 2).add_(d(5, "x") + d(7, "y") + d(8, "z"), alpha=dt * inv_rho)
    return f


def _pad(a, n):
    return torch.nn.functional.pad(a, (n,) * 6)


def _exact_heat_grad(c, inp, obs, rec):
    D, n = c["D"], c["steps"]
    w = (0.05,) * 3
    u, kap = inp["u"].double(), _inside(inp["kappa"].double(), D)
    x, y, z = (torch.as_tensor(rec[:, a].astype(np.int64), device="cuda") for a in range(3))
    us, syn = [], []
    for _ in range(n):
        us.append(u.clone())
        _inside(u, D).add_(kap * _laplacian(u, D, w))
        syn.append(_inside(u, D)[z, y, x])
    syn = torch.stack(syn)
    res = syn - torch.as_tensor(obs, device="cuda").double()
    lam, g = torch.zeros_like(kap), torch.zeros_like(kap)
    for k in range(n - 1, -1, -1):
        lam.index_put_((z, y, x), res[k], accumulate=True)
        g += lam * _laplacian(us[k], D, w)
        lam += _laplacian(_pad(kap * lam, D), D, w)
    return float(0.5 * (res * res).sum()), g.cpu().numpy(), syn.cpu().numpy()


def _exact_wave_grad(c, inp, obs, rec):
    n, k = c["steps"], _DT / _H
    f = [a.double() for a in inp["f"]]
    lam, mu, b = (_inside(a.double(), 2) for a in inp["mat"])
    x, y, z = (torch.as_tensor(rec[:, a].astype(np.int64), device="cuda") for a in range(3))
    sx, sy, sz = inp["src"]
    E, A, syn = [], [], []      # every step's velocities and stress divergences, of which the gradients are made
    one = torch.ones((), dtype=torch.float64, device="cuda")
    for t in range(n):
        acc = _wave_velocity(f, one, 1.0)
        for i in range(3):
            _inside(f[i], 2).add_(k * b * acc[i])
        A.append(acc)
        E.append([f[i].clone() for i in range(3)])
        for i, d in enumerate(_wave_stress(f, lam, mu, k)):
            _inside(f[3 + i], 2).add_(d)
        for i in (3, 6, 8):
            _inside(f[i], 2)[sz, sy, sx] += float(inp["amps"][t])
        syn.append(_inside(f[1], 2)[z, y, x].clone())
    syn = torch.stack(syn)
    res = syn - torch.as_tensor(obs, device="cuda").double()
    vb = [torch.zeros_like(lam) for _ in range(3)]
    sb = [torch.zeros_like(lam) for _ in range(6)]
    g = [torch.zeros_like(lam) for _ in range(3)]
    for t in range(n - 1, -1, -1):
        vb[1].index_put_((z, y, x), res[t], accumulate=True)
        P, M = (lambda i, a: _diff(E[t][i], a, True)), (lambda i, a: _diff(E[t][i], a, False))
        exx, eyy, ezz = M(0, "x"), M(1, "y"), M(2, "z")
        tr = sb[0] + sb[3] + sb[5]
        g[0] += k * (exx + eyy + ezz) * tr
        g[1] += k * (2 * (exx * sb[0] + eyy * sb[3] + ezz * sb[5]) + (P(0, "y") + P(1, "x")) * sb[1] +
                     (P(0, "z") + P(2, "x")) * sb[2] + (P(1, "z") + P(2, "y")) * sb[4])
        q = [_pad(v, 2) for v in (2 * mu * sb[0] + lam * tr, mu * sb[1], mu * sb[2], 2 * mu * sb[3] + lam * tr,
                                  mu * sb[4], 2 * mu * sb[5] + lam * tr)]
        for i, d in enumerate(_wave_velocity([None] * 3 + q, one, k)):
            vb[i] -= d
        for i in range(3):
            g[2] += k * A[t][i] * vb[i]
        wv = [_pad(b * v, 2) for v in vb]
        p, m = (lambda i, a: _diff(wv[i], a, True)), (lambda i, a: _diff(wv[i], a, False))
        for i, d in enumerate((m(0, "x"), p(0, "y") + p(1, "x"), p(0, "z") + p(2, "x"), m(1, "y"),
                               p(1, "z") + p(2, "y"), m(2, "z"))):
            sb[i] -= k * d
    g[2] = -g[2] * b * b
    return float(0.5 * (res * res).sum()), tuple(v.cpu().numpy() for v in g), syn.cpu().numpy()


def exact(case, seed):
    c = case
    inp = _inputs(c, seed)
    kind = c["kind"]
    if kind == "heat":
        return _exact_heat(inp["u"], c["D"], c["steps"], c["alpha"], c["dz"], c["periodic"])
    if kind == "heat_batch":
        return [_exact_heat(u, D, n, 0.02) for u, (_, D, n) in zip(inp["us"], _items(c))]
    if kind == "wave":
        return _exact_wave(inp["f"], inp["mat"], inp["amps"], inp["src"], c["steps"], c["periodic"])
    if kind == "wave_ref":
        return _exact_ref(inp["f"], c)
    if kind == "wave_batch":
        shots = [_exact_wave(s["f"], s["mat"], s["amps"], s["src"], n)
                 for s, (_, _, n) in zip(inp["shots"], _items(c))]
        return [torch.cat([f[k].reshape(-1) for f in shots]) for k in range(9)]
    if kind == "heat_grad":
        return _exact_heat_grad(c, inp, _observed(c, seed, 0.3), _receivers(c))
    if kind == "wave_grad":
        return _exact_wave_grad(c, inp, _observed(c, seed, 0.003), _receivers(c))
    return None     # Game of Life: cells are whole numbers
