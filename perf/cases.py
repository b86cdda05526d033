"""The timed workloads of the hydro step: what a program using this package
calls again and again, through its public entry points.

``listed()`` gives the standing cases and ``draw(rng)`` further ones of the
same ranges; ``prepare`` builds what a program holds before the call,
``run`` makes one call, ``work`` counts what the call cannot do without and
``exact`` gives the same result in plain 64-bit torch.

Kinds of call:

* ``block64``   one RK3 step (CFL included) of an FP64 ``MeshBlock``;
* ``block32``   one RK3 step of an FP32-perturbation ``MeshBlockF32``;
* ``ensemble``  one step of a batched FP32 ``Ensemble``, eager or replayed
  from its captured graph;
* ``tendency``  one ``Hydro.forward`` (du of a state, the module-level call);
* ``rollout``   a differentiable rollout, forward and backward.

Problems: ``tube`` (1-D shock tube), ``current`` (2-D density current with
diffusion), ``bubble`` (dry warm bubbles, 2-D in a box or 3-D doubly
periodic), ``deep`` (H2-He atmosphere with passive tracers).
"""
import math
import random

import torch

from snapy_linfel_b200.config import Integration, MeshBlockOptions, make_config

IDN, IVX, IVY, IVZ, IPR = range(5)
RK3 = ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(name, kind, problem, nx1, nx2=1, nx3=1, **more):
    c = dict(name=name, kind=kind, problem=problem, nx1=nx1, nx2=nx2, nx3=nx3, riemann="lmars",
             recon="weno5", implicit=1, tracers=0)
    c.update(more)
    return c


def listed():
    return [
        # a shock-tube run: the smallest calls, latency and launches
        _case("tube-1024", "block64", "tube", 1024, riemann="hllc", implicit=0),
        # the density-current benchmark: 2-D, viscous, vertically implicit
        _case("current-1024x128", "block64", "current", 128, 1024),
        # a 2-D bubble in single-precision perturbations
        _case("bubble32-512x256", "block32", "bubble", 256, 512, riemann="hllc"),
        # one 3-D member on its own in double precision
        _case("bubble-128x128x128", "block64", "bubble", 128, 128, 128),
        # the module call on a ragged block with the full 5x5 implicit form
        _case("tendency-51x77x90", "tendency", "bubble", 90, 77, 51, riemann="roe", implicit=9),
        # explicit integration with limited linear slopes and one tracer
        _case("plm-96x80x64", "block64", "deep", 64, 80, 96, riemann="hllc", recon="plm",
              implicit=0, tracers=1),
        # the large domain, both precisions
        _case("deep-384x384x192", "block64", "deep", 192, 384, 384, riemann="roe", tracers=2),
        _case("deep32-384x384x192", "block32", "deep", 192, 384, 384, riemann="roe", tracers=2),
        # the 48-member ensemble, its step replayed from a graph
        _case("ensemble-48", "ensemble", "bubble", 1, members=48, layout=2024, graph=True, hmin=64,
              hmax=128, hstep=32, vmin=64, vmax=128, vstep=64),
        # a few small members of odd sizes, stepped eagerly
        _case("ensemble-7-ragged", "ensemble", "bubble", 1, members=7, layout=5, graph=False,
              hmin=17, hmax=61, hstep=1, vmin=21, vmax=70, vstep=1, riemann="hllc"),
        # gradient of a rollout with checkpoints (the 2-D adjoint workload)
        _case("rollout-512x256", "rollout", "bubble", 256, 512, riemann="hllc", steps=6, every=3),
        # gradient of a short 3-D rollout with tracers, stage inputs kept
        _case("rollout-64x60x48", "rollout", "deep", 48, 60, 64, riemann="roe", tracers=2, steps=2,
              every=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "flat64", "flat32", "solid64", "solid64", "solid32", "tendency",
                       "ensemble", "rollout", "rollout3"])
    solver = rng.choice(["lmars", "hllc", "roe"])
    if kind == "tube":
        c = _case("", "block64", "tube", _log_int(rng, 64, 2048), riemann=solver, implicit=0,
                  recon=rng.choice(["weno5", "weno5", "plm"]))
    elif kind == "flat64":
        c = _case("", "block64", rng.choice(["current", "bubble"]), _log_int(rng, 24, 200),
                  _log_int(rng, 64, 2000), riemann=solver, implicit=rng.choice([1, 1, 9]))
    elif kind == "flat32":
        c = _case("", "block32", "bubble", _log_int(rng, 24, 256), _log_int(rng, 64, 2000),
                  riemann=solver)
    elif kind == "solid64":
        p = rng.choice(["bubble", "deep"])
        c = _case("", "block64", p, _log_int(rng, 24, 160), _log_int(rng, 24, 256),
                  _log_int(rng, 24, 256), riemann=solver, implicit=rng.choice([0, 1, 1, 1]),
                  recon=rng.choice(["weno5", "weno5", "plm"]),
                  tracers=rng.choice([0, 2]) if p == "deep" else 0)
    elif kind == "solid32":
        p = rng.choice(["bubble", "deep"])
        c = _case("", "block32", p, _log_int(rng, 24, 160), _log_int(rng, 24, 256),
                  _log_int(rng, 24, 256), riemann=solver,
                  tracers=rng.choice([0, 2]) if p == "deep" else 0)
    elif kind == "tendency":
        c = _case("", "tendency", "bubble", _log_int(rng, 24, 128), _log_int(rng, 24, 128),
                  rng.choice([1, _log_int(rng, 24, 128)]), riemann=solver,
                  implicit=rng.choice([0, 1, 9]))
    elif kind == "ensemble":
        h, v = _log_int(rng, 16, 80), _log_int(rng, 16, 80)
        c = _case("", "ensemble", "bubble", 1, members=rng.randint(2, 24),
                  layout=rng.randrange(1 << 20), graph=rng.random() < 0.5, hmin=h, hmax=h + 24,
                  hstep=1, vmin=v, vmax=v + 40, vstep=1, riemann=solver)
    elif kind == "rollout":
        c = _case("", "rollout", "bubble", _log_int(rng, 32, 200), _log_int(rng, 64, 600),
                  riemann=solver, steps=rng.randint(1, 5), every=rng.choice([0, 2, 3]))
    else:
        c = _case("", "rollout", "deep", _log_int(rng, 20, 50), _log_int(rng, 20, 64),
                  _log_int(rng, 20, 64), riemann=solver, tracers=rng.choice([0, 1, 2]),
                  steps=1, every=0)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# configurations and initial states
# ---------------------------------------------------------------------------
def _sizes(case):
    """[(nx1, nx2, nx3)] of the blocks of a case."""
    if case["kind"] != "ensemble":
        return [(case["nx1"], case["nx2"], case["nx3"])]
    rng = random.Random(case["layout"])
    out = []
    for _ in range(case["members"]):
        h = [rng.randrange(case["hmin"], case["hmax"] + 1, case["hstep"]) for _ in range(2)]
        v = rng.randrange(case["vmin"], case["vmax"] + 1, case["vstep"])
        out.append((v, h[0], h[0] if case["hstep"] > 1 else h[1]))
    return out


def _options(case, size):
    nx1, nx2, nx3 = size
    common = dict(nx1=nx1, nx2=nx2, nx3=nx3, recon1=case["recon"], recon23=case["recon"],
                  riemann=case["riemann"], implicit_scheme=case["implicit"],
                  nscalar=case["tracers"], scalar_recon=case["recon"])
    if case["problem"] == "tube":
        cfg = make_config(x1=(0.0, 1.0), gammad=1.4, shock1=True, shock23=True,
                          bc=("outflow",) * 6, **common)
        return MeshBlockOptions(cfg, Integration(cfl=0.9))
    if case["problem"] == "deep":
        rd, cp, g, dz, dx, cfl = 3777.0, 13000.0, 24.8, 100.0, 200.0, 0.8
    else:
        rd, cp, g, cfl = 287.0, 1004.0, 9.81, 0.8
        dz = dx = 100.0 if nx3 > 1 else (50.0 if case["problem"] == "current" else 20.0e3 / 512)
    nu = 75.0 if case["problem"] == "current" else 0.0
    side = "periodic" if nx3 > 1 else "reflecting"
    cfg = make_config(x1=(0.0, nx1 * dz), x2=(0.0, nx2 * dx), x3=(0.0, nx3 * dx),
                      gammad=cp / (cp - rd), rgas=rd, grav=(-g, 0.0, 0.0), nu_iso=nu, kappa_iso=nu,
                      bc=("reflecting",) * 2 + (side,) * 4, **common)
    return MeshBlockOptions(cfg, Integration(cfl=cfl))


def _centers(lo, hi, nx, ng):
    if nx <= 1:
        return torch.tensor([0.5 * (lo + hi)], dtype=torch.float64, device="cuda")
    k = torch.arange(nx + 2 * ng, dtype=torch.float64, device="cuda")
    return lo + (hi - lo) / nx * (k - ng + 0.5)


def _state(case, opts, seed):
    """(hydro_w, scalar_r) of the seed, FP64 on the GPU, ghost cells included."""
    c = opts.hydro
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x1 = _centers(c.x1min, c.x1max, c.nx1, c.nghost)[None, None, :]
    x2 = _centers(c.x2min, c.x2max, c.nx2, c.nghost)[None, :, None]
    x3 = _centers(c.x3min, c.x3max, c.nx3, c.nghost)[:, None, None]
    shape = (c.nc3, c.nc2, c.nc1)
    w = torch.zeros((5,) + shape, dtype=torch.float64, device="cuda")
    noise = torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    if case["problem"] == "tube":
        at = rng.uniform(0.4, 0.6)
        left = (x1 < at).to(w.dtype)
        w[IDN] = (0.125 + 0.875 * left) * (1 + 1e-3 * noise)
        w[IPR] = 0.1 + 0.9 * left
        return w, None
    rd, g = c.rgas, -c.grav1
    cp = rd * c.gammad / (c.gammad - 1.0)
    p0, t0 = 1.0e5, 166.0 if case["problem"] == "deep" else 300.0
    # dry-adiabatic, above the tropopause (two thirds of a deep domain) isothermal
    zt = c.x1max * (2.0 / 3.0 if case["problem"] == "deep" else 2.0)
    tt = t0 - g * zt / cp
    temp = t0 - g * torch.clamp(x1, max=zt) / cp
    p = p0 * (temp / t0) ** (cp / rd) * torch.exp(-g * torch.clamp(x1 - zt, min=0.0) / (rd * tt))
    # a bubble (cold for the density current) and white noise in temperature
    size = rng.uniform(0.15, 0.3) * min(s for s, n in ((c.x1max, c.nx1), (c.x2max, c.nx2),
                                                       (c.x3max, c.nx3)) if n > 1)
    at = [rng.uniform(0.3, 0.7) * s for s in (c.x1max, c.x2max, c.x3max)]
    dist = torch.sqrt((x1 - at[0]) ** 2 + (x2 - at[1]) ** 2 +
                      ((x3 - at[2]) ** 2 if c.nx3 > 1 else 0.0)) / size
    amp = -15.0 if case["problem"] == "current" else rng.uniform(0.5, 3.0)
    dth = torch.where(dist <= 1, 0.5 * amp * (torch.cos(math.pi * dist) + 1.0), 0.0) + 0.01 * noise
    temp = temp + dth * (p / p0) ** (rd / cp)
    w[IPR] = p
    w[IDN] = p / (rd * temp)
    # a weak large-scale flow, so that no face sits exactly on a wave switch
    for v in (IVX, IVY, IVZ):
        if (v == IVY and c.nx2 == 1) or (v == IVZ and c.nx3 == 1):
            continue
        a, b, d = (rng.uniform(0.0, 2.0 * math.pi) for _ in range(3))
        w[v] = (torch.sin(2 * math.pi * x1 / c.x1max + a) +
                torch.cos(2 * math.pi * x2 / c.x2max + b) +
                torch.sin(2 * math.pi * x3 / c.x3max + d) + 0.05 * noise)
    if not c.nscalar:
        return w, None
    r = torch.stack([0.5 + 0.2 * torch.sin(2 * math.pi * (n + 1) * x1 / c.x1max +
                                           rng.uniform(0, 6)) * torch.cos(
        2 * math.pi * x2 / c.x2max + rng.uniform(0, 6)) + 0.2 * torch.cos(
        4 * math.pi * x3 / c.x3max + rng.uniform(0, 6)) + 0.0 * noise for n in range(c.nscalar)])
    return w, r


def _dt(c, cfl, w):
    """cfl times the CFL limit of the primitive state (over the axes that the
    time step is limited by), with the diffusive limit"""
    act = _active(c)
    it = _interior(c)
    use = list(act)
    if c.implicit_scheme & 1 and (act[1] or act[2]):
        use[0] = False
    cs = torch.sqrt(c.gammad * w[IPR][it] / w[IDN][it])
    dx = _spacing(c)
    lim = [(dx[a] / (w[IVX + a][it].abs() + cs)).min() for a in range(3) if use[a]]
    dt = torch.stack(lim).min()
    nu = max(c.nu_iso, c.kappa_iso)
    if nu > 0:
        d = min(dx[a] for a in range(3) if act[a])
        dt = torch.clamp(dt, max=d * d / (2.0 * sum(act) * nu))
    return cfl * dt


def _cotangents(case, opts, seed):
    """seeded output weights of a rollout's loss, scaled per variable"""
    c = opts.hydro
    gen = torch.Generator(device="cuda").manual_seed(seed + 1_000_003)
    gu = torch.randn(c.shape, dtype=torch.float64, device="cuda", generator=gen)
    scale = torch.tensor([1.0, 1.0, 1.0, 1.0, 1e-5], dtype=torch.float64, device="cuda")
    gs = torch.randn(c.scalar_shape, dtype=torch.float64, device="cuda", generator=gen)
    return gu * scale[:, None, None, None], gs


def _rollout_inputs(case, opts, seed):
    """(u, s, dts): conserved state with its ghosts, fixed step sizes"""
    c = opts.hydro
    w, r = _state(case, opts, seed)
    u, s, w = _conserved(c, w, r)
    dt = 0.9 * _dt(c, opts.integration.cfl, w)
    return u, s, dt.repeat(case["steps"])


# ---------------------------------------------------------------------------
# what is timed
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        from snapy_linfel_b200.ensemble import Ensemble

        members = []
        for m, size in enumerate(_sizes(case)):
            opts = _options(case, size)
            members.append((opts, *_state(case, opts, seed * 1009 + m)))
        ens = Ensemble(members)
        if case["graph"]:
            ens.capture()
        return {"kind": kind, "ens": ens}
    opts = _options(case, _sizes(case)[0])
    if kind in ("block64", "block32"):
        from snapy_linfel_b200.mesh import MeshBlock, MeshBlockF32

        mb = (MeshBlock if kind == "block64" else MeshBlockF32)(opts)
        mb.initialize(*_state(case, opts, seed))
        return {"kind": kind, "block": mb}
    if kind == "tendency":
        from snapy_linfel_b200.modules import Hydro

        w, r = _state(case, opts, seed)
        u, _, w = _conserved(opts.hydro, w, r)
        dt = _dt(opts.hydro, opts.integration.cfl, w).reshape(1)
        return {"kind": kind, "hydro": Hydro(opts), "u": u, "dt": dt}
    from snapy_linfel_b200.adjoint import StepRunner

    u, s, dts = _rollout_inputs(case, opts, seed)
    gu, gs = _cotangents(case, opts, seed)
    return {"kind": kind, "opts": opts, "u": u.requires_grad_(), "dts": dts, "gu": gu, "gs": gs,
            "s": s.requires_grad_() if s is not None else None, "every": case["every"],
            "runner": StepRunner(opts)}


def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        ens = state["ens"]
        ens.step()
        return {"u": [b.hydro_u for b in ens.blocks], "dt": ens.dts()}
    if kind in ("block64", "block32"):
        mb = state["block"]
        mb.step()
        return {"u": mb.hydro_u, "w": mb.hydro_w, "s": mb.scalar_s, "dt": mb.dt}
    if kind == "tendency":
        w = torch.empty_like(state["u"])
        return {"du": state["hydro"].forward(state["dt"], state["u"], w), "w": w}
    from snapy_linfel_b200.adjoint import rollout

    u, s = state["u"], state["s"]
    uT, sT = rollout(state["opts"], u, s, state["dts"], checkpoint_every=state["every"],
                     runner=state["runner"])
    if s is None:
        (gu,) = torch.autograd.grad(uT, u, state["gu"])
        return {"u": uT, "gu": gu}
    gu, gs = torch.autograd.grad((uT, sT), (u, s), (state["gu"], state["gs"]))
    return {"u": uT, "s": sT, "gu": gu, "gs": gs}


def work(case):
    """Per pass: the state (conserved and primitive variables, tracers) read
    once and written once, and the operations of the faces and columns of
    its stages (a divide, a square root and an addition count one each)."""
    item = 4 if case["kind"] in ("block32", "ensemble") else 8
    face = {"lmars": 75, "hllc": 120, "roe": 150}[case["riemann"]]
    nl = 1 + case["tracers"]  # variables with nonlinear weights, by default
    if case["recon"] == "plm":
        recon = 2 * 8 * (5 + case["tracers"])
    elif case["problem"] == "tube":
        recon = 2 * 60 * 5
    else:
        recon = 2 * 60 * nl + 2 * 9 * 4
    column = {0: 0, 1: 450, 9: 1500}[case["implicit"]]
    b = f = 0.0
    for size in _sizes(case):
        cells = float(size[0]) * size[1] * size[2]
        axes = sum(n > 1 for n in size)
        stage = axes * (face + recon + 2 * (5 + case["tracers"])) + column + 40
        if case["problem"] == "current":
            stage += axes * 90
        nv = 5 + case["tracers"]
        if case["kind"] == "tendency":
            b += cells * item * 3 * 5  # u in, w and du out
            f += cells * stage
        elif case["kind"] == "rollout":
            # states in and out, cotangents in, gradients out; reverse about twice the forward
            b += cells * item * 4 * nv
            f += cells * stage * 3 * case["steps"] * 3
        else:
            b += cells * item * 2 * (5 + nv)
            f += cells * stage * 3
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same calls in plain 64-bit torch
# ---------------------------------------------------------------------------
def _active(c):
    return (c.nx1 > 1, c.nx2 > 1, c.nx3 > 1)


def _spacing(c):
    return ((c.x1max - c.x1min) / c.nx1, (c.x2max - c.x2min) / c.nx2,
            (c.x3max - c.x3min) / c.nx3)


def _interior(c):
    return tuple(slice(c.nghost, c.nghost + n) if n > 1 else slice(0, 1)
                 for n in (c.nx3, c.nx2, c.nx1))


def _fill(c, x, kind):
    """Boundary fill: each axis copies from its own interior; reflecting axes
    flip the normal component of hydro variables ("u" or "w", not "s")."""
    ng = c.nghost
    for a, nx in enumerate((c.nx1, c.nx2, c.nx3)):
        if nx == 1:
            continue
        dim, n = 3 - a, nx + 2 * ng
        src, sign = list(range(n)), [1.0] * n
        for end, typ in ((0, c.bc[2 * a]), (1, c.bc[2 * a + 1])):
            for g in range(ng):
                i = ng - 1 - g if end == 0 else n - ng + g
                if typ == 1:  # reflecting
                    src[i], sign[i] = (2 * ng - 1 - i if end == 0 else 2 * (n - ng) - 1 - i), -1.0
                elif typ == 2:  # periodic
                    src[i] = i + nx if end == 0 else i - nx
                elif typ == 3:  # outflow
                    src[i] = ng if end == 0 else n - ng - 1
        x = x.index_select(dim, torch.tensor(src, device=x.device))
        if kind != "s" and -1.0 in sign:
            f = torch.ones((5, n), dtype=x.dtype, device=x.device)
            f[IVX + a] = torch.tensor(sign, dtype=x.dtype, device=x.device)
            view = [5, 1, 1, 1]
            view[dim] = n
            x = x * f.view(view)
    return x


def _conserved(c, w, r):
    """(u, s, w) with filled ghosts from primitive variables"""
    w = _fill(c, w, "w")
    m = w[IVX:IPR] * w[IDN]
    e = w[IPR] / (c.gammad - 1.0) + 0.5 * (m * w[IVX:IPR]).sum(0)
    u = _fill(c, torch.cat([w[:1], m, e[None]]), "u")
    if r is None:
        return u, None, w
    return u, _fill(c, w[:1] * _fill(c, r, "s"), "s"), w


def _primitive(c, u):
    """w of u; with gravity, density and pressure of the x1 ghosts follow the
    isentrope of the outermost interior cell in hydrostatic balance"""
    gam = c.gammad
    v = u[IVX:IPR] / u[IDN]
    rho, p = u[IDN], (gam - 1.0) * (u[IPR] - 0.5 * (v * u[IVX:IPR]).sum(0))
    if c.grav1 != 0.0:
        a, ng, lo, hi = (gam - 1.0) / gam, c.nghost, c.nghost, c.nghost + c.nx1 - 1
        dz = _spacing(c)[0]
        parts = {}
        for e, sgn in ((lo, 1.0), (hi, -1.0)):
            pe, re = p[..., e:e + 1], rho[..., e:e + 1]
            k = pe / re ** gam
            n = torch.arange(1, ng + 1, dtype=p.dtype, device=p.device)
            n = n.flip(0) if e == lo else n
            pn = (pe ** a + sgn * n * a * (-c.grav1) * dz / k ** (1.0 / gam)) ** (1.0 / a)
            parts[e] = (pn, (pn / k) ** (1.0 / gam))
        p = torch.cat([parts[lo][0], p[..., lo:hi + 1], parts[hi][0]], -1)
        rho = torch.cat([parts[lo][1], rho[..., lo:hi + 1], parts[hi][1]], -1)
    return torch.cat([rho[None], v, p[None]])


def _weno5(a, b, c, d, e):
    p = ((-a + 5 * b + 2 * c) / 6, (2 * b + 5 * c - d) / 6, (11 * c - 7 * d + 2 * e) / 6)
    s = (13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
         13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (d - b) ** 2,
         13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)
    al = [g / (x + 1e-6) ** 2 for g, x in zip((0.3, 0.6, 0.1), s)]
    return sum(x * y for x, y in zip(al, p)) / sum(al)


def _linear5(a, b, c, d, e):
    return (-3 * a + 27 * b + 47 * c - 13 * d + 2 * e) / 60


def _plm(q):
    def slope(l, m, r):
        x, y = m - l, r - m
        z = x * y
        safe = torch.where(z > 0, x + y, 1.0)
        return torch.where(z > 0, z / safe, 0.0)  # half the harmonic mean

    return q[2] + slope(q[1], q[2], q[3]), q[3] - slope(q[2], q[3], q[4])


def _faces(c, x, axis, lo, n, v):
    """left and right states of variable v at the faces lo .. lo + n of an axis"""
    typ, shock = ((c.recon1_type, c.recon1_shock) if axis == 0 else
                  (c.recon23_type, c.recon23_shock))
    if v >= 5:
        typ = c.scalar_recon_type
    q = [x.narrow(2 - axis, lo - 3 + t, n + 1) for t in range(6)]
    if typ == 1:
        L, R = _plm(q)
    else:
        f = _weno5 if v == IDN or v >= 5 or shock else _linear5
        L, R = f(q[4], q[3], q[2], q[1], q[0]), f(q[1], q[2], q[3], q[4], q[5])
    return (torch.clamp(L, min=0.0), torch.clamp(R, min=0.0)) if v >= 5 else (L, R)


def _energy(q, gam):
    return q[IPR] / (gam - 1.0) + 0.5 * q[IDN] * (q[IVX] ** 2 + q[IVY] ** 2 + q[IVZ] ** 2)


def _lmars(L, R, n, gam):
    rho = 0.5 * (L[IDN] + R[IDN])
    c = torch.sqrt(0.5 * gam * (L[IPR] + R[IPR]) / rho)
    p = 0.5 * (L[IPR] + R[IPR]) + 0.5 * rho * c * (L[n] - R[n])
    vel = 0.5 * (L[n] + R[n]) + 0.5 / (rho * c) * (L[IPR] - R[IPR])
    up = vel > 0
    h = torch.where(up, (_energy(L, gam) + L[IPR]) / L[IDN], (_energy(R, gam) + R[IPR]) / R[IDN])
    m = vel * torch.where(up, L[IDN], R[IDN])
    F = [m] + [m * torch.where(up, L[v], R[v]) for v in (IVX, IVY, IVZ)] + [m * h]
    F[n] = F[n] + p
    return F


def _hllc(L, R, n, gam):
    tiny = 1e-10
    cl, cr = (torch.sqrt(gam * q[IPR] / q[IDN]) for q in (L, R))
    pm = 0.5 * (L[IPR] + R[IPR] + (L[n] - R[n]) * 0.25 * (L[IDN] + R[IDN]) * (cl + cr))
    gf = (gam + 1.0) / (2.0 * gam)

    def q(p):
        return torch.sqrt(torch.clamp(1.0 + gf * (pm / p - 1.0), min=1.0))

    al, ar = L[n] - cl * q(L[IPR]), R[n] + cr * q(R[IPR])
    bp, bm = torch.where(ar > 0, ar, tiny), torch.where(al < 0, al, -tiny)
    tl = L[IPR] + (L[n] - al) * L[IDN] * L[n]
    tr = R[IPR] + (R[n] - ar) * R[IDN] * R[n]
    ml, mr = L[IDN] * (L[n] - al), -R[IDN] * (R[n] - ar)
    am, cp = (tl - tr) / (ml + mr), torch.clamp((ml * tr + mr * tl) / (ml + mr), min=0.0)
    left = am >= 0
    sl, sr = torch.where(left, am / (am - bm), 0.0), torch.where(left, 0.0, -am / (bp - am))
    sm = torch.where(left, -bm / (am - bm), bp / (bp - am))
    vl, vr = sl * (L[n] - bm), sr * (R[n] - bp)
    F = [vl * L[IDN] + vr * R[IDN]]
    F += [vl * L[IDN] * L[v] + vr * R[IDN] * R[v] for v in (IVX, IVY, IVZ)]
    F[n] = F[n] + sl * L[IPR] + sr * R[IPR] + sm * cp
    F.append(vl * _energy(L, gam) + vr * _energy(R, gam) + sl * L[IPR] * L[n] +
             sr * R[IPR] * R[n] + sm * cp * am)
    return F


def _roe(L, R, n, gam):
    tiny = 1e-10
    t = [v for v in (IVX, IVY, IVZ) if v != n]
    el, er = _energy(L, gam), _energy(R, gam)
    a, b = torch.sqrt(L[IDN]), torch.sqrt(R[IDN])
    rho = a * b
    vel = {v: (a * L[v] + b * R[v]) / (a + b) for v in (IVX, IVY, IVZ)}
    hl, hr = (el + L[IPR]) / L[IDN], (er + R[IPR]) / R[IDN]
    h = (a * hl + b * hr) / (a + b)
    c2 = (gam - 1.0) * (h - 0.5 * sum(x * x for x in vel.values()))
    c2 = torch.clamp(c2, min=tiny)
    c = torch.sqrt(c2)
    dp, dn = R[IPR] - L[IPR], R[n] - L[n]
    wm, wp = 0.5 * (dp / c2 - rho * dn / c), 0.5 * (dp / c2 + rho * dn / c)
    w0 = R[IDN] - L[IDN] - dp / c2
    sm, s0, sp = (x.abs() for x in (vel[n] - c, vel[n], vel[n] + c))
    diss = {IDN: sm * wm + s0 * w0 + sp * wp,
            n: sm * wm * (vel[n] - c) + s0 * w0 * vel[n] + sp * wp * (vel[n] + c),
            IPR: (sm * wm * (h - vel[n] * c) + sp * wp * (h + vel[n] * c) +
                  s0 * (rho * (hr - hl - vel[n] * dn) + w0 * h - dp))}
    for v in t:
        diss[v] = (sm * wm + sp * wp) * vel[v] + s0 * (w0 * vel[v] + rho * (R[v] - L[v]))

    def flux(q, e):
        F = [q[IDN] * q[n]] + [q[IDN] * q[n] * q[v] for v in (IVX, IVY, IVZ)]
        F[n] = F[n] + q[IPR]
        return F + [(e + q[IPR]) * q[n]]

    fl, fr = flux(L, el), flux(R, er)
    F = []
    for v in range(5):
        x = 0.5 * (fl[v] + fr[v]) - 0.5 * diss[v]
        F.append(torch.where(vel[n] - c > 0, fl[v], torch.where(vel[n] + c < 0, fr[v], x)))
    # intermediate densities below zero: local Lax-Friedrichs
    bad = (L[IDN] + wm < 0) | (L[IDN] + wm + w0 < 0)
    s = 0.5 * torch.maximum(L[n].abs() + torch.sqrt(gam * L[IPR] / L[IDN]),
                            R[n].abs() + torch.sqrt(gam * R[IPR] / R[IDN]))
    ul, ur = ([q[IDN]] + [q[IDN] * q[v] for v in (IVX, IVY, IVZ)] + [e] for q, e in ((L, el),
                                                                                    (R, er)))
    return [torch.where(bad, 0.5 * (fl[v] + fr[v]) - s * (ur[v] - ul[v]), F[v]) for v in range(5)]


def _diffusion(c, w):
    """area-weighted differences of the viscous and conductive fluxes"""
    act, dx = _active(c), _spacing(c)
    area = (dx[2] * dx[1], dx[2] * dx[0], dx[1] * dx[0])
    n = (c.nx1, c.nx2, c.nx3)
    out = 0.0
    for a in range(3):
        if not act[a]:
            continue

        def at(x, *shifts):
            """x at the faces of axis a, cells shifted by (axis, cells)"""
            for b in range(3):
                if act[b]:
                    x = x.narrow(2 - b, c.nghost + sum(s for k, s in shifts if k == b),
                                 n[b] + (b == a))
            return x

        def slope(x, b, *shifts):
            return (at(x, (b, 1), *shifts) - at(x, (b, -1), *shifts)) / (2.0 * dx[b])

        lo = (a, -1)
        rho = 0.5 * (at(w[IDN]) + at(w[IDN], lo))
        div = sum(0.5 * (slope(w[IVX + b], b) + slope(w[IVX + b], b, lo))
                  for b in range(3) if act[b])
        F = [torch.zeros_like(rho)]
        heat = 0.0
        for b in range(3):
            v = w[IVX + b]
            stress = (at(v) - at(v, lo)) / dx[a]
            if b == a:
                stress = 2.0 * stress - (2.0 / 3.0) * div
            elif act[b]:
                stress = stress + 0.5 * (slope(w[IVX + a], b) + slope(w[IVX + a], b, lo))
            m = -c.nu_iso * rho * stress
            F.append(m)
            heat = heat + 0.5 * (at(v) + at(v, lo)) * m
        temp = w[IPR] / (w[IDN] * c.rgas)
        cv = c.rgas / (c.gammad - 1.0)
        F.append(heat - c.kappa_iso * rho * cv * (at(temp) - at(temp, lo)) / dx[a])
        F = torch.stack(F)
        out = out + area[a] * (F.narrow(3 - a, 1, n[a]) - F.narrow(3 - a, 0, n[a]))
    return out


def _explicit(c, u, s, dt):
    """(du, ds, w): interior tendencies times dt, and the primitive state"""
    solver = (_roe, _lmars, _hllc)[c.riemann]
    w = _primitive(c, u)
    q = w if s is None else torch.cat([w, s / u[IDN]])
    act, dx, ng = _active(c), _spacing(c), c.nghost
    area = (dx[2] * dx[1], dx[2] * dx[0], dx[1] * dx[0])
    vol = dx[0] * dx[1] * dx[2]
    n = (c.nx1, c.nx2, c.nx3)
    it = _interior(c)
    div = 0.0
    for a in range(3):
        if not act[a]:
            continue
        cut = tuple(it[k] if k != 2 - a else slice(None) for k in range(3))
        L, R = zip(*[_faces(c, q[v][cut], a, ng, n[a], v) for v in range(q.shape[0])])
        L, R = list(L), list(R)
        if a == 0 and c.grav1 != 0.0:  # the walls' faces see the interior side only
            for v in (IDN, IPR):
                l, r = L[v], R[v]
                L[v] = torch.cat([r[..., :1], l[..., 1:]], -1)
                R[v] = torch.cat([r[..., :-1], l[..., -1:]], -1)
        F = solver(L, R, IVX + a, c.gammad)
        F += [F[IDN] * torch.where(F[IDN] > 0, L[v], R[v]) for v in range(5, q.shape[0])]
        F = torch.stack(F)
        div = div + area[a] * (F.narrow(3 - a, 1, n[a]) - F.narrow(3 - a, 0, n[a]))
    if c.nu_iso > 0 or c.kappa_iso > 0:
        div = div + _diffusion(c, w)
    d = -dt / vol * div
    du, ds = d[:5], d[5:]
    wi = w[(slice(None),) + it]
    zero = torch.zeros_like(wi[0])
    for k, g in enumerate((c.grav1, c.grav2, c.grav3)):
        if g != 0.0:
            add = [zero] * 5
            add[IVX + k] = dt * g * wi[IDN]
            add[IPR] = dt * g * wi[IDN] * wi[IVX + k]
            du = du + torch.stack(add)
    return du, ds, w


def _jacobian(w, gm1, sel):
    """rows and columns sel of the x1 flux Jacobian, [..., N, N]"""
    vx, vy, vz = w[IVX], w[IVY], w[IVZ]
    s2 = vx * vx + vy * vy + vz * vz
    hp = (gm1 + 1.0) / gm1 * w[IPR] / w[IDN]
    z, o = torch.zeros_like(vx), torch.ones_like(vx)
    J = [[z, o, z, z, z],
         [gm1 * s2 / 2 - vx * vx, (2 - gm1) * vx, -gm1 * vy, -gm1 * vz, gm1 * o],
         [-vx * vy, vy, vx, z, z],
         [-vx * vz, vz, z, vx, z],
         [((gm1 - 1) * s2 / 2 - hp) * vx, hp + s2 / 2 - gm1 * vx * vx, -gm1 * vx * vy,
          -gm1 * vx * vz, (gm1 + 1) * vx]]
    return torch.stack([torch.stack([J[r][q] for q in sel], -1) for r in sel], -2)


def _roe_matrix(l, r, gm1, sel):
    """rows and columns sel of |A| = R |lambda| R^-1 at the Roe average"""
    a, b = torch.sqrt(l[IDN]), torch.sqrt(r[IDN])
    vx, vy, vz = ((a * l[v] + b * r[v]) / (a + b) for v in (IVX, IVY, IVZ))
    gam = gm1 + 1.0
    h = ((_energy(l, gam) + l[IPR]) / a + (_energy(r, gam) + r[IPR]) / b) / (a + b)
    ke = 0.5 * (vx * vx + vy * vy + vz * vz)
    cs = torch.sqrt(gm1 * (h - ke))
    hp = h - ke
    z, o = torch.zeros_like(vx), torch.ones_like(vx)
    R = [[o, o, o, z, z], [vx - cs, vx, vx + cs, z, z], [vy, vy, vy, o, z], [vz, vz, vz, z, o],
         [h - vx * cs, ke, h + vx * cs, vy, vz]]
    k, i = 1.0 / (2.0 * cs * hp), 1.0 / hp
    V = [[(cs * ke + vx * hp) * k, -(hp + cs * vx) * k, -0.5 * vy * i, -0.5 * vz * i, 0.5 * i],
         [(hp - ke) * i, vx * i, vy * i, vz * i, -i],
         [(cs * ke - vx * hp) * k, (hp - cs * vx) * k, -0.5 * vy * i, -0.5 * vz * i, 0.5 * i],
         [-vy, z, o, z, z], [-vz, z, z, o, z]]
    lam = [(vx - cs).abs(), vx.abs(), (vx + cs).abs(), vx.abs(), vx.abs()]
    return torch.stack([torch.stack([sum(R[p][m] * lam[m] * V[m][q] for m in range(5))
                                     for q in sel], -1) for p in sel], -2)


def _implicit(c, du, w, dt):
    """vertically implicit correction: block-tridiagonal solve per column and
    the redistribution that keeps each column's mass; (du, mass fix)"""
    sel = range(5) if c.implicit_scheme & 8 else (IDN, IVX, IPR)
    gm1, dx, ng, nl = c.gammad - 1.0, _spacing(c), c.nghost, c.nx1
    it = _interior(c)
    col = w[(slice(None), it[0], it[1], slice(ng - 1, ng + nl + 1))]
    J = _jacobian(col, gm1, sel)
    A = _roe_matrix(col[..., :-1], col[..., 1:], gm1, sel)
    N = len(sel)
    half = 0.5 / dx[0]
    one = torch.eye(N, dtype=du.dtype, device=du.device)
    diag = one / dt
    diag = diag - torch.zeros_like(one).index_put(
        (torch.tensor([1, N - 1], device=du.device), torch.tensor([0, 1], device=du.device)),
        torch.tensor([c.grav1, c.grav1], dtype=du.dtype, device=du.device))
    mirror = one.clone()
    mirror[1, 1] = -1.0
    rhs = torch.stack([du[v] for v in sel], -1) / dt
    up, part = [], []
    for i in range(nl):
        Am, Ap = A[..., i, :, :], A[..., i + 1, :, :]
        a = half * (Am + Ap) + diag
        b = -half * (Am + J[..., i, :, :])
        d = -half * (Ap - J[..., i + 2, :, :])
        r = rhs[..., i, :, None]
        if i == 0:
            a = a + b @ mirror
        else:
            a, r = a - b @ up[-1], r - b @ part[-1]
        if i == nl - 1:
            a = a + d @ mirror
        x = torch.linalg.solve_ex(a, torch.cat([d, r], -1))[0]
        up.append(x[..., :N])
        part.append(x[..., N:])
    sol = [part[-1]]
    for i in range(nl - 2, -1, -1):
        sol.append(part[i] - up[i] @ sol[-1])
    x = torch.stack(sol[::-1], -3)[..., 0]
    rho = w[IDN][it]
    back = (du[IDN] - x[..., 0]).sum(-1, keepdim=True) / (rho * rho).sum(-1, keepdim=True)
    new = [du[v] for v in range(5)]
    for k, v in enumerate(sel):
        new[v] = x[..., k]
    new[IDN] = new[IDN] + rho * rho * back
    return torch.stack(new), x[..., 0] - du[IDN]


def _stage(c, k, dt, u, s, u0, s0):
    """one RK stage: (u, s, w) with w the primitive state of the input"""
    du, ds, w = _explicit(c, u, s, dt)
    it = (slice(None),) + _interior(c)
    if c.implicit_scheme:
        du, fix = _implicit(c, du, w, dt)
        if s is not None:
            ds = ds + fix * (s / u[IDN])[it]

    def advance(x, x0, d, kind):
        new = RK3[k][0] * x0[it] + RK3[k][1] * x[it] + RK3[k][2] * d
        pad = [n for nx in (c.nx1, c.nx2, c.nx3) for n in [c.nghost if nx > 1 else 0] * 2]
        return _fill(c, torch.nn.functional.pad(new, pad), kind)

    return advance(u, u0, du, "u"), None if s is None else advance(s, s0, ds, "s"), w


def _step(c, dt, u, s):
    u0, s0 = u, s
    for k in range(3):
        u, s, w = _stage(c, k, dt, u, s, u0, s0)
    return u, s, w


def _exact_block(case, opts, seed):
    c = opts.hydro
    w0, r = _state(case, opts, seed)
    u, s, w0 = _conserved(c, w0, r)
    dt = _dt(c, opts.integration.cfl, w0)
    u, s, w = _step(c, dt, u, s)
    if case["kind"] != "block64":  # stored about the horizontal mean of the initial state
        it = _interior(c)
        for v in (IDN, IPR):
            ref = w0[v][it[0], it[1], :].mean(dim=(0, 1))
            w[v] -= ref
            u[v] -= ref / (c.gammad - 1.0) if v == IPR else ref
    return u, w, s, dt.reshape(1)


def exact(case, seed):
    if case["kind"] == "ensemble":
        got = []
        for m, size in enumerate(_sizes(case)):
            got.append(_exact_block(case, _options(case, size), seed * 1009 + m))
        return {"u": [g[0] for g in got], "dt": torch.cat([g[3] for g in got])}
    opts = _options(case, _sizes(case)[0])
    c = opts.hydro
    if case["kind"] in ("block64", "block32"):
        u, w, s, dt = _exact_block(case, opts, seed)
        return {"u": u, "w": w, "s": s, "dt": dt}
    if case["kind"] == "tendency":
        w, r = _state(case, opts, seed)
        u, _, w = _conserved(c, w, r)
        dt = _dt(c, opts.integration.cfl, w)
        du, _, w = _explicit(c, u, None, dt)
        if c.implicit_scheme:
            du, _ = _implicit(c, du, w, dt)
        full = torch.zeros(c.shape, dtype=torch.float64, device="cuda")
        full[(slice(None),) + _interior(c)] = du
        return {"du": full, "w": w}
    u, s, dts = _rollout_inputs(case, opts, seed)
    gu, gs = _cotangents(case, opts, seed)
    leaves = [x.requires_grad_() for x in (u, s) if x is not None]
    for dt in dts:
        u, s, _ = _step(c, dt, u, s)
    if s is None:
        return {"u": u.detach(), "gu": torch.autograd.grad(u, leaves, gu)[0]}
    g = torch.autograd.grad((u, s), leaves, (gu, gs))
    return {"u": u.detach(), "s": s.detach(), "gu": g[0], "gs": g[1]}
