"""The implicit solves at the sizes where they can go wrong.

5x5 blocks of the FP64 form (sixteen lanes a column, from both ends): odd and
even columns, the shortest ones, CTAs with columns missing.

The one-warp solve (3x3 blocks) at the column lengths where its
split changes: 8, 16 and 32 lanes a column, chunks of one layer and of many,
chunks past the column's end, warps with columns missing, and the longest
column it takes.

FP64: the correction and the mass fix against the CPU oracle, bound 1e-12 of
the state scale per call (test_gpu_parity.py).  FP32 form: against the column
sweep (SNAPB_VIC_KERNEL=column), which forms the same FP32 blocks with other
roundings and eliminates in FP64 too; bound 1e-5 of each variable's scale, the
form's own accuracy target.  Ensembles: every member bit for bit its one-block
result, members of all three lane counts together."""
import ctypes

import numpy as np
import pytest

from snapy_linfel_b200 import problems
from snapy_linfel_b200.config import Integration, MeshBlockOptions, make_config

from errnorm import assert_finite, state_err, state_scale
from test_gpu_parity import call, dev, random_prim

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from snapy_linfel_b200 import _lib

    return _lib


def _config(nl, nx2, nx3, scheme=1, **kw):
    return make_config(nx1=nl, nx2=nx2, nx3=nx3, x1=(0.0, 0.1 * nl), x2=(0.0, 0.1 * nx2),
                       x3=(0.0, 0.1 * nx3), grav=(-0.2, 0.0, 0.0), implicit_scheme=scheme,
                       bc=("reflecting",) * 4 + ("periodic",) * 2, **kw)


@pytest.mark.parametrize("nl,nx2,nx3", [
    (3, 5, 1), (7, 3, 3), (8, 4, 1), (9, 5, 5), (31, 3, 1), (32, 7, 1), (33, 3, 1), (63, 5, 1),
    (64, 4, 3), (65, 3, 1), (100, 3, 3), (127, 3, 1), (128, 5, 1), (129, 3, 1), (192, 3, 1),
    (257, 3, 1), (1216, 3, 1), (1217, 3, 1)])
def test_correction_matches_oracle(L, oracle, nl, nx2, nx3):
    _correction(L, oracle, nl, nx2, nx3, 1, 0.05)


@pytest.mark.parametrize("dt", [0.05, 5.0])
@pytest.mark.parametrize("nl,nx2,nx3", [(3, 3, 1), (4, 7, 1), (5, 8, 1), (6, 9, 1), (31, 3, 3),
                                        (64, 5, 3), (129, 17, 1)])
def test_five_by_five_correction_matches_oracle(L, oracle, nl, nx2, nx3, dt):
    _correction(L, oracle, nl, nx2, nx3, 9, dt)


def _correction(L, oracle, nl, nx2, nx3, scheme, dt):
    c = _config(nl, nx2, nx3, scheme)
    rng = np.random.default_rng(nl)
    w = random_prim(rng, c.shape)
    u = oracle.prim2cons(c, w)
    du = 0.05 * (rng.random(c.shape) - 0.5)
    ref, m_ref = du.copy(), np.zeros_like(u)
    oracle.implicit_correction(c, dt, ref, w, m_ref)
    ws = torch.empty(L.lib().snapb_workspace_size(ctypes.byref(c)), dtype=torch.uint8,
                     device="cuda")
    dug, wg, mg = dev(du), dev(w), torch.zeros(c.shape, dtype=torch.float64, device="cuda")
    dtg = torch.tensor([dt], dtype=torch.float64, device="cuda")
    call(L, "snapb_implicit_correction", ctypes.byref(c), L.ptr(dtg), L.ptr(dug), L.ptr(wg),
         L.ptr(mg), L.ptr(ws), ctypes.c_size_t(ws.numel()), L.stream_ptr())
    it = c.interior()
    full = (slice(None),) + it
    assert state_err(dug.cpu().numpy()[full], ref[full], u[full]) < 1e-12
    got = mg.cpu().numpy()[0][it]
    assert_finite(got)
    assert np.max(np.abs(got - m_ref[0][it])) < 1e-12 * np.max(np.abs(u[0]))


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("nl,nx2,nx3,ns", [(5, 9, 1, 0), (20, 6, 7, 2), (50, 5, 3, 1),
                                           (64, 9, 1, 3), (150, 4, 3, 2), (128, 6, 5, 0)])
def test_step_matches_column_sweep(L, monkeypatch, form, nl, nx2, nx3, ns):
    from snapy_linfel_b200.mesh import MeshBlock, MeshBlockF32

    c = _config(nl, nx2, nx3, nscalar=ns, scalar_recon="weno5", riemann="roe")
    opts = MeshBlockOptions(c, Integration(cfl=0.3))
    rng = np.random.default_rng(nl)
    w, r = random_prim(rng, c.shape), rng.random(c.scalar_shape) if ns else None
    out = []
    for env in ("", "column"):
        monkeypatch.setenv("SNAPB_VIC_KERNEL", env)
        mb = (MeshBlock if form == "fp64" else MeshBlockF32)(opts)
        mb.initialize(w, r)
        mb.step(0.01)
        mb.step(0.01)
        torch.cuda.synchronize()
        out.append((mb.hydro_u.double().cpu().numpy(),
                    mb.scalar_s.double().cpu().numpy() if ns else None))
    tol = 1e-12 * 2 if form == "fp64" else 1e-5
    (a, sa), (b, sb) = out
    assert_finite(a, b)
    scale = np.maximum(state_scale(b), 1e-3)
    assert np.all(np.abs(a - b).reshape(5, -1).max(axis=1) < tol * scale)
    if ns:
        assert_finite(sa, sb)
        assert np.max(np.abs(sa - sb)) < tol * np.max(np.abs(sb))


def test_ensemble_of_all_lane_counts_is_exact(L):
    from snapy_linfel_b200.ensemble import Ensemble
    from snapy_linfel_b200.mesh import MeshBlockF32

    members = problems.ensemble_members(n=9, seed=5, horiz=(6, 9, 13), vert=(20, 45, 100),
                                        riemann="hllc")
    assert {m[0].hydro.nx1 for m in members} == {20, 45, 100}
    ens = Ensemble(members)
    for _ in range(2):
        ens.step()
    for (opts, w, r), b in zip(members, ens.blocks):
        mb = MeshBlockF32(opts)
        mb.initialize(w, r)
        for _ in range(2):
            mb.step()
        assert torch.equal(mb.hydro_u, b.hydro_u)


@pytest.mark.parametrize("nl,nx2,nx3,ns", [(3, 5, 1, 0), (9, 7, 1, 1), (33, 5, 4, 2), (65, 3, 1, 0),
                                           (150, 5, 1, 2), (300, 3, 1, 0)])
def test_adjoint_solver_matches_sweep(L, monkeypatch, nl, nx2, nx3, ns):
    """the adjoint's two column solves by one warp per group of columns against
    the block-Thomas sweep (SNAPB_VADJ_SOLVE=sweep): the same stage gradient up
    to FP64 rounding, bound 1e-11 of each variable's largest entry (the bound
    of the sweep against cyclic reduction)"""
    from snapy_linfel_b200.adjoint import Adjoint
    from snapy_linfel_b200.mesh import MeshBlock

    c = _config(nl, nx2, nx3, nscalar=ns, scalar_recon="weno5", riemann="lmars")
    rng = np.random.default_rng(nl)
    mb = MeshBlock(MeshBlockOptions(c, Integration(cfl=0.3)))
    mb.initialize(random_prim(rng, c.shape), rng.random(c.scalar_shape) if ns else None)
    u = mb.hydro_u.clone()
    s = mb.scalar_s.clone() if ns else None
    dt = torch.tensor([0.02], dtype=torch.float64, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(nl)
    gout = torch.randn(u.shape, generator=gen, device="cuda", dtype=torch.float64)
    gsout = torch.randn(s.shape, generator=gen, device="cuda", dtype=torch.float64) if ns else None
    got = []
    for env in ("", "sweep"):
        monkeypatch.setenv("SNAPB_VADJ_SOLVE", env)
        gu0 = torch.zeros_like(u)
        gs0 = torch.zeros_like(s) if ns else None
        gu, gs = Adjoint(c).stage(1, dt, u, s, gout, gsout, gu0, gs0)
        torch.cuda.synchronize()
        got.append([gu.clone(), gu0.clone()] + ([gs.clone(), gs0.clone()] if ns else []))
    for a, b in zip(*got):
        assert torch.isfinite(a).all()
        for v in range(a.shape[0]):
            assert float((a[v] - b[v]).abs().max()) <= 1e-11 * float(b[v].abs().max()), v


@pytest.mark.parametrize("dt", [0.05, 5.0, 500.0])
@pytest.mark.parametrize("nl", [3, 6, 33, 64])
def test_five_by_five_column_is_its_own(L, nl, dt):
    """a column's result depends on no other column: the same bits when the
    column beside it in the warp holds another state, and when that state is
    not a number"""
    c = _config(nl, 4, 1, 9)
    rng = np.random.default_rng(nl)
    w = random_prim(rng, c.shape)
    du = 0.05 * (rng.random(c.shape) - 0.5)
    ws = torch.empty(L.lib().snapb_workspace_size(ctypes.byref(c)), dtype=torch.uint8,
                     device="cuda")
    dtg = torch.tensor([dt], dtype=torch.float64, device="cuda")
    ng, out = c.nghost, []
    for beside in ("same", "supersonic", "nan"):
        x = w.copy()
        if beside == "supersonic":
            x[1:4, :, ng + 1::2] *= 1e3
        elif beside == "nan":
            x[:, :, ng + 1::2] = np.nan
        dug, wg = dev(du), dev(x)
        call(L, "snapb_implicit_correction", ctypes.byref(c), L.ptr(dtg), L.ptr(dug), L.ptr(wg),
             None, L.ptr(ws), ctypes.c_size_t(ws.numel()), L.stream_ptr())
        got = dug.cpu().numpy()[:, 0, ng:ng + 4:2, ng:-ng]
        assert_finite(got)
        out.append(got)
    for got in out[1:]:
        assert np.array_equal(got, out[0])


def _solve80(c, du, w, dt):
    """the 3x3 correction of a 2-D block in 80 bits: pivoted block elimination from
    the lower wall up"""
    T, ng, nl = np.longdouble, c.nghost, c.nx1
    w, du = (x.astype(T)[:, 0, ng:-ng] for x in (w, du))
    sel, gm1, half = (0, 1, 4), T(c.gammad) - 1, nl / (2 * (T(c.x1max) - T(c.x1min)))
    col = w[..., ng - 1:ng + nl + 1]

    def rows(J):  # the rows and columns sel, [columns, layers, 3, 3]
        return np.stack([np.stack([J[r][q] for q in sel], -1) for r in sel], -2) * half

    rho, u, v, z, p = col
    o, n, s2, hp = np.ones_like(u), np.zeros_like(u), u * u + v * v + z * z, (gm1 + 1) / gm1 * p / rho
    J = rows([[n, o, n, n, n], [gm1 * s2 / 2 - u * u, (2 - gm1) * u, n, n, gm1 * o], None, None,
              [((gm1 - 1) * s2 / 2 - hp) * u, hp + s2 / 2 - gm1 * u * u, n, n, (gm1 + 1) * u]])
    l, r = col[..., :-1], col[..., 1:]
    a, b = np.sqrt(l[0]), np.sqrt(r[0])
    u, v, z = ((a * l[k] + b * r[k]) / (a + b) for k in (1, 2, 3))
    en = [x[4] / gm1 + x[0] * (x[1] ** 2 + x[2] ** 2 + x[3] ** 2) / 2 for x in (l, r)]
    h = ((en[0] + l[4]) / a + (en[1] + r[4]) / b) / (a + b)
    ke = (u * u + v * v + z * z) / 2
    hp = h - ke
    cs, o, n = np.sqrt(gm1 * hp), np.ones_like(u), np.zeros_like(u)
    R = {0: [o, o, o, n, n], 1: [u - cs, u, u + cs, n, n], 4: [h - u * cs, ke, h + u * cs, v, z]}
    k, i = 1 / (2 * cs * hp), 1 / hp
    V = [[(cs * ke + u * hp) * k, -(hp + cs * u) * k, 0, 0, i / 2],
         [(hp - ke) * i, u * i, 0, 0, -i],
         [(cs * ke - u * hp) * k, (hp - cs * u) * k, 0, 0, i / 2],
         [-v, n, 0, 0, n], [-z, n, 0, 0, n]]
    lam = [abs(u - cs), abs(u), abs(u + cs), abs(u), abs(u)]
    A = rows({p: {q: sum(R[p][m] * lam[m] * V[m][q] for m in range(5)) for q in sel} for p in sel})
    g = np.zeros((3, 3), T)
    g[1, 0] = g[2, 1] = c.grav1
    diag, mirror = np.eye(3, dtype=T) / T(dt) - g, np.diag(np.array([1, -1, 1], T))
    D = du[..., ng:ng + nl]

    def solve(a, r):
        a, r, ix = a.copy(), r.copy(), np.arange(len(a))
        for j in range(3):
            size = np.abs(a[:, j:, j]) / np.maximum(np.abs(a[:, j:]).max(-1), T(1e-300))
            pv = j + np.argmax(size, 1)
            for m in (a, r):
                m[ix, pv], m[:, j] = m[:, j].copy(), m[ix, pv].copy()
            piv = a[:, j, j][:, None].copy()
            a[:, j], r[:, j] = a[:, j] / piv, r[:, j] / piv
            for i in set(range(3)) - {j}:
                f = a[:, i, j][:, None].copy()
                a[:, i], r[:, i] = a[:, i] - f * a[:, j], r[:, i] - f * r[:, j]
        return r

    up, part = [], []
    for i in range(nl):
        a = A[:, i] + A[:, i + 1] + diag
        b, d = -(A[:, i] + J[:, i]), -(A[:, i + 1] - J[:, i + 2])
        r = np.stack([D[v][:, i] for v in sel], -1)[..., None] / T(dt)
        if i == 0:
            a = a + b @ mirror
        else:
            a, r = a - b @ up[-1], r - b @ part[-1]
        if i == nl - 1:
            a = a + d @ mirror
        x = solve(a, np.concatenate([d, r], -1))
        up.append(x[..., :3])
        part.append(x[..., 3:])
    x = [part[-1]]
    for i in range(nl - 2, -1, -1):
        x.append(part[i] - up[i] @ x[-1])
    x, out = np.stack(x[::-1], 1)[..., 0], D.copy()
    rho = w[0][..., ng:ng + nl]
    out[1], out[4] = x[..., 1], x[..., 2]
    back = (D[0] - x[..., 0]).sum(-1, keepdims=True) / (rho * rho).sum(-1, keepdims=True)
    out[0] = x[..., 0] + rho * rho * back
    return out


def _column_state(kind, c, seed):
    """rough: independent cells; smooth: a stratified column whose vertical flow
    (300 m/s, near sonic) changes its sign a few times; du of either"""
    rng = np.random.default_rng(seed)
    w = random_prim(rng, c.shape)
    du = 0.05 * (rng.random(c.shape) - 0.5)
    if kind == "smooth":
        z = (np.arange(c.shape[-1]) - 2.5) * 100.0
        x = np.linspace(0, 2 * np.pi, c.shape[-1])
        wave = [sum(rng.standard_normal((1, c.shape[2], 1)) *
                    np.sin(k * x + 6 * rng.random((1, c.shape[2], 1))) for k in (1, 2, 3, 5))
                for _ in range(5)]
        w[4] = 1e5 * np.exp(-z / 8000.0) * (1 + 1e-3 * np.clip(wave[4], -3, 3))
        w[0] = w[4] / (287.0 * (300.0 - 0.0065 * z)) * (1 + 1e-3 * np.clip(wave[0], -3, 3))
        w[1:4] = 300.0 * np.stack(wave[1:4])
        du *= w[[0, 0, 0, 0, 4]]
    return w, du


@pytest.mark.parametrize("kind,nl,dt", [("rough", 3, 20.0), ("rough", 8, 20.0), ("rough", 17, 20.0),
                                        ("rough", 33, 20.0), ("rough", 64, 20.0),
                                        ("rough", 90, 20.0), ("rough", 129, 1.0),
                                        ("smooth", 30, 10.0), ("smooth", 64, 10.0),
                                        ("smooth", 128, 3.0), ("smooth", 128, 30.0)])
def test_correction_at_large_courant_numbers(L, oracle, kind, nl, dt):
    """vertical Courant numbers of 10 to 300 where the flow converges in stretches
    of layers, which are then nearly singular: no further from 80 bits than 64 times
    the oracle's sequential FP64 solve (the columns that the chunked solve keeps are
    within 26 times), or 64 units of 2^-53 where the oracle is nearer than one"""
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no 80-bit floating point")
    big = kind == "smooth"
    c = make_config(nx1=nl, nx2=12, x1=(0.0, (100.0 if big else 0.1) * nl), x2=(0.0, 1200.0),
                    grav=(-9.8 if big else -0.2, 0.0, 0.0), implicit_scheme=1,
                    bc=("reflecting",) * 4 + ("periodic",) * 2)
    w, du = _column_state(kind, c, nl)
    exact = _solve80(c, du, w, dt)
    ref = du.copy()
    oracle.implicit_correction(c, dt, ref, w, np.zeros_like(w))
    ws = torch.empty(L.lib().snapb_workspace_size(ctypes.byref(c)), dtype=torch.uint8,
                     device="cuda")
    dug, wg = dev(du), dev(w)
    dtg = torch.tensor([dt], dtype=torch.float64, device="cuda")
    call(L, "snapb_implicit_correction", ctypes.byref(c), L.ptr(dtg), L.ptr(dug), L.ptr(wg), None,
         L.ptr(ws), ctypes.c_size_t(ws.numel()), L.stream_ptr())
    ng = c.nghost
    scale = np.abs(exact).reshape(5, -1).max(1)[:, None, None]
    err = [np.max(np.abs(x[:, 0, ng:-ng, ng:-ng] - exact) / scale)
           for x in (dug.cpu().numpy(), ref)]
    assert_finite(np.array(err, dtype=np.float64))
    assert err[0] < 64 * max(err[1], 2.0 ** -53), err


def test_adjoint_at_large_courant_numbers(L, monkeypatch):
    """the adjoint's two column solves on such a column against the sequential
    sweep, whose own error is near 1e-11: bound 1e-6 of each variable's largest
    entry (1e-2 apart where the chunked solves kept the columns)"""
    from snapy_linfel_b200.adjoint import Adjoint
    from snapy_linfel_b200.mesh import MeshBlock

    c = make_config(nx1=128, nx2=12, x1=(0.0, 12800.0), x2=(0.0, 1200.0), grav=(-9.8, 0.0, 0.0),
                    implicit_scheme=1, riemann="lmars", bc=("reflecting",) * 4 + ("periodic",) * 2)
    mb = MeshBlock(MeshBlockOptions(c, Integration(cfl=0.3)))
    mb.initialize(_column_state("smooth", c, 128)[0])
    u = mb.hydro_u.clone()
    dt = torch.tensor([30.0], dtype=torch.float64, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(1)
    gout = torch.randn(u.shape, generator=gen, device="cuda", dtype=torch.float64)
    got = []
    for env in ("", "sweep"):
        monkeypatch.setenv("SNAPB_VADJ_SOLVE", env)
        gu, _ = Adjoint(c).stage(1, dt, u, None, gout, None, torch.zeros_like(u), None)
        got.append(gu.clone())
    a, b = got
    assert torch.isfinite(a).all() and torch.isfinite(b).all()
    for v in range(5):
        assert float((a[v] - b[v]).abs().max()) <= 1e-6 * float(b[v].abs().max()), v


@pytest.mark.parametrize("nl", [17, 40, 128, 300])
def test_columns_solved_in_sequence_are_their_own(L, nl):
    """columns that need the sequential solve beside ones that do not, in one
    warp: each has the bits that it has among its like"""
    c = _config(nl, 8, 1)
    rng = np.random.default_rng(nl)
    calm, wild = random_prim(rng, c.shape), random_prim(rng, c.shape)
    calm[:] = calm[..., :1]
    calm[1:4] *= 1e-3
    wild[1] = 3.0 * (rng.random(wild[1].shape) - 0.5)
    mixed, ng = calm.copy(), c.nghost
    mixed[:, :, ng + 1::2] = wild[:, :, ng + 1::2]
    du = 0.05 * (rng.random(c.shape) - 0.5)
    ws = torch.empty(L.lib().snapb_workspace_size(ctypes.byref(c)), dtype=torch.uint8,
                     device="cuda")
    dtg = torch.tensor([2.0], dtype=torch.float64, device="cuda")
    got = []
    for w in (calm, wild, mixed):
        dug, wg = dev(du), dev(w)
        call(L, "snapb_implicit_correction", ctypes.byref(c), L.ptr(dtg), L.ptr(dug), L.ptr(wg),
             None, L.ptr(ws), ctypes.c_size_t(ws.numel()), L.stream_ptr())
        got.append(dug.cpu().numpy()[:, 0, ng:-ng, ng:-ng])
        assert_finite(got[-1])
    assert np.array_equal(got[2][:, ::2], got[0][:, ::2])
    assert np.array_equal(got[2][:, 1::2], got[1][:, 1::2])


@pytest.mark.parametrize("nl", [17, 40, 128])
def test_fp32_columns_solved_in_sequence(L, nl):
    """the FP32 form's sequential solve, one stage on a supersonic rough state:
    finite, and the bits of the batched form"""
    from snapy_linfel_b200.ensemble import Ensemble
    from snapy_linfel_b200.mesh import MeshBlockF32

    members = []
    for n2 in (8, 11):
        c = _config(nl, n2, 1, riemann="lmars")
        w = random_prim(np.random.default_rng(nl + n2), c.shape)
        w[1] *= 60.0
        members.append((MeshBlockOptions(c, Integration(cfl=0.3)), w, None))
    ens = Ensemble(members)
    ens.dts().fill_(3.0)
    ens.stage(0)
    for (opts, w, r), b in zip(members, ens.blocks):
        mb = MeshBlockF32(opts)
        mb.initialize(w, r)
        mb.set_dt(3.0)
        mb.forward(0)
        assert torch.isfinite(mb.hydro_u).all()
        assert torch.equal(mb.hydro_u, b.hydro_u)
