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
