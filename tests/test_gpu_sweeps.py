"""The FP64 sweeps at the sizes where their split changes: segments and packed
columns of the x1 sweep, remainders of 32-cell rounds, short march segments,
every compile-time face profile and the run-time one, against the CPU oracle.

One RK3 step of a rough random state; the bound is the per-step one of
test_gpu_parity.py (1e-12 of each variable's state scale per step)."""
import numpy as np
import pytest

from snapy_linfel_b200.config import Integration, MeshBlockOptions, make_config

from errnorm import assert_finite, state_err
from test_gpu_parity import _run_gpu, _run_oracle, random_prim

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _check(oracle, nx, seed=3, **kw):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ns = kw.get("nscalar", 0)
    grav = kw.pop("g", -0.2)
    cfg = make_config(nx1=nx[0], nx2=nx[1], nx3=nx[2], x1=(0.0, 0.1 * nx[0]),
                      x2=(0.0, 0.1 * nx[1]), x3=(0.0, 0.1 * nx[2]),
                      grav=(grav if nx[0] > 1 else 0.0, 0.0, 0.0), **kw)
    opts = MeshBlockOptions(cfg, Integration(cfl=0.3))
    rng = np.random.default_rng(seed)
    w = random_prim(rng, cfg.shape)
    r = rng.random(cfg.scalar_shape) if ns else None
    dts = [0.01]
    mb, _ = _run_gpu(opts, w, r, 1, dts=dts)
    u, s, _ = _run_oracle(oracle, opts, w, r, 1, dts=dts)
    got = mb.hydro_u.cpu().numpy()
    assert state_err(got, u, u) < 1e-12  # ghost cells included
    if ns:
        gs = mb.scalar_s.cpu().numpy()
        assert_finite(gs)
        assert np.max(np.abs(gs - s)) < 1e-12 * np.max(np.abs(s))


@pytest.mark.parametrize("nx1", [3, 28, 29, 30, 31, 33, 61, 62, 127, 257, 1500])
@pytest.mark.parametrize("bc", ["outflow", "reflecting", "periodic"])
def test_one_dimensional_segments(oracle, nx1, bc):
    """a column split into segments over warps, ghosts filled by the cells"""
    _check(oracle, (nx1, 1, 1), shock1=True, bc=(bc,) * 6, nscalar=nx1 % 2,
           scalar_recon="weno5", g=-0.2 if bc == "reflecting" else 0.0)


@pytest.mark.parametrize("nx", [(30, 7, 1), (31, 40, 1), (65, 3, 5), (5, 60, 50), (9, 61, 45),
                                (33, 50, 50), (64, 52, 48)])
def test_column_packing_and_remainders(oracle, nx):
    """whole columns end to end in one warp, and a few long ones"""
    _check(oracle, nx, riemann="lmars", bc=("reflecting",) * 4 + ("periodic",) * 2)


@pytest.mark.parametrize("n2", [3, 7, 8, 9, 33, 64, 65])
def test_march_segments(oracle, n2):
    _check(oracle, (6, n2, 4), riemann="roe", bc=("outflow",) * 2 + ("reflecting",) * 4)


@pytest.mark.parametrize("riemann", ["lmars", "hllc", "roe"])
@pytest.mark.parametrize("recon", ["weno5", "shock", "scaled", "plm", "weno3", "cp3", "mixed"])
@pytest.mark.parametrize("nscalar", [0, 1, 2, 3])
def test_face_profiles(oracle, riemann, recon, nscalar):
    kw = {"weno5": dict(scalar_recon="weno5"),
          "shock": dict(shock1=True, shock23=True, scalar_recon="weno5"),
          "scaled": dict(scale1=True, scale23=True, scalar_recon="weno5", scalar_scale=True),
          "plm": dict(recon1="plm", recon23="plm", scalar_recon="plm"),
          "weno3": dict(recon1="weno3", recon23="weno3", scalar_recon="weno3"),
          "cp3": dict(recon1="cp3", recon23="cp3", scalar_recon="cp3"),
          "mixed": dict(recon1="plm", recon23="weno5", scalar_recon="dc")}[recon]
    _check(oracle, (11, 6, 5), riemann=riemann, nscalar=nscalar,
           bc=("reflecting",) * 2 + ("periodic",) * 4, **kw)


@pytest.mark.parametrize("riemann,nscalar", [("lmars", 0), ("hllc", 1), ("roe", 2), ("lmars", 3)])
@pytest.mark.parametrize("nx", [(3, 5, 1), (29, 40, 1), (62, 3, 5), (90, 1, 1), (300, 4, 1),
                                (5, 50, 48), (20, 61, 45), (64, 52, 48)])
def test_fp32_sweeps_match_fp64(nx, riemann, nscalar):
    """The FP32 form's sweeps at the sizes where their split changes (segments,
    packed columns, short march segments; a 1-D column is not cut), without a
    reference profile, against the FP64 form of the same state: 1e-5 of each
    variable's scale, the FP32 form's accuracy target."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from snapy_linfel_b200.mesh import MeshBlock, MeshBlockF32

    cfg = make_config(nx1=nx[0], nx2=nx[1], nx3=nx[2], x1=(0.0, 0.1 * nx[0]),
                      x2=(0.0, 0.1 * nx[1]), x3=(0.0, 0.1 * nx[2]), grav=(-0.2, 0.0, 0.0),
                      riemann=riemann, nscalar=nscalar, scalar_recon="weno5",
                      bc=("reflecting",) * 4 + ("periodic",) * 2)
    opts = MeshBlockOptions(cfg, Integration(cfl=0.3))
    rng = np.random.default_rng(sum(nx))
    w = random_prim(rng, cfg.shape)
    r = rng.random(cfg.scalar_shape) if nscalar else None
    m64, m32 = MeshBlock(opts), MeshBlockF32(opts)
    m64.initialize(w, r)
    m32.initialize(w, r, reference=None)
    for m in (m64, m32):
        m.step(0.01)
    a, b = m32.state64().cpu().numpy(), m64.hydro_u.cpu().numpy()
    assert state_err(a, b, b) < 1e-5
    if nscalar:
        sa, sb = m32.scalar_s.double().cpu().numpy(), m64.scalar_s.cpu().numpy()
        assert_finite(sa)
        assert np.max(np.abs(sa - sb)) < 1e-5 * np.max(np.abs(sb))


@pytest.mark.parametrize("nu,kappa", [(0.02, 0.0), (0.0, 0.03), (0.02, 0.03)])
@pytest.mark.parametrize("nx", [(40, 1, 1), (1, 33, 1), (9, 17, 1), (1, 1, 21), (11, 1, 13),
                                (1, 9, 12), (12, 7, 19)])
def test_diffusion_axes(oracle, nx, nu, kappa):
    """every set of active axes of the diffusive fluxes"""
    _check(oracle, nx, nu_iso=nu, kappa_iso=kappa,
           bc=("reflecting",) * 2 + ("periodic",) * 4)


@pytest.mark.parametrize("nx", [(3, 1, 1), (300, 1, 1), (16, 16, 16), (17, 241, 1), (64, 65, 1),
                                (5, 60, 41), (129, 7, 9), (200, 90, 80)])
def test_time_step_reduction(nx):
    """the CFL limit by one CTA, by many, and over several rounds of the grid;
    a cell without a finite speed does not count.  FP64: the same operations in
    the same order, within 2 ulp; FP32 speeds: within 4 FP32 ulp."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from snapy_linfel_b200.mesh import MeshBlock, MeshBlockF32

    cfg = make_config(nx1=nx[0], nx2=nx[1], nx3=nx[2], x1=(0.0, 0.1 * nx[0]),
                      x2=(0.0, 0.13 * nx[1]), x3=(0.0, 0.17 * nx[2]))
    opts = MeshBlockOptions(cfg, Integration(cfl=1.0))
    w = random_prim(np.random.default_rng(sum(nx)), cfg.shape)
    m64, m32 = MeshBlock(opts), MeshBlockF32(opts)
    m64.initialize(w)
    m32.initialize(w, reference=None)
    k, j, i = (n // 2 for n in w.shape[1:])
    w[0, k, j, i] = np.nan
    ng = [(n - m) // 2 for n, m in zip(w.shape[1:], nx[::-1])]
    v = w[(slice(None),) + tuple(slice(g, n - g) for g, n in zip(ng, w.shape[1:]))]
    cs = np.sqrt(cfg.gammad * v[4] / v[0])
    dt = min(np.nanmin(d / (np.abs(v[1 + a]) + cs))
             for a, (d, n) in enumerate(zip((0.1, 0.13, 0.17), nx)) if n > 1)
    for m, tol in ((m64, 5e-16), (m32, 5e-7)):
        m.hydro_w.copy_(torch.from_numpy(w))
        assert abs(float(m.max_time_step()) / dt - 1.0) < tol


@pytest.mark.parametrize("riemann", ["lmars", "hllc", "roe"])
@pytest.mark.parametrize("kw", [{}, dict(shock1=True, shock23=True),
                                dict(scale1=True, scale23=True)])
def test_no_mass_through_walls(riemann, kw):
    """a face on a reflecting wall has exactly mirrored states on its sides, so
    no mass crosses it: the mass of a closed block changes by the rounding of
    its own updates only (cells x 2^-53 x 3 stages of the mean cell mass)"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from snapy_linfel_b200.mesh import MeshBlock

    cfg = make_config(nx1=12, nx2=9, nx3=7, x1=(0.0, 1.2), x2=(0.0, 0.9), x3=(0.0, 0.7),
                      riemann=riemann, bc=("reflecting",) * 6, **kw)
    mb = MeshBlock(MeshBlockOptions(cfg, Integration(cfl=0.3)))
    mb.initialize(random_prim(np.random.default_rng(8), cfg.shape))
    it = (0,) + cfg.interior()
    m0 = mb.hydro_u[it].sum().item()
    mb.step(0.01)
    m1 = mb.hydro_u[it].sum().item()
    assert abs(m1 - m0) < m0 * 3 * 2.0 ** -53 * np.sqrt(12 * 9 * 7)


# lengths that segments of 30 cells leave one or two cells over of
SHORT_REST = [842, 871, 872, 901, 1022]


@pytest.mark.parametrize("nx", [(n, 1, 1) for n in SHORT_REST] +
                         [(842, 4, 1), (871, 4, 1), (871, 20, 1), (901, 4, 4), (872, 1, 4)])
@pytest.mark.parametrize("nghost", [3, 4])
def test_short_last_segment_under_gravity(oracle, nx, nghost):
    """the segment below a wall's reads no ghost cell: only the wall's own
    segment revises them"""
    _check(oracle, nx, nghost=nghost, nscalar=1, scalar_recon="weno5",
           bc=("reflecting",) * 4 + ("periodic",) * 2)


@pytest.mark.parametrize("nx", [(842, 4, 1), (871, 20, 1), (901, 3, 3)])
def test_fp32_short_last_segment_under_gravity(nx):
    """as above in the FP32 form (only its 2-D and 3-D columns are cut), against
    the FP64 form, and in an ensemble with a larger member, where a member is cut
    for its share of the chip: bit for bit the one-block run"""
    test_fp32_sweeps_match_fp64(nx, "lmars", 0)
    from snapy_linfel_b200.ensemble import Ensemble
    from snapy_linfel_b200.mesh import MeshBlockF32

    members = []
    for n in (nx, (60, 40, 30) if nx[2] > 1 else (200, 300, 1)):
        cfg = make_config(nx1=n[0], nx2=n[1], nx3=n[2], x1=(0.0, 0.1 * n[0]),
                          x2=(0.0, 0.1 * n[1]), x3=(0.0, 0.1 * n[2]), grav=(-0.2, 0.0, 0.0),
                          bc=("reflecting",) * 4 + ("periodic",) * 2)
        members.append((MeshBlockOptions(cfg, Integration(cfl=0.3)),
                        random_prim(np.random.default_rng(n[0]), cfg.shape), None))
    ens = Ensemble(members)
    ens.step()
    for (opts, w, r), b in zip(members, ens.blocks):
        mb = MeshBlockF32(opts)
        mb.initialize(w, r)
        mb.step()
        assert torch.equal(mb.hydro_u, b.hydro_u)


def test_no_mass_through_segments():
    """the two warps that form the face between their segments form the same
    flux: the mass of a closed block with gravity changes by the rounding of its
    own updates only (the bound of test_no_mass_through_walls)"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from snapy_linfel_b200.mesh import MeshBlock

    cfg = make_config(nx1=871, nx2=4, x1=(0.0, 87.1), x2=(0.0, 0.4), grav=(-0.2, 0.0, 0.0),
                      bc=("reflecting",) * 6)
    mb = MeshBlock(MeshBlockOptions(cfg, Integration(cfl=0.3)))
    mb.initialize(random_prim(np.random.default_rng(8), cfg.shape))
    it = (0,) + cfg.interior()
    m0 = mb.hydro_u[it].sum().item()
    mb.step(0.01)
    m1 = mb.hydro_u[it].sum().item()
    assert abs(m1 - m0) < m0 * 3 * 2.0 ** -53 * np.sqrt(871 * 4)


@pytest.mark.parametrize("gammad", [1.4, 5.0 / 3.0])
@pytest.mark.parametrize("units", ["air", "giant"])
def test_isentropic_ghosts_to_rounding(gammad, units):
    """the density and pressure that an x1 ghost takes from the edge cell, against
    45 digits.  With y = 1 +- n a g dz rho / p, p y^(1/a) and rho y^(1/a) / y: y
    holds 1.6 units of 2^-53 (its sum, and six roundings of a term below 0.1),
    1 / a <= 3.5 times that enters the power, which adds 4 (2 ulp), and the last
    products one each: 11.6 units for the pressure, 15 for the density."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ctypes
    from decimal import Decimal as D, getcontext

    from snapy_linfel_b200 import _lib

    dz, grav = (100.0, -9.8) if units == "air" else (2000.0, -24.8)
    cfg = make_config(nx1=12, nx2=70, x1=(0.0, 12 * dz), x2=(0.0, 7e3), gammad=gammad,
                      grav=(grav, 0.0, 0.0), bc=("reflecting",) * 4 + ("periodic",) * 2)
    rng = np.random.default_rng(4)
    w = random_prim(rng, cfg.shape)
    if units == "air":
        w[4] = rng.uniform(1e4, 1.2e5, w[4].shape)
        w[0] = w[4] / (287.0 * rng.uniform(200.0, 310.0, w[4].shape))
    else:
        w[4] = 10.0 ** rng.uniform(4.0, 6.0, w[4].shape)
        w[0] = w[4] / (3700.0 * rng.uniform(150.0, 400.0, w[4].shape))
    wg = torch.from_numpy(w).cuda()
    ug, du = torch.empty_like(wg), torch.empty_like(wg)
    L = _lib.lib()
    ws = torch.empty(L.snapb_workspace_size(ctypes.byref(cfg)), dtype=torch.uint8, device="cuda")
    dt = torch.tensor([1e-3], dtype=torch.float64, device="cuda")
    P = _lib.ptr
    _lib.check(L.snapb_prim2cons(ctypes.byref(cfg), P(wg), P(ug), _lib.stream_ptr()))
    _lib.check(L.snapb_hydro_forward(ctypes.byref(cfg), P(dt), P(ug), P(wg), P(du), None, P(ws),
                                     ctypes.c_size_t(ws.numel()), _lib.stream_ptr()))
    got = wg.cpu().numpy()[:, 0]
    getcontext().prec = 45
    g, h = D(cfg.gammad), D(cfg.grav1) * (D(cfg.x1max) - D(cfg.x1min)) / cfg.nx1
    a, ng = (g - 1) / g, cfg.nghost
    worst = [0.0, 0.0]
    for j in range(got.shape[1]):
        for edge, up in ((ng, -1), (ng + cfg.nx1 - 1, 1)):
            re, pe = D(float(got[0, j, edge])), D(float(got[4, j, edge]))
            for n in range(1, ng + 1):
                y = 1 + up * n * a * h * re / pe
                z = (y.ln() / a).exp()
                for q, (v, ref) in enumerate(((4, pe * z), (0, re * z / y))):
                    x = D(float(got[v, j, edge + up * n]))
                    worst[q] = max(worst[q], float(abs((x - ref) / ref)))
    assert worst[0] < 11.6 * 2.0 ** -53 and worst[1] < 15 * 2.0 ** -53, worst


@pytest.mark.parametrize("var", [0, 4])
def test_ghosts_of_an_unphysical_edge_are_nan(var):
    """a negative density or pressure in the edge cell has no isentropic ghosts"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ctypes

    from snapy_linfel_b200 import _lib

    cfg = make_config(nx1=12, nx2=5, x1=(0.0, 1.2), x2=(0.0, 0.5), grav=(-0.2, 0.0, 0.0),
                      bc=("reflecting",) * 4 + ("periodic",) * 2)
    w = random_prim(np.random.default_rng(4), cfg.shape)
    ng = cfg.nghost
    w[var, 0, ng + 2, ng] *= -1.0
    wg = torch.from_numpy(w).cuda()
    ug, du = torch.empty_like(wg), torch.empty_like(wg)
    L = _lib.lib()
    ws = torch.empty(L.snapb_workspace_size(ctypes.byref(cfg)), dtype=torch.uint8, device="cuda")
    dt = torch.tensor([1e-3], dtype=torch.float64, device="cuda")
    P = _lib.ptr
    _lib.check(L.snapb_prim2cons(ctypes.byref(cfg), P(wg), P(ug), _lib.stream_ptr()))
    _lib.check(L.snapb_hydro_forward(ctypes.byref(cfg), P(dt), P(ug), P(wg), P(du), None, P(ws),
                                     ctypes.c_size_t(ws.numel()), _lib.stream_ptr()))
    got = wg.cpu().numpy()[:, 0]
    assert np.isnan(got[[0, 4], ng + 2, :ng]).all()
    assert np.isfinite(got[[0, 4], ng + 1, :ng]).all()


@pytest.mark.parametrize("nx,grav", [((40, 1, 1), (0.0, 0.0, 0.0)), ((12, 9, 1), (0.0, 0.1, 0.0)),
                                     ((9, 6, 5), (0.0, 0.0, -0.1)), ((1, 9, 12), (-0.2, 0.1, 0.0)),
                                     ((1, 30, 1), (-0.2, 0.0, 0.0)), ((11, 7, 1), (-0.2, 0.1, 0.0))])
def test_hydrostatic_correction_only_where_it_is_formed(oracle, nx, grav):
    """non_hydrostatic < 1 without gravity along an active x1: the correction is
    zero (it was read from workspace that nothing had written, or past its end)"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = make_config(nx1=nx[0], nx2=nx[1], nx3=nx[2], x1=(0.0, 0.1 * nx[0]),
                      x2=(0.0, 0.1 * nx[1]), x3=(0.0, 0.1 * nx[2]), grav=grav,
                      non_hydrostatic=0.5, bc=("reflecting",) * 6)
    opts = MeshBlockOptions(cfg, Integration(cfl=0.3))
    w = random_prim(np.random.default_rng(5), cfg.shape)
    mb, _ = _run_gpu(opts, w, None, 1, dts=[0.01])
    u, _, _ = _run_oracle(oracle, opts, w, None, 1, dts=[0.01])
    assert state_err(mb.hydro_u.cpu().numpy(), u, u) < 1e-12
