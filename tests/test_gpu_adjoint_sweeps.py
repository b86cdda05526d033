"""The reverse of the x2 / x3 sweeps at the sizes where its segments change
(one short segment, remainders, many), every compile-time profile and the
run-time one, with the comparisons and bounds of test_gpu_adjoint.py: each entry
against torch autograd, and finite differences where there are tracers."""
import pytest

import test_gpu_adjoint as base
from test_gpu_adjoint import L  # noqa: F401

pytestmark = pytest.mark.gpu


def _spec(nx, riemann, **kw):
    return dict(cfg=dict(nx1=nx[0], nx2=nx[1], nx3=nx[2], x1=(0.0, 0.1 * nx[0]),
                         x2=(0.0, 0.1 * nx[1]), x3=(0.0, 0.1 * nx[2]), riemann=riemann,
                         bc=("outflow", "reflecting", "reflecting", "outflow", "periodic",
                             "periodic"), **kw), grav=False)


@pytest.mark.parametrize("recon23", ["weno5", "cp5"])
@pytest.mark.parametrize("riemann", ["lmars", "hllc", "roe"])
@pytest.mark.parametrize("nx", [(5, 3, 1), (4, 6, 3), (33, 7, 1), (3, 14, 5), (4, 15, 1),
                                (3, 5, 30), (3, 47, 1)])
def test_segments_match_autograd(L, nx, riemann, recon23, monkeypatch):  # noqa: F811
    monkeypatch.setitem(base.AUTOGRAD_CONFIGS, "case", _spec(nx, riemann, recon23=recon23))
    base.test_stage_adjoint_matches_torch_autograd(L, "case", 1)


@pytest.mark.parametrize("riemann", ["lmars", "hllc", "roe"])
@pytest.mark.parametrize("nscalar", [1, 2, 3])
@pytest.mark.parametrize("nx", [(6, 23, 1), (5, 7, 15)])
def test_segments_with_tracers_fd(L, nx, nscalar, riemann, monkeypatch):  # noqa: F811
    monkeypatch.setitem(base.CONFIGS, "case",
                        _spec(nx, riemann, nscalar=nscalar, scalar_recon="weno5"))
    base.test_stage_adjoint_fd(L, "case", 2)
