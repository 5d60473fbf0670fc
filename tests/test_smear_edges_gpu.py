"""Smearing kernels where their forms change hands, against the oracle: dense
time-slices of every remainder, point sources (whose empty spins and sites are
left out) beside dense ones, links that are not finite, and the two forms of
the SU(3) projection (closed form; Newton's iteration for ill-conditioned
sums). Bounds: a Gaussian step is a dozen FP64 operations of size 1 per value
(1e-13, as in test_smear_gpu.py); the closed projection loses 50 eps kappa^2
with kappa <= 20, the iteration 50 eps kappa with kappa <= 1000 among these
few hundred random links: both below 1e-11."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("L", [(2, 2, 2, 2), (3, 5, 3, 7), (4, 4, 4, 2), (5, 4, 8, 9)])
@pytest.mark.parametrize("kind", ["point", "dense"])
def test_gauss3d_slices(gpu, orc, L, kind):
    u = orc.gauge_synthetic(L, 41, EPS_PLAQ_060)
    t = L[0] - 1
    v = orc.gaussian_spinor(L, 42)
    if kind == "point":
        v[:] = 0.0
        v[t + L[0] * (1 + L[1] * (0 + L[2] * (L[3] - 1))), 2, 1, 0] = 1.0
    ref = v
    for _ in range(4):
        ref = orc.gauss3d(ref, u, L, 4.0, t)
    g, f = q.Gauge(L, TH).load(u), q.Field(L).load(v)
    q.gauss3d(f, g, 4.0, t, 4)
    out = f.store()
    assert rel(out, ref) <= 1e-13
    assert np.array_equal(out == 0.0, ref == 0.0)
    g.close()
    f.close()


def test_gauss3d_infinite_link_is_not_left_out(gpu, orc):
    """zero times an infinite link is not a number: nothing is skipped then"""
    L = (2, 4, 4, 4)
    u = orc.gauge_synthetic(L, 43, EPS_PLAQ_060)
    u[1 + L[0] * (2 + L[1] * (2 + L[2] * 2)), 1, 0, 0, 0] = np.inf
    v = np.zeros_like(orc.gaussian_spinor(L, 44))
    v[1, 0, 0, 0] = 1.0  # far from the infinite link
    g, f = q.Gauge(L, TH).load(u), q.Field(L).load(v)
    q.gauss3d(f, g, 4.0, 1, 1)
    with np.errstate(invalid="ignore"):
        ref = orc.gauss3d(v, u, L, 4.0, 1)
    assert np.isnan(ref).any()
    assert np.array_equal(np.isnan(f.store()), np.isnan(ref))
    g.close()
    f.close()


@pytest.mark.parametrize("links", ["synthetic", "random", "unit"])
@pytest.mark.parametrize("L", [(2, 3, 5, 2), (4, 4, 6, 3)])
def test_ape3d_projection_forms(gpu, orc, links, L):
    if links == "random":  # not in SU(3), any conditioning
        u = np.random.RandomState(45).standard_normal(orc.gauge_unit(L).shape)
    else:
        u = orc.gauge_unit(L) if links == "unit" else orc.gauge_synthetic(L, 46, EPS_PLAQ_060)
    g, o = q.Gauge(L, TH).load(u), q.Gauge(L, TH)
    q.ape3d(o, g, 0.5, 1)
    out, ref = o.store(), orc.ape3d(u, L, 0.5)
    assert rel(out, ref) <= (1e-11 if links == "random" else 1e-12)
    assert np.array_equal(out[:, 0], ref[:, 0])
    g.close()
    o.close()


@pytest.mark.parametrize("ape_n", [0, 1, 3])
def test_smeared_source_smears_the_slice_only(gpu, orc, ape_n):
    L = (5, 3, 4, 5)
    u = orc.gauge_synthetic(L, 47, EPS_PLAQ_060)
    ua = u
    for _ in range(ape_n):
        ua = orc.ape3d(ua, L, 0.5)
    x = (4, 2, 0, 3)
    ref = np.zeros((int(np.prod(L)), 4, 3, 2))
    ref[x[0] + L[0] * (x[1] + L[1] * (x[2] + L[2] * x[3])), 3, 2, 0] = 1.0
    for _ in range(6):
        ref = orc.gauss3d(ref, ua, L, 4.0, x[0])
    g, f = q.Gauge(L, TH).load(u), q.Field(L)
    q.smeared_source(f, g, x, 3, 2, 0.5, ape_n, 4.0, 6)
    assert rel(f.store(), ref) <= 1e-12
    assert np.array_equal(g.store(), u)
    g.close()
    f.close()
