"""GCR at the step counts where its Gram-Schmidt passes change shape (one pass
of fields per eight basis vectors, the norm summed in the last), on a lattice
with padding, against the oracle (1e-11, as in test_solvers_gpu.py)."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("shipped", [False, True])
@pytest.mark.parametrize("n", [1, 2, 8, 9, 17])
def test_gcr_steps(gpu, orc, n, shipped):
    L = (3, 5, 4, 7)
    u, b = orc.gauge_synthetic(L, 61, EPS_PLAQ_060), orc.gaussian_spinor(L, 62)
    geo = q.Geometry(L, TH)
    gf, src, sol = q.GaugeField(geo), q.Vector(geo), q.Vector(geo)
    gf.a[:] = u
    src.a[:] = b
    lib = q.lib()
    lib.qcdgpu_set_gcr_compat(int(shipped))
    try:
        assert lib.gcr(sol.ref, src.ref, gf.ref, 0.15, 0.02, n, geo.s) == 0
    finally:
        lib.qcdgpu_set_gcr_compat(0)
    ref, rc = orc.gcr(b, u, L, TH, 0.15, 0.02, n, fixed=not shipped)
    assert rc == 0
    assert np.max(np.abs(sol.a - ref)) <= 1e-11 * np.max(np.abs(ref))
    for o in (src, sol, gf):
        o.close()
    geo.close()


def test_gcr_zero_source_is_an_error(gpu, orc):
    """the norm of the second basis vector is not a number"""
    L = (4, 4, 4, 4)
    geo = q.Geometry(L, TH)
    gf, src, sol = q.GaugeField(geo), q.Vector(geo), q.Vector(geo)
    gf.a[:] = orc.gauge_synthetic(L, 63, EPS_PLAQ_060)
    src.a[:] = 0.0
    assert q.lib().gcr(sol.ref, src.ref, gf.ref, 0.15, 0.0, 3, geo.s) == 1
    for o in (src, sol, gf):
        o.close()
    geo.close()
