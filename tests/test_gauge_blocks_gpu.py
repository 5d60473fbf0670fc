"""FP32 and FP16 links lie in blocks of 32 sites: what goes in comes out on
lattices of whole blocks, of one partial block and of blocks with a remainder,
for complete (FP32) and for two-row storage."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


# entries are at most 1: half an ulp of 2^-24 or 2^-11 each, and the rebuilt
# row adds eight products of them (FP32 arithmetic apart, in double)
@pytest.mark.parametrize("prec,tol,su3", [(q.F32, 6e-7, True), (q.F32, 1.2e-7, False), (q.F16, 4e-3, True)])
@pytest.mark.parametrize("L", [(4, 2, 2, 2), (2, 2, 2, 2), (3, 5, 4, 7), (4, 4, 4, 4)])
def test_links_round_trip(gpu, orc, L, prec, tol, su3):
    u = orc.gauge_synthetic(L, 81, EPS_PLAQ_060)
    if not su3:
        u[..., 2, :, :] *= 0.5  # the last row is no longer the rebuilt one
    g = q.Gauge(L, TH, prec).load(u)
    assert np.max(np.abs(g.store() - u)) <= tol
    g.close()
