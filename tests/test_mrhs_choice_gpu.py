"""The choice that mrhs_tuned reports can be asked for, and gives the same bits."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("n", [1, 3, 4, 6, 10])
def test_reported_choice_is_accepted(gpu, n):
    L = (4, 6, 4, 6)
    g, f = q.Gauge(L, TH).synthetic(97, EPS_PLAQ_060), q.Field(L)
    a, b = q.MField(L, n), q.MField(L, n)
    for k in range(n):
        a.set(k, f.gaussian(98 + k))

    def apply():
        q.dslash_mrhs(b, a, g, 0.15, 0.02)
        return [b.get(k, f).store() for k in range(n)]

    ref = apply()
    variant, threads = q.mrhs_tuned(L, n)
    assert variant == "simt"
    try:
        q.set_mrhs_variant(threads)
        for x, y in zip(apply(), ref):
            assert np.array_equal(x, y)
    finally:
        q.set_mrhs_variant(-1)
    for o in (a, b, f, g):
        o.close()
