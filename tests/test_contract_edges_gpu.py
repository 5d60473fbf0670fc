"""The proton contraction at the edges of its launches, against the oracle
(1e-12 of the largest value, as in test_contract_gpu.py): one time-slice, site
counts off the block's 32, an x extent beyond the Fourier sum's 256 threads,
and more momenta than the work field holds."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.golden.make_golden import twop_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,xsrc,t0,t1,nmom", [
    ((2, 3, 3, 5), (1, 2, 0, 4), 0, 1, 1),
    ((5, 3, 2, 3), (3, 0, 1, 2), 2, 2, 4),
    ((3, 260, 2, 2), (2, 259, 1, 0), 0, 2, 2),
    ((4, 2, 2, 2), (0, 1, 1, 1), 1, 3, 400),
])
def test_twop_edges(gpu, orc, L, xsrc, t0, t1, nmom):
    _, cu, cd, prop = twop_inputs(orc, L, 51)
    moms = [(k % 3 - 1, k // 3 % 5 - 2, k // 15 % 3) for k in range(nmom)]
    fu, fd = [q.Field(L).load(c) for c in cu], [q.Field(L).load(c) for c in cd]
    corr = q.twop_proton(fu, fd, xsrc, t0, t1, moms)
    want = orc.twop_proton(prop(cu), prop(cd), L, xsrc, t0, t1, moms)
    assert np.max(np.abs(corr - want)) <= 1e-12 * np.max(np.abs(want))
    for f in fu + fd:
        f.close()
