"""GCR's passes over whole fields, after calls that used the library's memory
before it, on lattices whose component blocks are padded (a volume that is no
multiple of 128). Against the oracle, 1e-11 as in test_solvers_gpu.py."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060
from tests.golden.make_golden import twop_inputs

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


class Gcr:
    """gcr() and the oracle's on one lattice"""

    def __init__(self, orc, L, seed=71):
        self.orc, self.L = orc, L
        self.u, self.b = orc.gauge_synthetic(L, seed, EPS_PLAQ_060), orc.gaussian_spinor(L, seed + 1)
        self.geo = q.Geometry(L, TH)
        self.g, self.src, self.sol = q.GaugeField(self.geo), q.Vector(self.geo), q.Vector(self.geo)
        self.g.a[:] = self.u

    def run(self, src, sol, n):
        return q.lib().gcr(sol.ref, src.ref, self.g.ref, 0.15, 0.02, n, self.geo.s)

    def check(self, n, src=None, sol=None):
        src, sol = src or self.src, sol or self.sol
        src.a[:] = self.b
        assert self.run(src, sol, n) == 0
        ref, rc = self.orc.gcr(self.b, self.u, self.L, TH, 0.15, 0.02, n, fixed=True)
        assert rc == 0
        assert np.max(np.abs(sol.a - ref)) <= 1e-11 * np.max(np.abs(ref))

    def close(self):
        for o in (self.src, self.sol, self.g, self.geo):
            o.close()


def test_gcr_after_a_contraction(gpu, orc):
    L = (3, 5, 4, 7)
    _, cu, cd, _ = twop_inputs(orc, L, 51)
    fu, fd = [q.Field(L).load(c) for c in cu], [q.Field(L).load(c) for c in cd]
    s = Gcr(orc, L)
    q.release_work()
    q.twop_proton(fu, fd, (1, 2, 0, 4), 0, L[0] - 1, [(-1, -1, k - 3) for k in range(7)])
    s.check(9)
    s.close()
    for f in fu + fd:
        f.close()


@pytest.mark.parametrize("ape_n,Ls,L", [(2, (5, 6, 6, 6), (8, 6, 6, 6)), (0, (4, 4, 4, 5), (7, 4, 4, 5))])
def test_gcr_after_a_smeared_source(gpu, orc, ape_n, Ls, L):
    """L: the lattice of as many time-slices as the smearing's copies of a slice of Ls take"""
    g, f = q.Gauge(Ls, TH).load(orc.gauge_synthetic(Ls, 73, EPS_PLAQ_060)), q.Field(Ls)
    s = Gcr(orc, L)
    q.release_work()
    q.smeared_source(f, g, (3, 1, 2, 0), 1, 2, 0.5, ape_n, 4.0, 5)
    s.check(9)
    s.close()
    g.close()
    f.close()


def test_gcr_after_one_that_broke_down(gpu, orc):
    """the coefficients of a zero source are not numbers; they reach no padding"""
    s = Gcr(orc, (3, 5, 4, 7))
    q.release_work()
    s.src.a[:] = 0.0
    assert s.run(s.src, s.sol, 3) == 1
    other = q.Vector(s.geo)
    s.check(9, src=s.src, sol=other)  # with its basis and residual fields
    s.check(9, src=s.sol, sol=other)  # and with its solution as the next source
    other.close()
    s.close()
