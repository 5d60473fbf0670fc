"""The float-float operator where its launches change shape (one or four
groups of warps per 32 sites, below and above 9,728 sites; partial blocks) and
where its conversions do: empty sites, values outside the short split's range,
results whose low words are zero. Against the CPU oracle at the operator's
1e-13 per-site bar, D, D^+ and Q with twisted mass; the even/odd form by a
solve's FP64 true residual."""
import numpy as np
import pytest

import qcd_gb300 as q
from oracle.oracle import site_rel_err
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.2, 0.0)


@pytest.mark.parametrize("L", [(2, 2, 2, 2), (3, 5, 4, 7), (16, 8, 8, 8), (19, 8, 8, 8), (9, 9, 11, 11), (10, 11, 9, 12)])
def test_operator_on_both_sides_of_the_line(gpu, orc, L):
    u, v = orc.gauge_synthetic(L, 81, EPS_PLAQ_060), orc.gaussian_spinor(L, 82)
    g, fin, fout = q.Gauge(L, TH).load(u), q.Field(L).load(v), q.Field(L)
    for op, o in ((q.OP_D, "D"), (q.OP_DDAG, "Ddag"), (q.OP_Q, "Q")):
        q.dslash(fout, fin, g, 0.15, 0.07, op, q.ARITH_DF64)
        assert site_rel_err(fout.store(), orc.dslash(v, u, L, TH, kappa=0.15, tm=0.07, op=o)) <= 1e-13, o
    for f in (g, fin, fout):
        f.close()


@pytest.mark.parametrize("L", [(4, 4, 4, 4), (10, 11, 9, 12)])
@pytest.mark.parametrize("kind", ["point", "half", "tiny", "mixed"])
def test_operator_on_values_outside_the_short_split(gpu, orc, L, kind):
    u, v = orc.gauge_synthetic(L, 83, EPS_PLAQ_060), orc.gaussian_spinor(L, 84)
    if kind == "point":
        v[:] = 0.0
        v[5, 1, 2, 0] = 1.0
    elif kind == "half":
        v[np.random.RandomState(85).rand(*v.shape) < 0.5] = 0.0
    elif kind == "tiny":
        v *= 1e-28
    else:  # sites of very different sizes
        v *= (10.0 ** (np.arange(v.shape[0]) % 50 - 30)).reshape(-1, 1, 1, 1)
    g, fin, fout = q.Gauge(L, TH).load(u), q.Field(L).load(v), q.Field(L)
    q.dslash(fout, fin, g, 0.15, 0.07, q.OP_D, q.ARITH_DF64)
    out, ref = fout.store(), orc.dslash(v, u, L, TH, kappa=0.15, tm=0.07, op="D")
    n = np.linalg.norm(ref.reshape(len(ref), -1), axis=1)
    err = np.linalg.norm((out - ref).reshape(len(ref), -1), axis=1)
    assert np.all(err <= 1e-13 * n)
    for f in (g, fin, fout):
        f.close()


@pytest.mark.parametrize("prec", [q.F64, q.F16])
def test_even_odd_solve_above_the_line(gpu, orc, prec):
    L = (16, 10, 12, 12)  # 11,520 sites per parity
    u, v = orc.gauge_synthetic(L, 86, EPS_PLAQ_060), orc.gaussian_spinor(L, 87)
    g, b, x = q.Gauge(L, TH).load(u), q.Field(L).load(v), q.Field(L)
    p = q.solve(x, b, g, 0.13, 0.03, solver=q.SOLVER_CGNR_EO, inner_prec=prec, tol=1e-10)
    assert p.status == 0
    assert orc.true_residual(x.store(), v, u, L, TH, 0.13, 0.03) <= 1e-10
    for f in (g, b, x):
        f.close()
