"""The CG solvers add the search directions to the solution two at a time, and
what is pending when a chunk of 16 iterations ends with its reliable update:
the solution after k iterations, k at the edges of pairs and chunks, against
the same iteration in NumPy on the oracle's operator. The last step is at least
1.3 % of the solution at every k here, so a lost or doubled one shows."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)
KAPPA, MU = 0.15, 0.02
KS = (1, 2, 3, 15, 16, 17, 18)


@pytest.fixture(scope="module")
def host(orc):
    L = (3, 5, 4, 7)
    u, b = orc.gauge_synthetic(L, 71, EPS_PLAQ_060), orc.gaussian_spinor(L, 72)

    def op(v, name):
        return orc.dslash(v, u, L, TH, kappa=KAPPA, tm=MU, op=name)

    x = np.zeros_like(b)
    r = op(b, "Ddag")
    p, rr, xs = r.copy(), np.vdot(r, r).real, {}
    for k in range(1, max(KS) + 1):
        t = op(p, "D")
        a = rr / np.vdot(t, t).real
        x = x + a * p
        r = r - a * op(t, "Ddag")
        new = np.vdot(r, r).real
        p, rr = r + new / rr * p, new
        xs[k] = x
    return L, u, b, xs


# FP64 and FP32: rounding of up to 18 iterations; FP16: four roundings (2^-11)
# of the residual's share of the solution per iteration, their sum well under
# half of the smallest last step
@pytest.mark.parametrize("prec,tol", [(q.F64, 1e-10), (q.F32, 1e-4), (q.F16, 5e-3)])
def test_solution_after_k_iterations(gpu, host, prec, tol):
    L, u, b, xs = host
    g, fb, fx = q.Gauge(L, TH).load(u), q.Field(L).load(b), q.Field(L)
    for k in KS:
        fx.load(np.zeros_like(b))
        p = q.solve(fx, fb, g, KAPPA, MU, solver=q.SOLVER_CGNR, inner_prec=prec, tol=1e-30, maxiter=k)
        assert p.iters == k and p.status == 1
        assert np.linalg.norm(fx.store() - xs[k]) <= tol * np.linalg.norm(xs[k]), k
    for f in (g, fb, fx):
        f.close()


@pytest.mark.parametrize("eo", [False, True], ids=["full", "eo"])
def test_batch_after_one_chunk(gpu, orc, eo):
    """16 iterations of three slots, beside the FP64 solver's: the last step of
    the even/odd system is 0.4 % of its solution and a third of its residual"""
    L = (8, 6, 4, 8)
    u = orc.gauge_synthetic(L, 71, EPS_PLAQ_060)
    g = q.Gauge(L, TH).load(u)
    batch = q.Batch(g, 4, eo=eo)
    fb = [q.Field(L).load(orc.gaussian_spinor(L, 72 + i)) for i in range(3)]
    fx = [q.Field(L) for _ in fb]
    for i in range(3):
        assert batch.add(fx[i], fb[i], KAPPA, 0.0, q.OP_D, tol=1e-30, maxiter=16, tag=i) >= 0
    batch.step(16)
    done = {tag: (st, it, res) for tag, st, it, res in batch.poll()}
    fy = q.Field(L)
    for i in range(3):
        fy.load(np.zeros_like(fx[i].store()))
        p = q.solve(fy, fb[i], g, KAPPA, 0.0, solver=q.SOLVER_CGNR_EO if eo else q.SOLVER_CGNR, inner_prec=q.F64,
                    tol=1e-30, maxiter=16)
        assert done[i][:2] == (1, 16) and p.iters == 16
        assert abs(done[i][2] - p.true_residual) <= 0.15 * p.true_residual
        x, y = fx[i].store(), fy.store()
        assert np.linalg.norm(x - y) <= (2e-3 if eo else 5e-3) * np.linalg.norm(y)
    batch.close()
    for f in (g, fy, *fb, *fx):
        f.close()
