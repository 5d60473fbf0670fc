"""Multi-RHS fields and batches where slots and sites do not fill the kernels'
pairs and warps: odd slot counts (the last pair is one slot), odd
occupied counts, site counts off 32. The operator against the oracle (4e-3 per
RHS, the FP16 bar of test_mrhs_gpu.py); FP16 fields go in and come out
unchanged; odd-capacity batches reach their tolerance."""
import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("nrhs,nact", [(1, 1), (3, 3), (7, 6), (8, 5)])
@pytest.mark.parametrize("L", [(2, 2, 2, 2), (3, 5, 2, 7)])
def test_odd_slots_and_sites(gpu, orc, L, nrhs, nact):
    u = orc.gauge_synthetic(L, 71, EPS_PLAQ_060)
    g = q.Gauge(L, TH).load(u)
    mi, mo, f = q.MField(L, nrhs), q.MField(L, nrhs), q.Field(L)
    src = [orc.gaussian_spinor(L, 700 + r) for r in range(nrhs)]
    for r in range(nrhs):
        mi.set(r, f.load(src[r]))
    q.dslash_mrhs(mo, mi, g, 0.15, 0.03, q.OP_D, nact)
    for r in range(nact):
        ref = orc.dslash(src[r], u, L, TH, kappa=0.15, tm=0.03)
        assert np.linalg.norm(mo.get(r, f).store() - ref) <= 4e-3 * np.linalg.norm(ref)
    for r in range(nact, nrhs):  # slots that were not asked for stay empty
        assert not mo.get(r, f).store().any()
    for o in (g, mi, mo, f):
        o.close()


@pytest.mark.parametrize("L", [(3, 5, 2, 7), (4, 4, 4, 4)])
def test_fp16_fields_pass_unchanged(gpu, orc, L):
    m, a, b = q.MField(L, 3), q.Field(L, q.F16), q.Field(L, q.F16)
    for r in range(3):
        m.set(r, a.load(orc.gaussian_spinor(L, 720 + r) * 10.0 ** (3 * r)))
        assert np.array_equal(m.get(r, b).store(), a.store())
    for o in (m, a, b):
        o.close()


@pytest.mark.parametrize("cap,n", [(1, 2), (3, 4)])
@pytest.mark.parametrize("eo", [False, True])
def test_odd_capacity_batches(gpu, orc, cap, n, eo):
    L = (8, 4, 4, 4)
    u = orc.gauge_synthetic(L, 73, EPS_PLAQ_060)
    g = q.Gauge(L, TH).load(u)
    batch = q.Batch(g, cap, eo=eo)
    src = [orc.gaussian_spinor(L, 730 + r) for r in range(n)]
    fb, fx = [q.Field(L).load(v) for v in src], [q.Field(L) for _ in range(n)]
    nxt = 0
    while nxt < n or batch.active:
        while nxt < n and batch.add(fx[nxt], fb[nxt], 0.14, 0.01, tol=1e-10, tag=nxt) >= 0:
            nxt += 1
        batch.step(16)
    assert sorted(t for t, st, _, _ in batch.poll() if st == 0) == list(range(n))
    for v, x in zip(src, fx):
        assert orc.true_residual(x.store(), v, u, L, TH, 0.14, 0.01) <= 1e-10
    batch.close()
    for o in fb + fx + [g]:
        o.close()


@pytest.mark.parametrize("L", [(8, 8, 8, 8), (16, 16, 16, 16)])
@pytest.mark.parametrize("N", [1, 7, 10, 16, 18])
def test_launch_shapes_agree(gpu, orc, L, N):
    """Slots per thread, warps per block and blocks over the slots follow the
    lattice and the occupied slots; a slot's result is the same bits in all."""
    u = orc.gauge_synthetic(L, 91, EPS_PLAQ_060)
    g = q.Gauge(L, TH).load(u)
    inp, out = q.MField(L, N), q.MField(L, N)
    f = q.Field(L)
    for r in range(N):
        inp.set(r, f.load(orc.gaussian_spinor(L, 910 + r)))
    want = {}
    try:
        for v in (64, 65, 128, 129, 256, 257, -1):
            q.set_mrhs_variant(v)
            for n in {1, 2, 3, N}:
                if n <= N:
                    q.dslash_mrhs(out, inp, g, 0.15, 0.02, nact=n)
                    x = out.get(n - 1, f).store()
                    assert np.array_equal(want.setdefault(n, x), x), (v, n)
    finally:
        q.set_mrhs_variant(-1)
    for o in (g, inp, out, f):
        o.close()
