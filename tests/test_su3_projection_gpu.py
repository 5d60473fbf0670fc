"""The SU(3) projection of an APE step against a wider arithmetic: links of a
given condition number (an APE step with alpha = 0 projects each link alone).
Newton's iteration for the polar factor, in 64 bits, is off by 3.1e-16 to
4.4e-16 in the root mean square of a link's Frobenius norm at these condition
numbers and by 1.7e-15 at the worst of 20,000 links (restated on a CPU against
113 bits); the bounds are twice that."""
import numpy as np
import pytest

import qcd_gb300 as q

pytestmark = pytest.mark.gpu


def polar_su3(m):
    """m [n][3][3] complex: unitary polar factor times exp(-i arg(det) / 3), in long doubles"""
    w = m.astype(np.clongdouble)

    def cof(a):
        c = np.empty_like(a)
        for i in range(3):
            for j in range(3):
                i1, i2, j1, j2 = (i + 1) % 3, (i + 2) % 3, (j + 1) % 3, (j + 2) % 3
                c[:, i, j] = a[:, i1, j1] * a[:, i2, j2] - a[:, i1, j2] * a[:, i2, j1]
        return c

    for _ in range(12):
        c = cof(w)
        det = (w[:, 0] * c[:, 0]).sum(-1)
        w = (w + (c / det[:, None, None]).conj()) / 2
    det = (w[:, 0] * cof(w)[:, 0]).sum(-1)
    return w * np.exp(-1j * np.angle(det) / 3)[:, None, None]


@pytest.mark.parametrize("kappa", [1.1, 1.5, 3.0, 8.0, 20.0])
def test_projection_error(gpu, kappa):
    L = (2, 8, 8, 8)
    V = int(np.prod(L))
    r = np.random.RandomState(91)

    def unitary(n):
        return np.linalg.qr(r.standard_normal((n, 3, 3)) + 1j * r.standard_normal((n, 3, 3)))[0]

    n = 4 * V
    s = np.stack([np.full(n, kappa), np.exp(r.uniform(0.0, np.log(kappa), n)), np.ones(n)], 1)
    m = unitary(n) * s[:, None, :] @ unitary(n)
    g, o = q.Gauge(L).load(m.reshape(V, 4, 3, 3).view(np.float64).reshape(V, 4, 3, 3, 2)), q.Gauge(L)
    q.ape3d(o, g, 0.0, 1)
    out = o.store().view(np.complex128)[..., 0][:, 1:].reshape(-1, 3, 3)
    ref = polar_su3(m.reshape(V, 4, 3, 3)[:, 1:].reshape(-1, 3, 3))
    err = np.sqrt((np.abs(out - ref) ** 2).sum((1, 2)).astype(np.float64))
    assert np.sqrt((err**2).mean()) <= 8.8e-16
    assert err.max() <= 3.4e-15
    g.close()
    o.close()
