"""The rounding of the proton contraction against a wider arithmetic, on
propagators of unit Gaussians. Restated on a CPU against 113 bits, the
written-out sum over the colour indices is off by 2.9e-16 in the root mean
square of the block sums (boundary phase included), the factorised one by
3.4e-16 with one chain of multiply-adds over all four ku and by 2.6e-16 with
one chain for each; the bound is the written-out sum's and 4 % for the sample."""
import numpy as np
import pytest

import qcd_gb300 as q

pytestmark = pytest.mark.gpu


def cross(a, b):
    """sum over eps(c1 c2 c3) eps(d1 d2 d3) a[c1][d1] b[c2][d2]"""
    e = np.zeros(np.broadcast(a, b).shape, a.dtype)
    for c in range(3):
        for d in range(3):
            c1, c2, d1, d2 = (c + 1) % 3, (c + 2) % 3, (d + 1) % 3, (d + 2) % 3
            e[..., c, d] = (a[..., c1, d1] * b[..., c2, d2] - a[..., c2, d1] * b[..., c1, d2]
                            - a[..., c1, d2] * b[..., c2, d1] + a[..., c2, d2] * b[..., c1, d1])
    return e


def proton(u, d, Lt, phase):
    """u, d [site][sink spin][source spin][c1][c2] with t fastest; corr [t][momentum]; phase [momentum][spatial site]"""
    block = np.zeros(u.shape[0], np.clongdouble)
    X = sum(u[:, g, g] + 1j * u[:, g, g + 2] + 1j * u[:, g + 2, g] - u[:, g + 2, g + 2] for g in range(2))
    for mu in range(4):
        for ku in range(4):
            e = cross(u[:, mu, ku], X)
            for g in range(2):
                e = e + cross(u[:, mu, g] + 1j * u[:, mu, g + 2], u[:, g, ku] + 1j * u[:, g + 2, ku])
            sign = -1 if (mu ^ ku) & 1 == 0 else 1
            block += sign * (e * d[:, mu ^ 1, ku ^ 1]).sum((-1, -2))
    t = np.arange(Lt).astype(np.longdouble)
    arg = 3 * t / Lt * np.arccos(np.longdouble(-1))
    block = -0.5j * block.reshape(-1, Lt) * (np.cos(arg) + 1j * np.sin(arg))
    return 0.5 * np.einsum("xt,px->tp", block, phase.astype(np.longdouble))


def test_twop_rounding(gpu):
    L = (64, 2, 2, 2)
    V = int(np.prod(L))
    r = np.random.RandomState(95)
    props = r.standard_normal((2, 12, V, 4, 3, 2))  # flavour, column, site, sink spin, colour
    fu, fd = [[q.Field(L).load(c) for c in p] for p in props]
    xyz = [(k & 1, k >> 1 & 1, k >> 2) for k in range(8)]
    corr = q.twop_proton(fu, fd, (0, 0, 0, 0), 0, L[0] - 1, xyz)
    c = props.view(np.complex128)[..., 0].astype(np.clongdouble).reshape(2, 4, 3, V, 4, 3)
    u, d = np.moveaxis(c, [3, 4, 1, 5, 2], [1, 2, 3, 4, 5])
    phase = np.array([[(-1.0) ** int(np.dot(p, x)) for x in xyz] for p in xyz])  # exp(-i pi p.x)
    ref = proton(u, d, L[0], phase)
    err = np.sqrt((np.abs(corr - ref) ** 2).sum() / (np.abs(ref) ** 2).sum())
    assert err <= 3.0e-16
    for f in fu + fd:
        f.close()
