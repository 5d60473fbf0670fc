"""Calls on one stream after the other: each result is the one of the calls
apart, bit for bit (the kernels sum in a fixed order)."""
import contextlib

import numpy as np
import pytest

import qcd_gb300 as q
from tests.conftest import EPS_PLAQ_060

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
TH = (np.pi, 0.0, 0.0, 0.0)


@contextlib.contextmanager
def on_stream(s):
    q.set_stream(s.cuda_stream)
    try:
        yield
    finally:
        q.set_stream(None)


def two_streams():
    torch.cuda.synchronize()
    return torch.cuda.Stream(), torch.cuda.Stream()


def test_smeared_source_is_there_when_the_call_returns(gpu):
    L = (2, 24, 24, 24)
    g, f = q.Gauge(L, TH).synthetic(81, EPS_PLAQ_060), q.Field(L)
    args = ((1, 3, 4, 5), 2, 1, 0.5, 4, 4.0, 100)
    q.smeared_source(f, g, *args)
    ref = f.store()
    f.load(np.zeros_like(ref))
    a, b = two_streams()
    with on_stream(a):
        q.smeared_source(f, g, *args)
    with on_stream(b):
        out = f.store()
    assert np.array_equal(out, ref)
    f.close()
    g.close()


def test_gauss3d_on_two_streams(gpu):
    L = (2, 24, 24, 24)
    g = q.Gauge(L, TH).synthetic(82, EPS_PLAQ_060)
    fs, ref = [q.Field(L) for _ in range(2)], []
    for k, f in enumerate(fs):
        q.gauss3d(f.gaussian(83 + k), g, 4.0, k, 100)
        ref.append(f.store())
        f.gaussian(83 + k)
    streams = two_streams()
    for k, s in enumerate(streams):
        with on_stream(s):
            q.gauss3d(fs[k], g, 4.0, k, 100)
    torch.cuda.synchronize()
    for f, r in zip(fs, ref):
        assert np.array_equal(f.store(), r)
        f.close()
    g.close()


def test_gcr_on_two_streams(gpu, orc):
    """on resident vectors no copy to the host makes the caller wait"""
    L = (16, 12, 12, 12)
    geo = q.Geometry(L, TH)
    g = q.GaugeField(geo)
    g.a[:] = orc.gauge_synthetic(L, 85, EPS_PLAQ_060)
    lib = q.lib()
    assert lib.qcdgpu_gauge_upload(g.ref) == 0
    src, sol = [q.Vector(geo) for _ in range(2)], [q.Vector(geo) for _ in range(2)]
    for k in range(2):
        src[k].a[:] = orc.gaussian_spinor(L, 86 + k)
        for v in (src[k], sol[k]):
            assert lib.qcdgpu_vector_make_resident(v.ref) == 0

    def gcr(k):
        assert lib.gcr(sol[k].ref, src[k].ref, g.ref, 0.15, 0.02, 17, geo.s) == 0

    def result(k):
        assert lib.qcdgpu_vector_to_host(sol[k].ref) == 0
        return sol[k].a.copy()

    ref = []
    for k in range(2):
        gcr(k)
        ref.append(result(k))
    streams = two_streams()
    for k, s in enumerate(streams):
        with on_stream(s):
            gcr(k)
    torch.cuda.synchronize()
    for k in range(2):
        assert np.array_equal(result(k), ref[k])
    for o in (*src, *sol, g, geo):
        o.close()


def test_gauss3d_under_capture(gpu):
    """a recorded smearing, replayed beside a smearing on another stream"""
    L = (2, 12, 12, 12)
    g = q.Gauge(L, TH).synthetic(89, EPS_PLAQ_060)
    f, other = q.Field(L).gaussian(90), q.Field(L).gaussian(91)
    q.gauss3d(f, g, 4.0, 1, 6)
    ref = f.store()
    f.gaussian(90)
    a, b = two_streams()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a), on_stream(a):
        q.gauss3d(f, g, 4.0, 1, 6)
    for _ in range(2):
        f.gaussian(90)
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            graph.replay()
        with on_stream(b):
            q.gauss3d(other, g, 4.0, 1, 20)
        torch.cuda.synchronize()
        assert np.array_equal(f.store(), ref)
    del graph
    for o in (f, other, g):
        o.close()
