"""The work a program gives this library, case by case, for timing and for comparing results.

Every case is one pass through the public Python entry points. Lattices are L = (t, x, y, z) extents, t fastest in
memory; kappa, theta = (pi, 0, 0, 0) and the link ensemble (exp(i eps H), eps = 0.43374, mean plaquette about 0.60) are
those of the repository's benchmark. Inputs come from a torch generator, so that exact() can rebuild them without the
library.
"""
import math

import numpy as np
import torch

import qcd_gb300 as q

EPS = 0.43374
THETA = (math.pi, 0.0, 0.0, 0.0)
PREC = {"f64": q.F64, "f32": q.F32, "f16": q.F16}
OP = {"D": q.OP_D, "Q": q.OP_Q, "DDAG": q.OP_DDAG, "DDAGD": q.OP_DDAGD}
BYTES = {"f64": 8, "f32": 4, "f16": 2}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the operator on the smallest lattice in use (a test ensemble): launch latency
        case("apply", "apply_f64_8x16", (16, 8, 8, 8), prec="f64", op="D", mu=0.0),
        # the operator in double precision on the ordinary 24^3 x 48 lattice
        case("apply", "apply_f64_24x48", (48, 24, 24, 24), prec="f64", op="D", mu=0.0),
        # Q with a twisted mass in single precision on odd extents (solvers without even/odd splitting)
        case("apply", "apply_f32_odd", (45, 31, 29, 33), prec="f32", op="Q", mu=0.05),
        # the half-precision operator of a mixed-precision solver written by the caller, 32^3 x 64
        case("apply", "apply_f16_32x64", (64, 32, 32, 32), prec="f16", op="D", mu=0.0),
        # 16 right-hand sides per gauge-field read, then each one's result as a field of its own
        case("mrhs", "mrhs16_24x48", (48, 24, 24, 24), nrhs=16, op="D", mu=0.0),
        # the drop-in for existing C hosts: vectors in page-locked host memory, copied in and out by the call
        case("host", "host_apply_24x48", (48, 24, 24, 24), mu=0.0),
        # the production solve: one propagator column, even/odd CGNR with FP16 inner iterations
        case("solve", "solve_eo_f16_24x48", (48, 24, 24, 24), kappa=0.150, mu=0.0),
        # the twelve columns of one propagator through the batched solver
        case("batch", "batch12_eo_16x32", (32, 16, 16, 16), nrhs=12, kappa=0.150, mu=0.0),
        # the reference's own solver: one GCR cycle on host vectors
        case("gcr", "gcr32_16x32", (32, 16, 16, 16), n=32, mu=0.0),
        # source construction from the raw links: 20 APE steps, point source, 50 Gaussian steps
        case("source", "smeared_source_24x48", (48, 24, 24, 24), ape_n=20, gauss_n=50),
        # the Gaussian part alone for the twelve sources of a propagator, on links smeared before
        case("gauss", "gauss12_32x64", (64, 32, 32, 32), nsrc=12, gauss_n=50),
        # the proton correlator of two propagators, all time-slices, seven momenta
        case("twop", "proton_24x48", (48, 24, 24, 24), nmom=7),
    ]


def case(kind, name, L, **kw):
    c = {"name": name} if name else {}
    c.update(kind=kind, lt=L[0], lx=L[1], ly=L[2], lz=L[3], **kw)
    return c


def extents(rng, lo, hi, even):
    """Extents of a lattice whose volume lies between lo and hi (spread over its logarithm)."""
    while True:
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        s = (v / 2.0) ** 0.25
        L = [max(2, int(round(s * rng.uniform(0.8, 1.25) * (2 if i == 0 else 1)))) for i in range(4)]
        if even:
            L = [n + n % 2 for n in L]
        if lo <= L[0] * L[1] * L[2] * L[3] <= hi:
            return tuple(L)


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "mrhs", "host", "solve", "batch", "gcr", "source", "gauss", "twop"])
    mu = rng.choice([0.0, 0.0, 0.03])
    if kind == "apply":
        return case(kind, None, extents(rng, 2048, 2097152, False), prec=rng.choice(["f64", "f32", "f16"]),
                    op=rng.choice(["D", "Q", "DDAG"]), mu=mu)
    if kind == "mrhs":
        n = rng.choice([2, 4, 7, 8, 12, 16, 24, 32, 48])
        return case(kind, None, extents(rng, 8192, 663552 * 16 // max(n, 16), False), nrhs=n,
                    op=rng.choice(["D", "DDAG"]), mu=mu)
    if kind == "host":
        return case(kind, None, extents(rng, 8192, 663552, False), mu=mu)
    if kind == "solve":
        return case(kind, None, extents(rng, 8192, 400000, True), kappa=rng.choice([0.140, 0.145, 0.150]), mu=mu)
    if kind == "batch":
        return case(kind, None, extents(rng, 8192, 131072, True), nrhs=rng.choice([3, 8, 12]),
                    kappa=rng.choice([0.140, 0.145, 0.150]), mu=mu)
    if kind == "gcr":
        return case(kind, None, extents(rng, 4096, 131072, False), n=rng.randint(5, 32), mu=mu)
    if kind == "source":
        return case(kind, None, extents(rng, 4096, 600000, False), ape_n=rng.randint(1, 20), gauss_n=rng.randint(5, 60))
    if kind == "gauss":
        return case(kind, None, extents(rng, 4096, 1500000, False), nsrc=rng.choice([1, 4, 12]),
                    gauss_n=rng.randint(5, 60))
    return case(kind, None, extents(rng, 4096, 500000, False), nmom=rng.choice([1, 4, 7, 19]))


def lat(c):
    return (c["lt"], c["lx"], c["ly"], c["lz"])


def sites(c):
    return c["lt"] * c["lx"] * c["ly"] * c["lz"]


def work(c):
    """Each input read once and each output written once; flops of the operator by the usual count of 1320 a site."""
    V, kind = sites(c), c["kind"]
    if kind == "apply":
        b = BYTES[c["prec"]]
        links = 72 if c["prec"] == "f64" else 48
        norms = 8 if c["prec"] == "f16" else 0
        return {"bytes": V * (48 * b + links * b + norms), "flops": 1320 * V}
    if kind == "mrhs":  # the fields that come out are read and written once more
        return {"bytes": V * (c["nrhs"] * 104 + 288 + c["nrhs"] * 104), "flops": 1320 * V * c["nrhs"]}
    if kind == "host":
        return {"bytes": V * (384 + 576), "flops": 1320 * V}
    if kind == "solve":  # about 130 iterations of four half-lattice hops, update and direction in FP16 / FP32
        return {"bytes": 130 * V * (2 * 200 + 500) / 2, "flops": 130 * 2 * 1320 * V}
    if kind == "batch":
        return {"bytes": 110 * V * (c["nrhs"] * 700 + 4 * 288) / 2, "flops": 110 * 2 * 1320 * V * c["nrhs"]}
    if kind == "gcr":  # n applies; k projections read for each step's dots and again for its update
        n = c["n"]
        return {"bytes": V * (n * 960 + 192 * (n * n + 3 * n)), "flops": V * (1320 * n + 96 * n * (n - 1) + 96 * n * n // 2)}
    if kind == "source":  # per step three staple sums (16 products of 3 x 3 matrices each pair) and projections
        V3 = V // c["lt"]
        return {"bytes": V * 2 * 576 * c["ape_n"] + V * 192, "flops": V * c["ape_n"] * 3 * 8 * 216 + V3 * c["gauss_n"] * 1800}
    if kind == "gauss":
        V3 = V // c["lt"]
        return {"bytes": V3 * (384 * c["nsrc"] + 432), "flops": V3 * c["nsrc"] * c["gauss_n"] * 1800}
    return {"bytes": V * 24 * 192, "flops": V * 14000}


# ------------------------------------------------------------------ inputs
def gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + what)
    return g


def normal(shape, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def links(L, seed):
    """[V][4][3][3] complex SU(3) links exp(i eps H), H = sum_a g_a lambda_a / 2, rows re-orthonormalised."""
    V = L[0] * L[1] * L[2] * L[3]
    U = torch.empty((V, 4, 3, 3), dtype=torch.complex128, device="cuda")
    g = gen(seed, 1)
    for mu in range(4):
        a = normal((8, V), g) * (0.5 * EPS)
        H = torch.zeros((V, 3, 3), dtype=torch.complex128, device="cuda")
        s3 = 1.0 / math.sqrt(3.0)
        H[:, 0, 0] = a[2] + a[7] * s3
        H[:, 1, 1] = -a[2] + a[7] * s3
        H[:, 2, 2] = -2.0 * s3 * a[7]
        for i, j, k in ((0, 1, 0), (0, 2, 3), (1, 2, 5)):
            H[:, i, j] = torch.complex(a[k], -a[k + 1])
            H[:, j, i] = torch.complex(a[k], a[k + 1])
        M = 1j * H
        E = M + torch.eye(3, dtype=torch.complex128, device="cuda")
        P = M
        for n in range(2, 7):
            P = mm(P, M) / n
            E = E + P
        r0 = E[:, 0] / E[:, 0].abs().square().sum(-1, keepdim=True).sqrt()
        r1 = E[:, 1] - (r0.conj() * E[:, 1]).sum(-1, keepdim=True) * r0
        r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
        U[:, mu, 0], U[:, mu, 1] = r0, r1
        U[:, mu, 2] = torch.linalg.cross(r0, r1).conj()
    return U


def spinor(L, seed, what=2):
    V = L[0] * L[1] * L[2] * L[3]
    return torch.view_as_complex(normal((V, 4, 3, 2), gen(seed, what)))


def point(c, seed, k):
    """The site of the seed's point source and the source's spin and colour for column k."""
    L = lat(c)
    r = np.random.RandomState(seed % (1 << 31))
    x = tuple(int(r.randint(0, n)) for n in L)
    return x, (k % 12) // 3, k % 3


def source(c, seed, k):
    x, s, col = point(c, seed, k)
    L = lat(c)
    v = torch.zeros((sites(c), 4, 3), dtype=torch.complex128, device="cuda")
    v[x[0] + L[0] * (x[1] + L[1] * (x[2] + L[2] * x[3])), s, col] = 1.0
    return v


def momenta(n):
    all_p = sorted(((x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)),
                   key=lambda p: (sum(a * a for a in p), p))
    return all_p[:n]


def propagator(c, seed, col, what):
    """One column: Gaussian components, falling off with the time distance from the source as a propagator does."""
    L = lat(c)
    v = spinor(L, seed, what + col)
    t = torch.arange(L[0], device="cuda", dtype=torch.float64)
    x, _, _ = point(c, seed, 0)
    d = (t - x[0]) % L[0]
    fall = torch.exp(-0.25 * torch.minimum(d, L[0] - d))
    return (v.view(-1, L[0], 4, 3) * fall.view(1, -1, 1, 1)).view(v.shape)


# ------------------------------------------- the library's objects as owners
class Owner:
    """Closes a library object when the last user of it or of its memory is gone."""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.obj.close()
        except Exception:
            pass


class Memory:
    """The memory of an owner's object, as torch and numpy read it without a copy."""

    def __init__(self, owner, ptr, shape, typestr, host=False):
        self.owner = owner
        d = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 3}
        if host:
            self.__array_interface__ = d
        else:
            self.__cuda_array_interface__ = d


def device_views(owner):
    """The values of a field: complex components in its storage order; FP16 fields as halves and their site norms."""
    f = owner.obj
    V, ptr = f.V, q.lib().qcdgpu_field_data(f.h)
    stride = (V + 127) // 128 * 128

    def view(at, shape, t):
        return torch.as_tensor(Memory(owner, ptr + at, shape, t), device="cuda")

    if f.prec == q.F64:
        return [view(0, (12, stride, 2), "<f8")[:, :V]]
    if f.prec == q.F32:
        return [view(0, (6, stride, 4), "<f4")[:, :V]]
    return [view(0, (3, stride, 8), "<f2")[:, :V], view(48 * stride, (stride,), "<f4")[:V]]


def stored(v, prec):
    """[V][4][3] complex values as device_views() lays them out, in 64 bits."""
    V = v.shape[0]
    r = torch.view_as_real(v.reshape(V, 12))
    if prec == "f64":
        return [r.permute(1, 0, 2).contiguous()]
    if prec == "f32":
        return [r.reshape(V, 6, 4).permute(1, 0, 2).contiguous()]
    m = r.reshape(V, 24).abs().amax(1)
    return [(r.reshape(V, 24) / m[:, None]).reshape(V, 3, 8).permute(1, 0, 2).contiguous(), m]


def host_array(t):
    t = torch.view_as_real(t)
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def gauge(L, U, prec="f64"):
    g = Owner(q.Gauge(L, THETA, PREC[prec]))
    g.obj.load(host_array(U))
    return g


def field(L, v=None, prec="f64"):
    f = Owner(q.Field(L, PREC[prec]))
    if v is not None:
        if prec == "f64":
            device_views(f)[0].copy_(stored(v, prec)[0])
        else:
            f.obj.load(host_array(v))
    return f


def host_vector(geo, v=None):
    o = Owner(q.Vector(geo.obj))
    o.geo = geo  # the geometry outlives its vectors
    if v is not None:
        o.obj.a[:] = torch.view_as_real(v).cpu().numpy()
    return o


def host_gauge(geo, U):
    o = Owner(q.GaugeField(geo.obj))
    o.geo = geo
    o.obj.a[:] = torch.view_as_real(U).cpu().numpy()
    if q.lib().qcdgpu_gauge_upload(o.obj.ref) != 0:
        raise RuntimeError("gauge upload failed")
    return o


def prepare(c, seed):
    L, kind = lat(c), c["kind"]
    s = {"kind": kind, "case": c, "kappa": c.get("kappa", 0.150), "mu": c.get("mu", 0.0)}
    U = None if kind in ("twop",) else links(L, seed)
    if kind == "apply":
        s["g"] = gauge(L, U, c["prec"])
        s["in"], s["out"] = field(L, spinor(L, seed), c["prec"]), field(L, None, c["prec"])
        s["got"], s["op"] = device_views(s["out"]), OP[c["op"]]
    elif kind == "mrhs":
        s["g"], s["op"] = gauge(L, U), OP[c["op"]]
        s["in"], s["out"] = Owner(q.MField(L, c["nrhs"])), Owner(q.MField(L, c["nrhs"]))
        for k in range(c["nrhs"]):
            f = field(L, spinor(L, seed, 10 + k))
            s["in"].obj.set(k, f.obj)
        s["cols"] = [field(L, None, "f16") for _ in range(c["nrhs"])]
        s["got"] = [device_views(f) for f in s["cols"]]
    elif kind in ("host", "gcr"):
        geo = Owner(q.Geometry(L, THETA))
        s["g"], s["in"], s["out"] = host_gauge(geo, U), host_vector(geo, spinor(L, seed)), host_vector(geo)
        s["geo"] = geo
        s["got"] = np.asarray(Memory(s["out"], s["out"].obj.s.D, (sites(c), 4, 3, 2), "<f8", host=True))
        s["m"] = 1.0 / (2.0 * s["kappa"]) - 4.0
    elif kind == "solve":
        s["g"], s["b"], s["x"] = gauge(L, U), field(L, source(c, seed, seed % 12)), field(L)
        s["got"] = device_views(s["x"])
    elif kind == "batch":
        s["g"] = gauge(L, U)
        s["batch"] = Owner(q.Batch(s["g"].obj, c["nrhs"], eo=True))
        s["batch"].gauge = s["g"]
        s["b"] = [field(L, source(c, seed, k)) for k in range(c["nrhs"])]
        s["x"] = [field(L) for _ in range(c["nrhs"])]
        s["got"] = [device_views(f) for f in s["x"]]
    elif kind == "source":
        s["g"], s["x"] = gauge(L, U), field(L)
        s["point"], s["spin"], s["colour"] = point(c, seed, seed % 12)
        s["got"] = device_views(s["x"])
    elif kind == "gauss":
        # the raw links stand in for smeared ones: the same type, size and layout
        s["g"], s["t"] = gauge(L, U), point(c, seed, 0)[0][0]
        s["src"] = [field(L, source(c, seed, k)) for k in range(c["nsrc"])]
        s["x"] = [field(L) for _ in range(c["nsrc"])]
        s["got"] = [device_views(f) for f in s["x"]]
    else:
        s["up"] = [field(L, propagator(c, seed, k, 100)) for k in range(12)]
        s["dn"] = [field(L, propagator(c, seed, k, 200)) for k in range(12)]
        s["point"] = point(c, seed, 0)[0]
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "apply":
        q.dslash(s["out"].obj, s["in"].obj, s["g"].obj, s["kappa"], s["mu"], s["op"])
    elif kind == "mrhs":
        q.dslash_mrhs(s["out"].obj, s["in"].obj, s["g"].obj, s["kappa"], s["mu"], s["op"])
        for k, f in enumerate(s["cols"]):
            s["out"].obj.get(k, f.obj)
    elif kind == "host":
        if q.lib().qcd_applyWilsonTMOp(s["out"].obj.ref, s["in"].obj.ref, s["g"].obj.ref, s["m"], s["mu"]) != 0:
            raise RuntimeError("apply failed")
    elif kind == "gcr":
        if q.lib().gcr(s["out"].obj.ref, s["in"].obj.ref, s["g"].obj.ref, s["kappa"], s["mu"], s["case"]["n"],
                       s["geo"].obj.s) != 0:
            raise RuntimeError("gcr failed")
    elif kind == "solve":
        p = q.solve(s["x"].obj, s["b"].obj, s["g"].obj, s["kappa"], s["mu"], q.SOLVER_CGNR_EO, inner_prec=q.F16,
                    tol=1e-10)
        if p.status != 0:
            raise RuntimeError("solve: status %d" % p.status)
    elif kind == "batch":
        b = s["batch"].obj
        for k, (x, rhs) in enumerate(zip(s["x"], s["b"])):
            b.add(x.obj, rhs.obj, s["kappa"], s["mu"], tol=1e-10, tag=k)
        while b.active:
            b.step(16)
        if any(st != 0 for _, st, _, _ in b.poll()):
            raise RuntimeError("batch: a right-hand side did not converge")
    elif kind == "source":
        q.smeared_source(s["x"].obj, s["g"].obj, s["point"], s["spin"], s["colour"], 0.5, s["case"]["ape_n"], 4.0,
                         s["case"]["gauss_n"])
    elif kind == "gauss":
        for x, v in zip(s["x"], s["src"]):
            x.obj.copy_from(v.obj)
            q.gauss3d(x.obj, s["g"].obj, 4.0, s["t"], s["case"]["gauss_n"])
    else:
        return q.twop_proton([f.obj for f in s["up"]], [f.obj for f in s["dn"]], s["point"], 0,
                             s["case"]["lt"] - 1, momenta(s["case"]["nmom"]))
    return s["got"]


# ------------------------------------------- the same in 64 bits, with torch
GAMMA_COL = ((2, 3, 0, 1), (3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1))
GAMMA_VAL = ((-1, -1, -1, -1), (-1j, -1j, 1j, 1j), (-1, 1, 1, -1), (-1j, 1j, 1j, -1j))


def mm(a, b):
    """Products of 3 x 3 matrices in the last two dimensions."""
    return (a.unsqueeze(-1) * b.unsqueeze(-3)).sum(-2)


def shift(v, L, mu, n):
    """v(x + n mu) for values [V][...]."""
    w = v.view((L[3], L[2], L[1], L[0]) + v.shape[1:])
    return torch.roll(w, -n, 3 - mu).reshape(v.shape)


def colour(u, v):
    """u v on the last dimension of [..., V][4][3]."""
    return (u.unsqueeze(-3) * v.unsqueeze(-2)).sum(-1)


def phased(L, U):
    W = U.clone()
    for mu in range(4):
        W[:, mu] *= complex(math.cos(THETA[mu] / L[mu]), math.sin(THETA[mu] / L[mu]))
    return W


def gamma5(v):
    return torch.cat([v[:, :2], -v[:, 2:]], 1)


def apply64(L, W, v, mp4, tm, dag=False):
    """The operator (or its adjoint) on one spinor, links with their boundary phases in."""
    out = mp4 * v + (-1j if dag else 1j) * tm * gamma5(v)
    for mu in range(4):
        col = list(GAMMA_COL[mu])
        val = torch.tensor(GAMMA_VAL[mu], dtype=v.dtype, device=v.device).view(1, 4, 1)
        sf = 1.0 if dag else -1.0
        w = colour(W[:, mu], shift(v, L, mu, 1))
        out -= 0.5 * (w + sf * val * w[:, col])
        w = shift(colour(W[:, mu].mH, v), L, mu, -1)
        out -= 0.5 * (w - sf * val * w[:, col])
    return out


def operator64(L, W, v, mp4, tm, op):
    if op == "DDAGD":
        return apply64(L, W, apply64(L, W, v, mp4, tm), mp4, tm, True)
    w = apply64(L, W, v, mp4, tm, op == "DDAG")
    return 1j * gamma5(w) if op == "Q" else w


def dot(a, b):
    return (a.conj() * b).sum()


def solve64(L, W, b, mp4, tm):
    """D x = b to about 1e-14: CG on the normal equations in 32 bits, corrected in 64 bits."""
    W32 = W.to(torch.complex64)
    x, bn = torch.zeros_like(b), float(torch.linalg.vector_norm(b))
    for _ in range(8):
        r64 = b - apply64(L, W, x, mp4, tm)
        rn = float(torch.linalg.vector_norm(r64))
        if rn <= 3e-15 * bn:
            break
        r = apply64(L, W32, (r64 / rn).to(torch.complex64), mp4, tm, True)
        e, p = torch.zeros_like(r), r
        rr = first = float(torch.linalg.vector_norm(r)) ** 2
        for _ in range(2000):
            t = apply64(L, W32, p, mp4, tm)
            ap = apply64(L, W32, t, mp4, tm, True)
            al = rr / float(torch.linalg.vector_norm(t)) ** 2
            e, r = e + al * p, r - al * ap
            new = float(torch.linalg.vector_norm(r)) ** 2
            if new <= 1e-9 * first:
                break
            p, rr = r + (new / rr) * p, new
        x = x + rn * e.to(torch.complex128)
    return x


def gcr64(L, W, b, mp4, tm, n):
    """n steps of generalised conjugate residuals on Q = i g5 D, from zero."""
    x, r, basis = torch.zeros_like(b), b, []
    for _ in range(n):
        p, ap = r, operator64(L, W, r, mp4, tm, "Q")
        for _ in range(2):
            for u, au in basis:
                f = dot(au, ap)
                p, ap = p - f * u, ap - f * au
        nrm = torch.linalg.vector_norm(ap)
        p, ap = p / nrm, ap / nrm
        basis.append((p, ap))
        f = dot(ap, r)
        x, r = x + f * p, r - f * ap
    return x


def det3(m):
    return (m[..., 0, :] * torch.linalg.cross(m[..., 1, :], m[..., 2, :])).sum(-1)


def project64(M):
    """The unitary polar factor (Newton) with its determinant's phase taken out."""
    ph = torch.angle(det3(M)) / 3.0
    W = M
    for _ in range(12):
        r0, r1, r2 = W[..., 0, :], W[..., 1, :], W[..., 2, :]
        cof = torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0), torch.linalg.cross(r0, r1)], -2)
        W = 0.5 * (W + (cof / det3(W)[..., None, None]).conj())
    return W * torch.polar(torch.ones_like(ph), -ph)[..., None, None]


def ape64(L, U, alpha):
    out = U.clone()
    for mu in (1, 2, 3):
        S = torch.zeros_like(U[:, mu])
        for nu in (1, 2, 3):
            if nu == mu:
                continue
            A, B = U[:, nu], U[:, mu]
            S += mm(mm(A, shift(B, L, nu, 1)), shift(A, L, mu, 1).mH)
            S += shift(mm(mm(A.mH, B), shift(A, L, mu, 1)), L, nu, -1)
        out[:, mu] = project64(U[:, mu] + alpha * S)
    return out


def gauss64(L, U, v, t, alpha, n):
    """n Gaussian steps of v on time-slice t; the other slices stay."""
    L3 = (1,) + tuple(L[1:])
    u = U.view(-1, L[0], 4, 3, 3)[:, t]
    w = v.view(-1, L[0], 4, 3)[:, t].clone()
    for _ in range(n):
        h = torch.zeros_like(w)
        for nu in (1, 2, 3):
            h += colour(u[:, nu], shift(w, L3, nu, 1))
            h += shift(colour(u[:, nu].mH, w), L3, nu, -1)
        w = (w + alpha * h) / (1.0 + 6.0 * alpha)
    out = v.clone()
    out.view(-1, L[0], 4, 3)[:, t] = w
    return out


EPS3 = [(0, 1, 2, 1), (2, 0, 1, 1), (1, 2, 0, 1), (2, 1, 0, -1), (0, 2, 1, -1), (1, 0, 2, -1)]
CG5 = ((0, 1, 1), (1, 0, -1), (2, 3, 1), (3, 2, -1))
BCG5 = ((0, 1, -1), (1, 0, 1), (2, 3, -1), (3, 2, 1))
P13 = ((0, 0, .5j), (0, 2, -.5), (1, 1, .5j), (1, 3, -.5), (2, 0, -.5), (2, 2, -.5j), (3, 1, -.5), (3, 3, -.5j))


def pair(a, b):
    """sum eps eps' a[c1][d1] b[c2][d2] as a matrix [c3][d3], for [S][3][3]."""
    out = torch.zeros_like(a)
    for c1, c2, c3, s in EPS3:
        for d1, d2, d3, z in EPS3:
            out[:, c3, d3] += s * z * a[:, c1, d1] * b[:, c2, d2]
    return out


def proton64(c, seed):
    """The contraction on one time-slice after the other: corr[t][momentum]."""
    L, n, mom = lat(c), c["nmom"], momenta(c["nmom"])
    xs = point(c, seed, 0)[0]
    # [V][sink spin][source spin][sink colour][source colour]
    U, D = (torch.stack([propagator(c, seed, k, w) for k in range(12)], -1).view(-1, 4, 3, 4, 3).permute(0, 1, 3, 2, 4)
            for w in (100, 200))
    z, y, x = torch.meshgrid(*[torch.arange(L[i], device="cuda", dtype=torch.float64) for i in (3, 2, 1)], indexing="ij")
    ang = [2 * math.pi * (p[0] * (x - xs[1]) / L[1] + p[1] * (y - xs[2]) / L[2] + p[2] * (z - xs[3]) / L[3]).reshape(-1)
           for p in mom]
    ft = [torch.complex(a.cos(), -a.sin()) for a in ang]
    corr = np.zeros((L[0], n), dtype=np.complex128)
    for t in range(L[0]):
        u, d = (f.reshape((-1, L[0]) + f.shape[1:])[:, (t + xs[0]) % L[0]] for f in (U, D))
        block = torch.zeros(u.shape[0], dtype=torch.complex128, device="cuda")
        ps = sum(P * u[:, be, al] for al, be, P in P13)
        for m_, nu, s1 in CG5:
            for ku, lu, s2 in BCG5:
                dd = d[:, nu, lu]
                e = pair(u[:, m_, ku], dd)
                block -= s1 * s2 * (e * ps).sum((1, 2))
                for al in range(4):
                    w = sum(P * u[:, be, ku] for a_, be, P in P13 if a_ == al)
                    block -= s1 * s2 * (pair(u[:, m_, al], dd) * w).sum((1, 2))
        f = complex(math.cos(3 * math.pi * t / L[0]), math.sin(3 * math.pi * t / L[0]))
        for j in range(n):
            corr[t, j] = complex((0.5 * f * (block * ft[j]).sum()).item())
    return corr


def exact(c, seed):
    L, kind = lat(c), c["kind"]
    mp4, mu = 1.0 / (2.0 * c.get("kappa", 0.150)), c.get("mu", 0.0)
    if kind == "twop":
        return proton64(c, seed)
    U = links(L, seed)
    if kind == "source":
        t = point(c, seed, 0)[0][0]
        for _ in range(c["ape_n"]):
            U = ape64(L, U, 0.5)
        return stored(gauss64(L, U, source(c, seed, seed % 12), t, 4.0, c["gauss_n"]), "f64")
    if kind == "gauss":
        t = point(c, seed, 0)[0][0]
        return [stored(gauss64(L, U, source(c, seed, k), t, 4.0, c["gauss_n"]), "f64") for k in range(c["nsrc"])]
    W = phased(L, U)
    if kind == "apply":
        return stored(operator64(L, W, spinor(L, seed), mp4, mu, c["op"]), c["prec"])
    if kind == "mrhs":
        return [stored(operator64(L, W, spinor(L, seed, 10 + k), mp4, mu, c["op"]), "f16") for k in range(c["nrhs"])]
    if kind == "host":
        return torch.view_as_real(operator64(L, W, spinor(L, seed), mp4, mu, "D"))
    if kind == "gcr":
        return torch.view_as_real(gcr64(L, W, spinor(L, seed), mp4, mu, c["n"]))
    if kind == "solve":
        return stored(solve64(L, W, source(c, seed, seed % 12), mp4, mu), "f64")
    return [stored(solve64(L, W, source(c, seed, k), mp4, mu), "f64") for k in range(c["nrhs"])]
