"""Workloads of the library's entry points: the calls a user's program makes,
from the smallest to the largest, through the C ABI (device arrays), the
Python front end (host arrays), a plan (one geometry, many strengths) and a
batch of small problems.

A case is a dict:
  via      "call" (guru driver, device arrays), "host" (Python front end),
           "plan" (resident geometry, one evaluation) or "batch"
  kernel   "l" (lfmm2d), "c" (cfmm2d), "r" (rfmm2d) or "h" (hfmm2d)
  ns, nt   sources and targets (batch: of every problem together)
  nd       densities
  eps      requested accuracy (the default precision runs mixed from 0.5e-6)
  charge, dipole   which strengths
  pg, pgt  outputs at sources / targets (0 none, 1 potential, 2 + gradient,
           3 + Hessian)
  dist     "uniform", "blobs" or "starfish"
  zk, zki  wavenumber (Helmholtz)
  problems number of problems (batch)
"""
import ctypes
import math

import numpy as np
import torch

import fmm2d_c_translation_b200 as fmm

P = ctypes.c_void_p
KID = {"l": 0, "c": 1}


def _case(name, via, kernel, ns, nt, eps, charge, dipole, pg, pgt, dist, nd=1, zk=0.0, zki=0.0,
          problems=1):
    c = dict(via=via, kernel=kernel, ns=ns, nt=nt, nd=nd, eps=eps, charge=charge, dipole=dipole,
             pg=pg, pgt=pgt, dist=dist, zk=zk, zki=zki, problems=problems)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: latency of one evaluation of a few hundred
        # points, the size of the package's own tests
        _case("laplace_300", "call", "l", 200, 100, 1e-6, True, True, 2, 2, "uniform"),
        # particle potentials and forces at 10^5 points, the plain configuration
        _case("laplace_1e5", "call", "l", 100000, 0, 1e-6, True, False, 2, 0, "uniform"),
        # the headline size: every strength kind, potential and gradient everywhere
        _case("laplace_2e7", "call", "l", 10000000, 10000000, 1e-6, True, True, 2, 2, "uniform"),
        # double-layer potential of a boundary curve, evaluated off it (deep adaptive tree)
        _case("laplace_starfish_8e6", "call", "l", 4000000, 4000000, 1e-9, False, True, 1, 1,
              "starfish"),
        # the all-FP64 form at close to full accuracy, ragged sizes
        _case("laplace_fp64_3e6", "call", "l", 1500007, 1499989, 1e-12, True, True, 2, 2,
              "uniform"),
        # complex-analytic sums with second derivatives on clustered points
        _case("cauchy_hess_4e5", "call", "c", 300007, 123457, 1e-9, True, True, 3, 3, "blobs"),
        # several real densities at once from host arrays, as a numpy program calls it
        _case("real_host_nd3", "host", "r", 50021, 0, 1e-6, True, True, 2, 0, "blobs", nd=3),
        # scattering at 32 wavelengths across the box, the Helmholtz configuration
        _case("helmholtz_2e6", "call", "h", 2000000, 0, 1e-6, True, True, 1, 0, "uniform",
              zk=200.0),
        # a small Helmholtz solve with every output, the size of the package's own tests
        _case("helmholtz_2e3", "call", "h", 1000, 1001, 0.51e-8, True, True, 3, 3, "uniform",
              zk=10.0),
        # a clustered Helmholtz problem in all FP64
        _case("helmholtz_blobs_1e5", "call", "h", 70001, 30011, 1e-9, True, False, 2, 2, "blobs",
              zk=30.0),
        # one matrix-vector product of an iterative boundary-integral solver
        _case("plan_starfish_2e5", "plan", "l", 200003, 0, 1e-9, False, True, 1, 0, "starfish"),
        # a stream's small requests evaluated together
        _case("batch_64", "batch", "l", 250000, 0, 1e-6, True, False, 1, 0, "uniform",
              problems=64),
    ]


def draw(rng):
    def between(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    u = rng.random()
    dist = rng.choice(["uniform", "uniform", "blobs", "starfish"])
    if u < 0.12:
        k = rng.randint(8, 100)
        return _case(None, "batch", "l", between(1000 * k, 5000 * k), 0, rng.choice([1e-3, 1e-6]),
                     True, False, rng.choice([1, 2]), 0, "uniform", problems=k)
    if u < 0.24:
        return _case(None, "plan", rng.choice("lc"), between(2000, 1000000), 0,
                     rng.choice([1e-6, 1e-9, 1e-12]), False, True, rng.choice([1, 2]), 0,
                     dist)
    charge, dipole = rng.choice([(True, False), (False, True), (True, True)])
    pg, pgt = rng.choice([(1, 0), (2, 0), (0, 1), (1, 1), (2, 2), (3, 3)])
    eps = rng.choice([1e-3, 1e-6, 1e-6, 1e-9, 1e-12])
    if u < 0.34:
        n = between(500, 200000)
        return _case(None, "host", rng.choice("lr"), n, n // 3 if pgt else 0, eps, charge, dipole,
                     pg, pgt, dist, nd=rng.choice([1, 2, 3]))
    if u < 0.62:
        n = between(300, 300000 if eps < 1e-8 else 800000)
        zk = math.exp(rng.uniform(0.0, math.log(200.0)))
        return _case(None, "call", "h", n, between(100, n) if pgt else 0, eps, charge, dipole, pg,
                     pgt, dist, zk=zk, zki=rng.choice([0.0, 0.0, 0.1]))
    n = between(100, 1000000 if eps < 5e-7 else 4000000)
    return _case(None, "call", rng.choice("llc"), n, between(100, n) if pgt else 0, eps, charge,
                 dipole, pg, pgt, dist)


# ---- inputs ---------------------------------------------------------------
def _starfish(t):
    """Points and outward unit normals of r = 1 + 0.3 cos(5 t)."""
    r, dr = 1 + 0.3 * torch.cos(5 * t), -1.5 * torch.sin(5 * t)
    c, s = torch.cos(t), torch.sin(t)
    tx, ty = dr * c - r * s, dr * s + r * c
    n = torch.sqrt(tx * tx + ty * ty)
    return torch.stack([r * c, r * s], 1), torch.stack([ty / n, -tx / n], 1)


def _inputs(case, seed):
    """src (ns, 2), trg (nt, 2), q / d (ns, nd), v (ns, 2, nd), on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev = dict(device="cuda", dtype=torch.float64)
    ns, nt, nd, dist = case["ns"], case["nt"], case["nd"], case["dist"]
    real = case["kernel"] == "r"

    def rand(*shape):
        return torch.rand(*shape, generator=g, **dev)

    def normal(*shape):
        return torch.randn(*shape, generator=g, **dev)

    normals = None
    if dist == "starfish":
        t = (torch.arange(ns, **dev) + rand(1)) * (2 * math.pi / ns)
        src, normals = _starfish(t)
        x, nrm = _starfish(rand(nt) * 2 * math.pi)
        off = 10.0 ** (-3 + 2 * rand(nt)) * torch.where(rand(nt) < 0.5, -1.0, 1.0)
        trg = x + off[:, None] * nrm
    elif dist == "blobs":
        cen = rand(8, 2)

        def blob(n):
            k = torch.randint(0, 8, (n,), generator=g, device="cuda")
            return cen[k] + 0.01 * normal(n, 2)

        src, trg = blob(ns), blob(nt)
    else:
        src, trg = rand(ns, 2), rand(nt, 2)

    def strength():
        a = normal(ns, nd)
        return a if real else torch.complex(a, normal(ns, nd))

    q = strength() if case["charge"] else None
    d = v = None
    if case["dipole"]:
        d = strength()
        if normals is not None:
            if not real:
                d = torch.complex(d.real.contiguous(), torch.zeros_like(d.real))
            v = normals[:, :, None].expand(ns, 2, nd).contiguous()
        else:
            a = rand(ns, nd) * 2 * math.pi
            v = torch.stack([torch.cos(a), torch.sin(a)], 1).contiguous()
    return dict(src=src.contiguous(), trg=trg.contiguous(), q=q, d=d, v=v)


def _comps(kernel):
    return (1, 1, 1) if kernel == "c" else (1, 2, 3)


def _outputs(case):
    dt = torch.float64 if case["kernel"] == "r" else torch.complex128
    return [[torch.empty(n, c, case["nd"], dtype=dt, device="cuda") if flag > k else None
             for k, c in enumerate(_comps(case["kernel"]))]
            for n, flag in ((case["ns"], case["pg"]), (case["nt"], case["pgt"]))]


def _ptr(t):
    return P(t.data_ptr() if t is not None and t.numel() else 0)


def _offsets(case, seed):
    """Where each problem of a batch begins: uneven sizes, every one at least 1."""
    r = np.random.default_rng(seed)
    w = r.uniform(0.2, 1.8, case["problems"])
    n = np.maximum(1, (w / w.sum() * case["ns"]).astype(np.int64))
    n[-1] += case["ns"] - n.sum()
    return np.concatenate([[0], np.cumsum(n)])


class _Plan:
    """A plan handle, destroyed with the object."""

    def __init__(self, case, x):
        L = self.L = fmm.lib()
        L.fmm2d_b200_plan_create.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_double,
                                             ctypes.c_int, P] + [ctypes.c_int] * 4 + \
            [P, ctypes.c_int, ctypes.POINTER(P)]
        L.fmm2d_b200_plan_eval.argtypes = [P] * 10
        L.fmm2d_b200_plan_destroy.argtypes = [P]
        self.h = P()
        torch.cuda.current_stream().synchronize()
        if L.fmm2d_b200_plan_create(KID[case["kernel"]], case["nd"], case["eps"], case["ns"],
                                    _ptr(x["src"]), int(case["charge"]), int(case["dipole"]),
                                    case["pg"], case["nt"], _ptr(x["trg"]), case["pgt"],
                                    ctypes.byref(self.h)):
            raise RuntimeError(fmm.last_error())

    def __del__(self):
        if self.h:
            self.L.fmm2d_b200_plan_destroy(self.h)


def prepare(case, seed):
    x = _inputs(case, seed)
    st = dict(case=case, x=x)
    if case["via"] == "host":
        def host(t, perm):
            return None if t is None else np.asfortranarray(t.cpu().numpy().transpose(perm))
        kw = dict(eps=case["eps"], sources=host(x["src"], (1, 0)), charges=host(x["q"], (1, 0)),
                  dipstr=host(x["d"], (1, 0)), dipvec=host(x["v"], (2, 1, 0)), pg=case["pg"],
                  nd=case["nd"])
        if case["nt"]:
            kw.update(targets=host(x["trg"], (1, 0)), pgt=case["pgt"])
        if case["kernel"] == "h":
            kw["zk"] = complex(case["zk"], case["zki"])
        st["kw"] = kw
        return st
    st["out"] = _outputs(case)
    (pot, grad, hess), (pt, gt, ht) = st["out"]
    outs = [_ptr(t) for t in (pot, grad, hess, pt, gt, ht)]
    if case["via"] == "plan":
        st["plan"] = _Plan(case, x)
        st["args"] = [_ptr(x["q"]), _ptr(x["d"]), _ptr(x["v"])] + outs
        return st
    if case["via"] == "batch":
        off = _offsets(case, seed)
        n = case["problems"]

        def plist(t, width):
            if t is None:
                return None
            return (P * n)(*[t.data_ptr() + int(o) * width for o in off[:-1]])
        ns = (ctypes.c_int * n)(*[int(k) for k in np.diff(off)])
        fmm.lib().fmm2d_b200_fmm2d_batch.argtypes = [ctypes.c_int, ctypes.c_int,
                                                     ctypes.c_double] + [P] * 5 + \
            [ctypes.c_int] + [P] * 5 + [ctypes.c_int] + [P] * 3
        st["args"] = [KID[case["kernel"]], n, case["eps"], ns, plist(x["src"], 16),
                      plist(x["q"], 16), plist(x["d"], 16), plist(x["v"], 16), case["pg"],
                      plist(pot, 16), plist(grad, 32), plist(hess, 48), None, None, 0, None, None,
                      None]
        return st
    I, D = ctypes.c_int, ctypes.c_double
    st["ier"] = I(0)
    keep = [I(case["nd"]), D(case["eps"]), (D * 2)(case["zk"], case["zki"]), I(case["ns"]),
            I(int(case["charge"])), I(int(case["dipole"])), I(0), I(case["pg"]), I(case["nt"]),
            I(case["pgt"])]
    nd, eps, zk, ns, ifc, ifd, iper, pg, nt, pgt = [ctypes.byref(k) for k in keep]
    st["keep"] = keep
    st["args"] = [nd, eps] + ([zk] if case["kernel"] == "h" else []) + \
        [ns, _ptr(x["src"]), ifc, _ptr(x["q"]), ifd, _ptr(x["d"])] + \
        ([_ptr(x["v"])] if case["kernel"] != "c" else []) + \
        [iper, pg] + outs[:3] + [nt, _ptr(x["trg"]), pgt] + outs[3:] + [ctypes.byref(st["ier"])]
    return st


def run(st):
    case = st["case"]
    if case["via"] == "host":
        o = {"l": fmm.lfmm2d, "c": fmm.cfmm2d, "r": fmm.rfmm2d, "h": fmm.hfmm2d}[
            case["kernel"]](**st["kw"])
        return [[o.pot, o.grad, o.hess], [o.pottarg, o.gradtarg, o.hesstarg]]
    L = fmm.lib()
    if case["via"] == "plan":
        ier = L.fmm2d_b200_plan_eval(st["plan"].h, *st["args"])
    elif case["via"] == "batch":
        ier = L.fmm2d_b200_fmm2d_batch(*st["args"])
    else:
        getattr(L, case["kernel"] + "fmm2d_")(*st["args"])
        ier = st["ier"].value
    if ier:
        raise RuntimeError(fmm.last_error())
    return st["out"]


# ---- what a pass cannot do without ---------------------------------------
def work(case):
    """Bytes: every input once, every output once.  Operations: those of an
    adaptive FMM on uniform points with the reference's order and leaf
    capacity: 9 leaves of near field per point and 27 translations per box."""
    ns, nt, nd, eps = case["ns"], case["nt"], case["nd"], case["eps"]
    real = case["kernel"] == "r"
    w = 8 if real else 16
    b = 16 * (ns + nt)
    b += w * nd * ns * (int(case["charge"]) + int(case["dipole"]))
    if case["dipole"] and case["kernel"] != "c":
        b += 16 * nd * ns
    cum = np.cumsum(_comps(case["kernel"]))
    vals = (ns * int(cum[case["pg"] - 1]) if case["pg"] else 0) + \
        (nt * int(cum[case["pgt"] - 1]) if case["pgt"] and nt else 0)
    b += w * nd * vals
    cap = 15 if eps >= 0.5e-6 else 20 if eps >= 0.5e-9 else 25
    ndc = nd * (2 if case["kernel"] == "l" else 1)
    p = next(j for j in range(2, 200) if (math.sqrt(0.5) ** j) / 1.5 ** (j + 1) < eps)
    pts = (ns if case["pg"] else 0) + (nt if case["pgt"] else 0)
    per = case["problems"] * cap
    near = pts * min(ns / case["problems"], 9 * cap * 0.6)
    per_pair = 10 + ndc * (int(case["charge"]) + int(case["dipole"])) * \
        (2, 10, 18)[max(case["pg"], case["pgt"]) - 1]
    boxes = max(0.0, 4 / 3 * ns / (0.6 * cap) - 2 * case["problems"]) if ns > per else 0.0
    terms = (2 * p + 1) if case["kernel"] == "h" else (p + 1)
    flops = near * per_pair * (4 if case["kernel"] == "h" else 1) + \
        27 * boxes * 8 * terms * terms * ndc + (ns + pts) * 8 * terms * ndc
    return {"bytes": float(b), "flops": float(flops)}


# ---- the sums themselves, in 64 bits -------------------------------------
def _laplace_sums(xt, xs, q, D, need):
    """sum q log z + D / z and its derivatives at xt: q (ns, k), D (ns, k)
    complex; the logarithm's real part only.  Coincident points are left out."""
    k = (q if q is not None else D).shape[1]
    out = [torch.zeros(xt.shape[0], k, dtype=torch.complex128, device="cuda") for _ in range(need)]
    step = max(1, 20_000_000 // xs.shape[0])
    zs = torch.view_as_complex(xs)
    for a in range(0, xt.shape[0], step):
        z = torch.view_as_complex(xt[a:a + step])[:, None] - zs[None, :]
        hit = z == 0
        w = 1.0 / torch.where(hit, 1.0, z)
        w[hit] = 0
        if q is not None:
            lg = torch.log(z.abs())
            lg[hit] = 0
            out[0][a:a + step] += torch.complex(lg @ q.real, lg @ q.imag)
        if D is not None:
            out[0][a:a + step] += w @ D
        if need > 1:
            w2 = w * w
            if q is not None:
                out[1][a:a + step] += w @ q
            if D is not None:
                out[1][a:a + step] -= w2 @ D
            if need > 2:
                if q is not None:
                    out[2][a:a + step] -= w2 @ q
                if D is not None:
                    out[2][a:a + step] += 2 * ((w2 * w) @ D)
    return out


def _complex_laplace(xt, xs, q, d, v, need):
    """lfmm2d's outputs (n, comps, nd): the real and imaginary parts of the
    strengths are two real-charge sums."""
    ns, nd = (q if q is not None else d).shape
    parts = []
    for part in ("real", "imag"):
        qq = None if q is None else getattr(q, part).to(torch.complex128)
        D = None
        if d is not None:
            D = torch.complex(-getattr(d, part) * v[:, 0], -getattr(d, part) * v[:, 1])
        f = _laplace_sums(xt, xs, qq, D, need)
        o = [f[0].real[:, None]]
        if need > 1:
            o.append(torch.stack([f[1].real, -f[1].imag], 1))
        if need > 2:
            o.append(torch.stack([f[2].real, -f[2].imag, -f[2].real], 1))
        parts.append(o)
    return [torch.complex(a.contiguous(), b.contiguous()) for a, b in zip(*parts)]


def _bessel01(x):
    """J0, Y0, J1, Y1 at real x > 0: ascending series below 4 (Abramowitz &
    Stegun 9.1.10, 9.1.11), Miller's recurrence with Neumann series below 25
    (9.1.46, 9.1.88), Hankel's asymptotic expansions beyond (9.2.5-9.2.10)."""
    gamma, pi = 0.57721566490153286, math.pi
    u = x.clamp(max=4.0)
    z, lg = u * u / 4, torch.log(u / 2) + gamma
    t0, t1, harm = torch.ones_like(z), u / 2, 0.0
    a0, a1, b0, b1 = t0.clone(), t1.clone(), torch.zeros_like(z), t1.clone()
    for k in range(1, 26):
        t0, t1, harm = -t0 * z / (k * k), -t1 * z / (k * (k + 1)), harm + 1.0 / k
        a0 += t0
        a1 += t1
        b0 -= harm * t0
        b1 += (2 * harm + 1.0 / (k + 1)) * t1
    low = (a0, 2 / pi * (lg * a0 + b0), a1, 2 / pi * (lg * a1 - 1 / u) - b1 / pi)
    u = x.clamp(4.0, 25.0)
    up, cur = torch.zeros_like(u), torch.full_like(u, 1e-120)
    norm, s0, s1 = torch.zeros_like(u), torch.zeros_like(u), torch.zeros_like(u)
    for n in range(80, 0, -1):  # cur = J_n up to a common factor
        k = n // 2
        if n % 2 == 0:
            norm += 2 * cur
            s0 += (-1) ** k / k * cur
        elif k:
            s1 += (-1) ** k * (2 * k + 1) / (k * (k + 1)) * cur
        j1, up, cur = cur, cur, 2 * n / u * cur - up
    norm += cur
    j0, j1, lg = cur / norm, j1 / norm, torch.log(u / 2) + gamma
    mid = (j0, 2 / pi * (lg * j0 - 2 * s0 / norm), j1,
           2 / pi * (-j0 / u + (lg - 1) * j1 - s1 / norm))
    u = x.clamp(min=25.0)
    high = []
    for nu in (0, 1):
        ps, qs, t = torch.ones_like(u), torch.zeros_like(u), torch.ones_like(u)
        for k in range(1, 24):
            t = t * (4 * nu * nu - (2 * k - 1) ** 2) / (8 * k * u)
            if k % 2:
                qs += (-1) ** (k // 2) * t
            else:
                ps += (-1) ** (k // 2) * t
        c, s, m = torch.cos(u), torch.sin(u), 1 / torch.sqrt(pi * u)
        # cos and sin of u - nu pi / 2 - pi / 4, without rounding u's difference
        c, s = (c + s, s - c) if nu == 0 else (s - c, -c - s)
        high += [m * (ps * c - qs * s), m * (ps * s + qs * c)]
    return [torch.where(x < 4, a, torch.where(x < 25, b, c)) for a, b, c in zip(low, mid, high)]


def _helmholtz_sums(xt, xs, zk, q, d, v, need):
    """(i/4) sum [c H0(kr) + k d (v . (x - y)) / r H1(kr)] and its
    derivatives, real k, one density."""
    out = [torch.zeros(xt.shape[0], c, dtype=torch.complex128, device="cuda") for c in (1, 2, 3)]
    step = max(1, 5_000_000 // xs.shape[0])
    for a in range(0, xt.shape[0], step):
        dx = xt[a:a + step, None, :] - xs[None]
        dx, dy = dx[..., 0], dx[..., 1]
        r = torch.sqrt(dx * dx + dy * dy)
        hit = r == 0
        r[hit] = 1.0
        j0, y0, j1, y1 = _bessel01(zk * r)
        h0, h1 = torch.complex(j0, y0), torch.complex(j1, y1)
        h0[hit] = 0
        h1[hit] = 0
        # radial functions: f = H0(kr), f1 = f'/r, f2 = (f1)'/r, f3 = (f2)'/r
        f1 = -zk * h1 / r
        f2 = -(zk * zk * h0 + 2 * f1) / (r * r)
        f3 = -(zk * zk * f1 + 4 * f2) / (r * r)
        o = slice(a, a + step)
        if q is not None:
            out[0][o, 0] += h0 @ q[:, 0]
            if need > 1:
                out[1][o, 0] += (f1 * dx) @ q[:, 0]
                out[1][o, 1] += (f1 * dy) @ q[:, 0]
            if need > 2:
                out[2][o, 0] += (f1 + f2 * dx * dx) @ q[:, 0]
                out[2][o, 1] += (f2 * dx * dy) @ q[:, 0]
                out[2][o, 2] += (f1 + f2 * dy * dy) @ q[:, 0]
        if d is not None:
            # k H1 (v.x) / r = -f1 (v.x)
            vx, vy = v[:, 0, 0], v[:, 1, 0]
            s = vx * dx + vy * dy
            out[0][o, 0] -= (f1 * s) @ d[:, 0]
            if need > 1:
                out[1][o, 0] -= (f2 * dx * s + f1 * vx) @ d[:, 0]
                out[1][o, 1] -= (f2 * dy * s + f1 * vy) @ d[:, 0]
            if need > 2:
                out[2][o, 0] -= (f3 * dx * dx * s + f2 * (s + 2 * dx * vx)) @ d[:, 0]
                out[2][o, 1] -= (f3 * dx * dy * s + f2 * (dx * vy + dy * vx)) @ d[:, 0]
                out[2][o, 2] -= (f3 * dy * dy * s + f2 * (s + 2 * dy * vy)) @ d[:, 0]
    return [0.25j * t[:, :, None] for t in out[:need]]


def exact(case, seed):
    ns, nd, kernel = case["ns"], case["nd"], case["kernel"]
    pts = (ns if case["pg"] else 0) + (case["nt"] if case["pgt"] else 0)
    pairs = float(ns) * pts / case["problems"] * nd
    if pairs > (8e8 if kernel == "h" else 1.2e10) or case["zki"] != 0.0 or \
            (kernel == "h" and nd > 1):
        return None
    x = _inputs(case, seed)

    def at(xt, xs, q, d, v, need):
        if kernel == "h":
            return _helmholtz_sums(xt, xs, case["zk"], q, d, v, need)
        if kernel == "c":
            f = [t[:, None] for t in _laplace_sums(xt, xs, q, d, need)]
            # (the far field's q log z carries branch terms that depend on the tree)
            return [None if q is not None else f[0]] + f[1:]
        if kernel == "r":
            f = _complex_laplace(xt, xs, None if q is None else q + 0j,
                                 None if d is None else d + 0j, v, need)
            return [t.real.contiguous() for t in f]
        return _complex_laplace(xt, xs, q, d, v, need)

    sides = []
    for xt, need in ((x["src"], case["pg"]), (x["trg"], case["pgt"])):
        if not need or not xt.shape[0]:
            sides.append([None, None, None])
            continue
        if case["via"] == "batch":
            off = _offsets(case, seed)
            got = [at(xt[a:b], x["src"][a:b], None if x["q"] is None else x["q"][a:b],
                      None if x["d"] is None else x["d"][a:b],
                      None if x["v"] is None else x["v"][a:b], need)
                   for a, b in zip(off[:-1].tolist(), off[1:].tolist())]
            got = [torch.cat(t) for t in zip(*got)]
        else:
            got = at(xt, x["src"], x["q"], x["d"], x["v"], need)
        if case["via"] == "host":  # the front end's shapes: (nd, [comps,] n), nd = 1 squeezed
            got = [t.permute(2, 1, 0) for t in got]
            got = [t[:, 0] if k == 0 else t for k, t in enumerate(got)]
            got = [np.asfortranarray((t[0] if nd == 1 else t).cpu().numpy()) for t in got]
        sides.append(got + [None] * (3 - len(got)))
    return sides
