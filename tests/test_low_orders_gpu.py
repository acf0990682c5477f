"""P2M and P2L at the lowest expansion orders (eps above 0.1: order 2; eps 0:
order 1), which have fewer powers than the lanes that build them.  All points
lie in tight clusters at the centers of their boxes, so that even these orders
give the far field to many digits, and ifnear = 0 leaves it alone: wrong
moments cannot hide behind the truncation or the near field."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DELTA = 2.5e-4  # half side of a cluster


@pytest.fixture(params=[1, 2], ids=["fp64", "mixed"])
def glib(request):
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(request.param)
    yield L, request.param == 2
    L.fmm2d_b200_set_precision(0)


def _far(lib, fam, eps, src, q, d, v, trg, ndiv):
    """Potentials at the sources without the near field (ndiv driver)."""
    P = ctypes.c_void_p
    ptr = lambda a: a.ctypes.data_as(P)
    ci = lambda x: ctypes.byref(ctypes.c_int(x))
    ns = src.shape[1]
    s, t = np.asfortranarray(src), np.asfortranarray(trg)
    q, d = np.ascontiguousarray(q, np.complex128), np.ascontiguousarray(d, np.complex128)
    v = np.asfortranarray(v)
    pot, ier, ti = np.zeros(ns, np.complex128), ctypes.c_int(-1), np.zeros(8)
    args = [ci(1), ctypes.byref(ctypes.c_double(eps)), ci(ns), ptr(s), ci(int(np.any(q))), ptr(q),
            ci(int(np.any(d))), ptr(d)] + ([ptr(v)] if fam == "l" else [])
    args += [ci(0), ci(1), ptr(pot), None, None, ci(t.shape[1]), ptr(t), ci(0), None, None, None,
             ci(ndiv), ci(0), ci(0), ptr(ti), ctypes.byref(ier)]
    getattr(lib, f"{fam}fmm2d_ndiv_")(*args)
    assert ier.value == 0
    return pot


def _direct(fam, src, q, d, v, i, j):
    """Potential at the points i of the sources j."""
    z = (src[0, i][:, None] - src[0, j]) + 1j * (src[1, i][:, None] - src[1, j])
    pot = np.log(np.abs(z)) @ q[j]
    if fam == "l":
        dv = v[0, j] * z.real + v[1, j] * z.imag
        return pot - (dv / np.abs(z) ** 2) @ d[j]
    return pot + (1.0 / z) @ d[j]


def _check(got, want, fam, ratio, order, mixed):
    # the neglected powers of (cluster size / distance), ten times over; the
    # mixed mode rounds to FP32 throughout
    tol = 10.0 * ratio ** order + 1e-12
    if mixed:
        tol = max(tol, 5e-6)
    if fam == "c":  # (the far field of a charge is q log z; the branch is free)
        got, want = got.real, want.real
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)


def _strengths(rng, n, fam, kind):
    q = 0.5 + rng.random(n) + (1j * rng.random(n) if fam == "l" else 0.0)
    d = 0.5 + rng.random(n) + 1j * rng.random(n)
    v = 0.5 + rng.random((2, n))
    return q * ("c" in kind), d * ("d" in kind), v


def _order(lib, eps):
    return lib.fmm2d_b200_laplace_nterms(ctypes.c_double(eps))


CORNERS = np.array([[0.0, 1.0], [0.0, 1.0]])
EPS = [0.5, 0.2, 0.1, 0.0]


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("m,ndiv", [(3, 5), (8, 10), (17, 20)])
@pytest.mark.parametrize("fam,kind", [("l", "c"), ("l", "d"), ("l", "cd"), ("c", "cd")])
def test_p2m(glib, fam, kind, eps, m, ndiv):
    """16 leaves of m sources, every far pair by one M2L between leaves."""
    lib, mixed = glib
    rng = np.random.default_rng(m)
    g = np.array([(x, y) for y in range(4) for x in range(4)])
    box = np.repeat(np.arange(16), m)
    src = ((g[box] + 0.5) / 4).T + DELTA * rng.uniform(-1, 1, (2, 16 * m))
    q, d, v = _strengths(rng, 16 * m, fam, kind)
    got = _far(lib, fam, eps, src, q, d, v, CORNERS, ndiv)
    want = np.zeros_like(got)
    for b in range(16):
        far = np.abs(g - g[b]).max(axis=1) >= 2
        i, j = np.flatnonzero(box == b), np.flatnonzero(far[box])
        want[i] = _direct(fam, src, q, d, v, i, j)
    # offsets of source and target, sqrt(2) DELTA each, over 1/2
    p = _order(lib, eps)
    _check(got, want, fam, 4 * np.sqrt(2) * DELTA, p if "d" in kind else p + 1, mixed)


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("m", [3, 8, 10])
@pytest.mark.parametrize("fam,kind", [("l", "c"), ("l", "d"), ("l", "cd"), ("c", "cd")])
def test_p2l(glib, fam, kind, eps, m):
    """m sources of a level-2 leaf, list 4 of two level-3 leaves."""
    lib, mixed = glib
    rng = np.random.default_rng(m)
    cen = [((x + 0.5) / 4, (y + 0.5) / 4) for y in range(4) for x in range(4) if (x, y) != (1, 1)]
    fine = [(x, y) for y in (0.3125, 0.4375) for x in (0.3125, 0.4375)]
    src = np.array([c for c in cen + fine for _ in range(8)]).T
    src = src + DELTA * rng.uniform(-1, 1, src.shape)
    lists4 = np.flatnonzero((np.abs(src[0] - 0.3125) < 0.01) & (np.abs(src[1] - 0.375) < 0.1))
    assert lists4.size == 16
    # the charged leaf (2, 1): m sources in its middle part
    keep = ~((np.abs(src[0] - 0.625) < 0.01) & (np.abs(src[1] - 0.375) < 0.01))
    lists4 = np.searchsorted(np.flatnonzero(keep), lists4)
    mid = np.array([[0.625], [0.375]]) + 0.07 * rng.uniform(-1, 1, (2, m))
    src = np.concatenate([src[:, keep], mid], axis=1)
    n = src.shape[1]
    q, d, v = _strengths(rng, n, fam, kind)
    q[:n - m] = d[:n - m] = 0.0
    got = _far(lib, fam, eps, src, q, d, v, CORNERS, 10)[lists4]
    want = _direct(fam, src, q, d, v, lists4, np.arange(n - m, n))
    # the target's offset, sqrt(2) DELTA, over the least distance, 0.24
    _check(got, want, fam, np.sqrt(2) * DELTA / 0.24, _order(lib, eps) + 1, mixed)
