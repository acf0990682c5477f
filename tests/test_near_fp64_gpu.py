"""The FP64 near field's reciprocal and logarithm (csrc/pairmath.cuh) against
the direct sum, which divides and calls log(): all points in one leaf, so the
evaluation is the near field alone.  Box sizes from 1e-6 to 1e6 move the
pairs' squared distances through every interval of the logarithm's table,
1 included."""
import ctypes

import numpy as np
import pytest

import wrappers as W

pytestmark = pytest.mark.gpu

# a pair's potential and derivatives carry at most about 15 roundings of
# 1.1e-16, and 20 pairs of either sign cancel at most about two digits:
# 2e-13; 5x room
TOL = 1e-12


@pytest.fixture(scope="module")
def glib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(1)
    yield L
    L.fmm2d_b200_set_precision(0)


def _p(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


# (squared distances outside the normal numbers, 1e-145 and 5e153, take the
# form that divides and calls log())
CASES = [(v, x) for v in ("t_c_p", "t_d_g", "t_cd_h") for x in (1e-6, 0.02, 0.7, 1.0, 3.0, 1e6)]
CASES += [("t_c_p", 1e-145), ("t_c_p", 5e153)]


@pytest.mark.parametrize("variant,scale", CASES)
@pytest.mark.parametrize("family", ["l", "c"])
def test_one_leaf_equals_direct_sum(glib, family, variant, scale):
    rng = np.random.default_rng(5)
    ns, nt = 20, 41
    src, trg = scale * rng.random((2, ns)), scale * rng.random((2, nt))
    src[:, 1] = src[:, 0] + scale * np.array([1.0, 0.0])  # a pair exactly `scale` apart
    trg[:, 0], trg[:, 1] = src[:, 2], src[:, 0]
    q = rng.standard_normal(ns) + 1j * rng.standard_normal(ns)
    d = rng.standard_normal(ns) + 1j * rng.standard_normal(ns)
    v = np.asfortranarray(rng.standard_normal((2, ns)))
    got, ier = W.call(glib, family, variant, 1e-9, src, q, d, v, trg)
    assert ier == 0
    _, cd, p = variant.split("_")
    pgh = {"p": 1, "g": 2, "h": 3}[p]
    ifc, ifd = int("c" in cd), int("d" in cd)
    gc, hc = (1, 1) if family == "c" else (2, 3)
    pot, grad, hess = (np.zeros(nt * m, np.complex128) for m in (1, gc, hc))
    s, t = np.asfortranarray(src), np.asfortranarray(trg)
    size = max(np.ptp(np.concatenate([src, trg], 1), axis=1))
    args = [1, ns, _p(s), ifc, _p(q) if ifc else None, ifd, _p(d) if ifd else None]
    if family == "l":
        args.append(_p(v) if ifd else None)
    args += [nt, _p(t), pgh, _p(pot), _p(grad), _p(hess), ctypes.c_double(size * 2.0 ** -51)]
    f = glib.fmm2d_b200_l2d_direct if family == "l" else glib.fmm2d_b200_c2d_direct
    assert f(*args) == 0
    for name, w, m in (("pottarg", pot, 1), ("gradtarg", grad, gc), ("hesstarg", hess, hc))[:pgh]:
        w = w.reshape(nt, m) if m > 1 else w
        assert W.rel_err(got[name], w) < TOL, name
