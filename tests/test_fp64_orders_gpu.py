"""The FP64 passes over the expansion orders: P2M and P2L take the orders in
chunks of 8 up to 32 and by lanes above, M2M and L2L of small levels go by
their matrices, the M2L by folded offsets for orders 16 to 39 -- against the
direct sum, and the M2L against its one-pair-at-a-time form."""
import ctypes

import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu

# orders 7 to 53 (orders below, at and above 16, 24, 32, 39 and 40)
EPS = [1e-2, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12, 1e-13, 1e-14, 1e-15]
# a call's relative error is below its eps for the potential; a derivative
# loses about the order (<= 40) against it; rounding adds 100 sums of 1e-16
FACTOR = {1: 2.0, 2: 40.0, 3: 1600.0}
ROUND = {1: 1e-13, 2: 1e-12, 3: 1e-11}


@pytest.fixture(scope="module")
def glib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(1)
    yield L
    L.fmm2d_b200_set_precision(0)


def _inputs(family, n, nd, points):
    rng = np.random.default_rng(n)
    src = ps.uniform(n, 1) if points == "uniform" else ps.blobs(n, 2)

    def strength():
        a = rng.standard_normal((nd, n))
        return a if family == "r" else a + 1j * rng.standard_normal((nd, n))

    return src, strength(), strength(), rng.standard_normal((nd, 2, n))


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("family,n,points", [("l", 3000, "blobs"), ("l", 70001, "blobs"),
                                             ("c", 5000, "uniform")])
def test_orders_match_direct_sum(glib, eps, family, n, points):
    src, q, d, v = _inputs(family, n, 1, points)
    got, ier = W.call(glib, family, "s_cd_h", eps, src, q[0], d[0], v[0])
    assert ier == 0
    m = 50
    gc, hc = (1, 1) if family == "c" else (2, 3)
    want = [np.zeros(m * k, np.complex128) for k in (1, gc, hc)]
    s, t = np.asfortranarray(src), np.asfortranarray(src[:, :m])
    qq, dd, vv = (np.ascontiguousarray(q[0]), np.ascontiguousarray(d[0]), np.asfortranarray(v[0]))
    args = [1, n, _p(s), 1, _p(qq), 1, _p(dd)] + ([_p(vv)] if family == "l" else [])
    args += [m, _p(t), 3] + [_p(w) for w in want]
    args.append(ctypes.c_double(max(np.ptp(src, axis=1)) * 2.0 ** -51))
    f = glib.fmm2d_b200_l2d_direct if family == "l" else glib.fmm2d_b200_c2d_direct
    assert f(*args) == 0
    for pgh, (name, w, k) in enumerate((("pot", want[0], 1), ("grad", want[1], gc),
                                        ("hess", want[2], hc)), 1):
        g, w = got[name][:m], w.reshape(m, k) if k > 1 else w
        if family == "c" and name == "pot":
            continue  # (complex charges: the far field has log z, the direct sum log |z|)
        assert W.rel_err(g, w) < FACTOR[pgh] * eps + ROUND[pgh], name


# sums of 27 x order terms in another order: at most 1000 roundings of 1.1e-16
# of terms no larger than the potential's, whose derivatives lose the order
@pytest.mark.parametrize("eps", EPS[4:])
@pytest.mark.parametrize("family,nd", [("l", 1), ("r", 3), ("c", 2)])
def test_m2l_forms_agree(glib, monkeypatch, eps, family, nd):
    src, q, d, v = _inputs(family, 9001, nd, "uniform")
    outs = []
    for form in (None, "simple"):
        if form is None:
            monkeypatch.delenv("FMM2D_B200_M2L", raising=False)
        else:
            monkeypatch.setenv("FMM2D_B200_M2L", form)
        got, ier = W.call_nd(glib, family, "s_cd_g", eps, src, nd, True, q, d, v)
        assert ier == 0
        outs.append(got)
    for name in outs[0]:
        assert W.rel_err(outs[0][name], outs[1][name]) < 1e-11, name
