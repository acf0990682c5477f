"""The Helmholtz passes that take all levels or both point sets at once --
device-built tables, folded M2M / L2L, one M2L launch, one evaluation launch
-- against the direct sum, for trees of one to about ten levels, real and
complex wavenumbers, several densities, and point sets that want equal,
unequal or no outputs."""
import ctypes

import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu

# requested accuracy 1e-12: the expansions are cut where J_n H_n falls below
# eps of the leading terms; each of the up to ten levels and the second
# derivatives' factors of the order (about 40) add to it, so 40 x 10 x 1e-12 /
# (2 digits that the tail of a geometric series stays below its bound) < 1e-11
# for a potential, and 1e-10 with derivatives
EPS = 1e-12
TOL = {1: 1e-11, 2: 1e-10, 3: 1e-10}


@pytest.fixture(scope="module")
def glib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(1)
    yield L
    L.fmm2d_b200_set_precision(0)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _direct(lib, zk, src, q, d, v, trg, pgh, size):
    n, nd = trg.shape[1], q.shape[0]
    out = [np.zeros((n, c, nd), np.complex128) for c in (1, 2, 3)]
    zka = np.array([zk.real, zk.imag])
    s, t = np.asfortranarray(src), np.asfortranarray(trg)
    qq, dd = np.ascontiguousarray(q.T), np.ascontiguousarray(d.T)
    vv = np.ascontiguousarray(np.transpose(v, (2, 1, 0)))
    assert lib.fmm2d_b200_h2d_direct(nd, _p(zka), src.shape[1], _p(s), 1, _p(qq), 1, _p(dd), _p(vv),
                                     n, _p(t), pgh, *[_p(o) for o in out],
                                     ctypes.c_double(abs(zk) * size * 2.0 ** -51)) == 0
    return out


@pytest.mark.parametrize("zk", [0.3 + 0j, 25 + 0j, 180 + 0j, 20 + 2j, 40 - 1j, 3j],
                         ids=lambda z: f"{z}")
@pytest.mark.parametrize("n,nd,points", [(60, 1, "uniform"), (700, 3, "uniform"),
                                         (3001, 1, "blobs"), (20011, 2, "blobs"),
                                         (30000, 1, "uniform")])
def test_all_levels_match_direct_sum(glib, zk, n, nd, points):
    rng = np.random.default_rng(n)
    src = ps.uniform(n, 1) if points == "uniform" else ps.blobs(n, 2)
    trg = ps.uniform(n // 3 + 1, 3)
    q = rng.standard_normal((nd, n)) + 1j * rng.standard_normal((nd, n))
    d = rng.standard_normal((nd, n)) + 1j * rng.standard_normal((nd, n))
    v = rng.standard_normal((nd, 2, n))
    got, ier = W.call_nd(glib, "h", "st_cd_h", EPS, src, nd, True, q, d, v, trg, zk=zk)
    assert ier == 0
    size = max(np.ptp(np.concatenate([src, trg], 1), axis=1))
    for where, pts in (("", src), ("targ", trg)):
        sub = pts[:, :100]
        want = _direct(glib, zk, src, q, d, v, sub, 3, size)
        for name, w, pgh in (("pot", want[0], 1), ("grad", want[1], 2), ("hess", want[2], 3)):
            g = got[name + where][:100].reshape(w.shape)
            assert W.rel_err(g, w) < TOL[pgh], (name, where)


# (sources alone, targets alone, the same outputs, different ones) x sizes on
# both sides of the lanes-per-point rule
@pytest.mark.parametrize("pgh", [(1, 0), (0, 2), (2, 2), (3, 1), (1, 3)])
@pytest.mark.parametrize("ns,nt", [(500, 33), (6000, 4000), (30000, 50000)])
@pytest.mark.parametrize("zk", [12 + 0j, 12 + 0.5j], ids=["real", "complex"])
def test_point_sets(glib, pgh, ns, nt, zk):
    import fmm2d_c_translation_b200 as fm
    rng = np.random.default_rng(3)
    src, trg = ps.uniform(ns, 1), ps.blobs(nt, 2)
    q = rng.standard_normal((1, ns)) + 1j * rng.standard_normal((1, ns))
    d = rng.standard_normal((1, ns)) + 1j * rng.standard_normal((1, ns))
    v = rng.standard_normal((1, 2, ns))
    o = fm.hfmm2d(eps=EPS, zk=zk, sources=src, charges=q[0], dipstr=d[0], dipvec=v[0],
                  targets=trg if pgh[1] else None, pg=pgh[0], pgt=pgh[1])
    both = np.concatenate([src, trg], 1) if pgh[1] else src
    size = max(np.ptp(both, axis=1))
    for where, pts, p in (("", src, pgh[0]), ("targ", trg, pgh[1])):
        if not p:
            continue
        want = _direct(glib, zk, src, q, d, v, pts[:, -60:], p, size)
        for name, w, c in (("pot", want[0], 1), ("grad", want[1], 2), ("hess", want[2], 3))[:p]:
            g = np.asarray(getattr(o, name + where))
            g = g.reshape(c, -1).T if c > 1 else g.reshape(-1, 1)
            assert W.rel_err(g[-60:], w[:, :, 0]) < TOL[c], (name, where)
