"""The near field of a positive real wavenumber (pair_add_real in
csrc/helmholtz.cu with the table of csrc/helm_bessel.cuh) against the direct
sum, which evaluates H0 and H1 with CUDA's Bessel functions: all points in
one leaf, so the evaluation is the near field alone."""
import numpy as np
import pytest

import wrappers as W
from test_helmholtz_gpu import h_direct

pytestmark = pytest.mark.gpu

# A pair's terms carry at most about 40 rounding errors of 1.1e-16 (Horner
# sums, logarithm, reciprocal), and the second derivatives cancel at most
# about one digit between their two parts: 5e-14; 20x room.
TOL = 1e-12


@pytest.fixture(scope="module")
def glib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(1)
    yield L
    L.fmm2d_b200_set_precision(0)


# x = k r up to 1.4 k: far below the first interval's center, inside the
# first few intervals, up to the table's end at x = 16, and beyond it
@pytest.mark.parametrize("zk", [1e-4, 0.9, 11.4, 60.0])
@pytest.mark.parametrize("variant", ["st_c_h", "st_d_h", "st_cd_h", "st_cd_p", "s_c_p", "t_d_g"])
def test_one_leaf_equals_direct_sum(glib, zk, variant):
    rng = np.random.default_rng(3)
    ns, nt = 18, 33
    src, trg = rng.random((2, ns)), rng.random((2, nt))
    trg[:, 0] = src[:, 4]  # a target on a source
    q = rng.standard_normal(ns) + 1j * rng.standard_normal(ns)
    d = rng.standard_normal(ns) + 1j * rng.standard_normal(ns)
    v = rng.standard_normal((2, ns))
    got, ier = W.call(glib, "h", variant, 1e-9, src, q, d, v, trg, zk=complex(zk))
    assert ier == 0
    st, cd, p = variant.split("_")
    pgh = {"p": 1, "g": 2, "h": 3}[p]
    for where, pts in (("", src), ("targ", trg)):
        if f"pot{where}" not in got:
            continue
        want = h_direct(glib, complex(zk), src, q, d, v, pts, pgh, int("c" in cd), int("d" in cd))
        for name, w in zip(("pot", "grad", "hess")[:pgh], want):
            assert W.rel_err(got[name + where], w) < TOL, (name + where)
