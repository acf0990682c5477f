"""The pipelined tensor-core M2L on every level (tile form) against the FP32
CUDA-core form: fewer tiles than SMs (one launch with the leading rows), more
tiles than SMs, orders of both operand widths, one to three densities."""
import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu

# TF32 x 3 products (2^-22) against FP32 ones (2^-24): a local coefficient sums
# 27 slots of at most 19 terms, so the forms differ by at most about
# 20 x 2.4e-7 of a term; 4x room for the derivatives' orders
TOL = 2e-5


@pytest.fixture(scope="module")
def mlib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(2)
    yield L
    L.fmm2d_b200_set_precision(0)


@pytest.mark.parametrize("n", [120, 6000, 30000, 400000])
@pytest.mark.parametrize("family,nd,variant", [("l", 1, "s_cd_g"), ("l", 1, "s_c_h"),
                                               ("c", 1, "s_cd_p"), ("r", 3, "s_cd_g")])
@pytest.mark.parametrize("eps", [1e-3, 1e-6])
def test_tile_form_equals_simt(mlib, monkeypatch, n, family, nd, variant, eps):
    rng = np.random.default_rng(n)
    src = ps.uniform(n, 1)

    def strength():
        a = rng.standard_normal((nd, n))
        return a if family == "r" else a + 1j * rng.standard_normal((nd, n))

    q, d, v = strength(), strength(), rng.standard_normal((nd, 2, n))
    outs = []
    for form in ("tile", "simt"):
        monkeypatch.setenv("FMM2D_B200_M2L", form)
        got, ier = W.call_nd(mlib, family, variant, eps, src, nd, True, q, d, v)
        assert ier == 0
        outs.append(got)
    for name in outs[0]:
        assert W.rel_err(outs[0][name], outs[1][name]) < TOL, name
