"""The mixed M2L's plans (run table, segment tables) and its leading-row
kernel: the default form against the FP32 CUDA-core form on the same tree, at
sizes whose levels hold less than a run, a tile of 32 boxes, of 128 rows, and
a little more."""
import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu

# TF32 x 3 products (2^-22) of the rows above the leading ones against FP32
# ones (2^-24): both sums hold 27 slots of at most 19 terms, so the forms
# differ by at most about 20 x 2.4e-7 of a term, and the upper rows carry less
# than a tenth of the potential and of its derivatives' norms: 5e-7; 4x room
TOL = 2e-6


@pytest.fixture(scope="module")
def mlib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(2)
    yield L
    L.fmm2d_b200_set_precision(0)


@pytest.mark.parametrize("n", [97, 400, 1700, 1701, 6900, 40000])
@pytest.mark.parametrize("family,nd,variant", [("l", 1, "s_cd_h"), ("l", 1, "s_c_g"),
                                               ("r", 3, "s_cd_g"), ("r", 1, "s_c_p")])
@pytest.mark.parametrize("points", ["uniform", "blobs"])
def test_default_form_equals_simt(mlib, monkeypatch, n, family, nd, variant, points):
    rng = np.random.default_rng(n)
    src = ps.uniform(n, 1) if points == "uniform" else ps.blobs(n, 2)

    def strength():
        a = rng.standard_normal((nd, n))
        return a if family == "r" else a + 1j * rng.standard_normal((nd, n))

    q, d, v = strength(), strength(), rng.standard_normal((nd, 2, n))
    outs = []
    for form in (None, "simt"):
        if form is None:
            monkeypatch.delenv("FMM2D_B200_M2L", raising=False)
        else:
            monkeypatch.setenv("FMM2D_B200_M2L", form)
        got, ier = W.call_nd(mlib, family, variant, 1e-6, src, nd, True, q, d, v)
        assert ier == 0
        outs.append(got)
    for name in outs[0]:
        assert W.rel_err(outs[0][name], outs[1][name]) < TOL, name
