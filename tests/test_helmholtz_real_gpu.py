"""The passes of a positive real wavenumber (csrc/helm_real.cuh and the table
near field) against the passes of a general one, on the same inputs: a
wavenumber whose imaginary part is too small to matter takes the general
kernels."""
import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu

# Both forms sum the same truncated series; a recurrence of at most 100 orders
# adds two roundings of 1.1e-16 per order (2e-14), and the second derivatives'
# sums cancel at most two digits: 2e-12; 5x room.
TOL = 1e-11


@pytest.fixture(scope="module")
def glib():
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    L.fmm2d_b200_set_precision(1)
    yield L
    L.fmm2d_b200_set_precision(0)


# zk: all levels low frequency; several wavelengths per leaf-parent; levels
# above and below the largest box that the real kernels take; a grid whose
# points lie on box centers
@pytest.mark.parametrize("zk,points", [(0.02, "uniform"), (10.0, "blobs"), (150.0, "uniform"),
                                       (420.0, "blobs"), (3.0, "grid")])
@pytest.mark.parametrize("variant", ["st_cd_h", "st_c_g", "t_d_p"])
def test_real_equals_general(glib, zk, points, variant):
    rng = np.random.default_rng(11)
    if points == "uniform":
        src, trg = ps.uniform(2500, 1), ps.uniform(1203, 2)
    elif points == "blobs":
        src, trg = ps.blobs(4000, 3), ps.blobs(1001, 4)
    else:
        src, trg = ps.grid_lines(40), ps.grid_lines(32)
    nd, ns = 2, src.shape[1]
    q = rng.standard_normal((nd, ns)) + 1j * rng.standard_normal((nd, ns))
    d = rng.standard_normal((nd, ns)) + 1j * rng.standard_normal((nd, ns))
    v = rng.standard_normal((nd, 2, ns))
    outs = []
    for k in (complex(zk), complex(zk, 1e-200)):
        got, ier = W.call_nd(glib, "h", variant, 1e-9, src, nd, True, q, d, v, trg, zk=k)
        assert ier == 0
        outs.append(got)
    for name in outs[0]:
        assert W.rel_err(outs[0][name], outs[1][name]) < TOL, name
    # one density: the near field with one warp per leaf
    one = [W.call(glib, "h", variant, 1e-9, src, q[0], d[0], v[0], trg, zk=k)[0]
           for k in (complex(zk), complex(zk, 1e-200))]
    for name in one[0]:
        assert W.rel_err(one[0][name], one[1][name]) < TOL, name
