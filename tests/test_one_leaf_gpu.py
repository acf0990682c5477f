"""Calls whose points fit one leaf: no pass counts refined boxes and no
cooperative launch restricts levels (three launches fewer, 0.238 -> 0.159 ms
for 10 points), and the sums are the direct ones."""
import ctypes

import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,nt", [(1, 1), (3, 300), (10, 10), (15, 5)])
def test_one_leaf(precision, n, nt):
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    src, trg = ps.uniform(n, 1), ps.uniform(nt, 2)
    q = np.random.default_rng(3).standard_normal(n) + 0j
    L.fmm2d_b200_set_precision(precision)
    try:
        W.call(L, "l", "s_c_p", 1e-6, src, q)
        before = L.fmm2d_b200_launch_count()
        W.call(L, "l", "s_c_p", 1e-6, src, q)
        assert L.fmm2d_b200_launch_count() - before <= 15
        got, ier = W.call(L, "l", "t_c_p", 1e-6, src, q, targ=trg)
    finally:
        L.fmm2d_b200_set_precision(0)
    assert ier == 0
    r = np.hypot(trg[0][:, None] - src[0], trg[1][:, None] - src[1])
    want = np.log(r) @ q
    # FP32 pairs: the logarithm's argument and value rounded to 6e-8
    assert np.abs(got["pottarg"] - want).max() < (1e-12 if precision else 2e-6) * np.abs(q).sum()


def test_tree_of_one_leaf_with_many_targets():
    """More targets than one warp sorts: they stay in input order."""
    import fmm2d_c_translation_b200 as fm
    got = fm.tree_build(ps.uniform(300, 1), ps.uniform(5000, 2), ndiv=300)
    assert (got["nlevels"], got["nboxes"]) == (0, 1)
    assert np.array_equal(got["isrc"], np.arange(1, 301))
    assert np.array_equal(got["itarg"], np.arange(1, 5001))
