"""The sort's form for 2^30 items and more (64-bit tile states) sorts smaller
sets as the 32-bit one does: same tree, bit for bit, over small and large
tiles and their remainders."""
import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 5121, 70001, 606207, 606208, 606211, 2000003])
def test_wide_states(n, monkeypatch):
    import fmm2d_c_translation_b200 as fm
    args = (ps.blobs(n, 1, nblob=5, sigma=1e-3), ps.uniform(n // 3, 2))
    monkeypatch.delenv("FMM2D_B200_SORT_WIDE", raising=False)
    want = fm.tree_build(*args, ndiv=12, lists=False)
    monkeypatch.setenv("FMM2D_B200_SORT_WIDE", "1")
    got = fm.tree_build(*args, ndiv=12, lists=False)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
