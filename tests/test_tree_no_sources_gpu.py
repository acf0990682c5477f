"""Trees of targets alone: with the source counts as the rule (idivflag 0) the
root is the only box, with the target counts the tree is the levelwise one."""
import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idivflag", [0, 1, 2])
@pytest.mark.parametrize("nt", [1, 100, 5000])
def test_targets_only(nt, idivflag, monkeypatch):
    import fmm2d_c_translation_b200 as fm
    trg = ps.blobs(nt, 3)
    monkeypatch.delenv("FMM2D_B200_TREE", raising=False)
    monkeypatch.delenv("FMM2D_B200_TREE_SYNC", raising=False)
    got = fm.tree_build(np.zeros((2, 0)), trg, ndiv=10, idivflag=idivflag)
    if idivflag == 0 or nt <= 10:
        assert (got["nlevels"], got["nboxes"]) == (0, 1)
        assert np.array_equal(got["itarg"], np.arange(1, nt + 1))
    monkeypatch.setenv("FMM2D_B200_TREE", "levelwise")
    want = fm.tree_build(np.zeros((2, 0)), trg, ndiv=10, idivflag=idivflag)
    assert sorted(got) == sorted(want)
    for k in got:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
