"""A tree that outgrows its limit is refused.  With ndiv = 0 every point goes
down to the last level, where box centers are rounding errors apart and the
level restriction multiplies the boxes by four per level: 11,000 boxes would
become 5e8, past the 32-bit places of the box arrays."""
import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["keys", "keys_sync", "levelwise"])
def test_refused_beyond_the_limit(form, monkeypatch):
    import fmm2d_c_translation_b200 as fm
    monkeypatch.delenv("FMM2D_B200_TREE", raising=False)
    monkeypatch.delenv("FMM2D_B200_TREE_SYNC", raising=False)
    if form == "levelwise":
        monkeypatch.setenv("FMM2D_B200_TREE", "levelwise")
    if form == "keys_sync":
        monkeypatch.setenv("FMM2D_B200_TREE_SYNC", "1")
    src = ps.blobs(60, 833618631, nblob=1, sigma=2.975897354769266e-06)
    with pytest.raises(fm.FmmError, match="tree too large"):
        fm.tree_build(src, None, ndiv=0)
    fm.lib().fmm2d_b200_release_memory()
    got = fm.tree_build(src, None, ndiv=5)
    assert np.array_equal(np.sort(got["isrc"]), np.arange(1, 61))
