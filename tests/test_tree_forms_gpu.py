"""The key-built tree (all levels at once, level restriction in one
cooperative launch) equals the level-by-level construction of the same tree
bit for bit: box arrays, permutations, ranges and lists.  The sizes also
cover the sort's and the scan's single-block, small-tile and large-tile
forms and their edges."""
import numpy as np
import pytest

import pointsets as ps
from test_tree_gpu import CASES

pytestmark = pytest.mark.gpu


def _mixture(n, seed):
    return np.concatenate([ps.uniform(n, seed), ps.blobs(n, seed + 1, nblob=3, sigma=1e-4)], axis=1)


FORMS = dict(CASES)
FORMS.update({
    # the one-block sort's end, small tiles' remainders, the large tiles' start
    **{f"uniform_{n}": (lambda n=n: (ps.uniform(n, 40), ps.uniform(n // 3 + 1, 41), 12, 0))
       for n in (1, 2, 33, 1023, 4095, 4096, 4097, 5121, 606207, 606208, 606211)},
    "mixture": lambda: (_mixture(40000, 42), ps.blobs(9000, 44), 7, 0),
    # more boxes added by the level restriction than were there before it
    "curve_deep": lambda: (ps.starfish(150000, 0)[0], ps.near_curve_targets(100000, 45), 20, 0),
    "line": lambda: (np.stack([np.linspace(0, 1, 30011), np.zeros(30011)]), None, 5, 0),
    # 31 and more digits per key: two and more key words
    "point_cluster": lambda: (np.concatenate([ps.uniform(900, 46),
                                              0.3 + 1e-11 * ps.uniform(900, 47)], axis=1),
                              ps.uniform(77, 48), 4, 0),
    "ndiv_1": lambda: (ps.uniform(3000, 49), ps.blobs(500, 50), 1, 0),
})


@pytest.mark.parametrize("name", sorted(FORMS))
def test_key_tree_equals_levelwise(name, monkeypatch):
    import fmm2d_c_translation_b200 as fm
    src, trg, ndiv, idiv = FORMS[name]()
    monkeypatch.delenv("FMM2D_B200_TREE", raising=False)
    monkeypatch.delenv("FMM2D_B200_TREE_SYNC", raising=False)
    got = fm.tree_build(src, trg, ndiv=ndiv, idivflag=idiv)
    monkeypatch.setenv("FMM2D_B200_TREE", "levelwise")
    want = fm.tree_build(src, trg, ndiv=ndiv, idivflag=idiv)
    assert sorted(got) == sorted(want)
    for k in got:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
