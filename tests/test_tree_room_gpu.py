"""Room for the boxes that the level restriction adds: a tree whose boxes fit
is built however much room would be wanted beside them, and a build that runs
out of room starts again with more and gives the same tree."""
import ctypes

import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu


def test_large_deep_tree_is_accepted():
    """One point per leaf: 2.9 boxes per point, many levels.  Three times these
    boxes are more than the 1.07e8 that a tree may have."""
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    n = 15_000_000
    src = np.random.default_rng(1).random((n, 2))
    h = ctypes.c_void_p()
    err = L.fmm2d_b200_tree_build(src.ctypes.data_as(ctypes.c_void_p), n, None, 0, 1, 0,
                                  ctypes.byref(h))
    assert err == 0, fm.last_error()
    nl, nb, lt = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    L.fmm2d_b200_tree_sizes(h, ctypes.byref(nl), ctypes.byref(nb), ctypes.byref(lt))
    L.fmm2d_b200_tree_free(h)
    L.fmm2d_b200_release_memory()
    assert nb.value > 36_000_000


@pytest.mark.parametrize("name", ["curve", "blobs"])
def test_rebuild_with_more_room(name, monkeypatch):
    import fmm2d_c_translation_b200 as fm
    if name == "curve":
        args = (ps.starfish(150000, 0)[0], ps.near_curve_targets(100000, 45))
    else:
        args = (ps.blobs(200000, 4, nblob=30, sigma=1e-4), ps.blobs(9000, 5))
    want = fm.tree_build(*args, ndiv=20)
    monkeypatch.setenv("FMM2D_B200_TREE_ROOM", "0")  # (1,024 boxes)
    got = fm.tree_build(*args, ndiv=20)
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
