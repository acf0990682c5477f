"""Units so small or large that the square of the wavenumber leaves the normal
numbers: potentials of charges depend on k r alone, so they are those of the
same points in ordinary units."""
import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu


# the two calls share the tree and the expansions to the bit (powers of two);
# the near field takes H0 from a table in one and from continued fractions in
# the other, each to a few 1e-16, and 2,000 charges of either sign cancel two
# digits at most
@pytest.mark.parametrize("k,e", [(1000.0, 505), (40 * 2.0 ** -22, -508), (40.0, 0)])
def test_units(k, e):
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    n = 2000
    src = ps.uniform(n, 1)
    rng = np.random.default_rng(2)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    want, ier = W.call(L, "h", "s_c_p", 1e-12, src, q, zk=k)
    assert ier == 0
    got, ier = W.call(L, "h", "s_c_p", 1e-12, src * 2.0 ** -e, q, zk=k * 2.0 ** e)
    assert ier == 0
    assert W.rel_err(got["pot"], want["pot"]) < 1e-12
