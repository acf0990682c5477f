"""M2M of large levels at orders above 39 (a thread per output): the sums, and
that its time stays near L2L's, which does the same arithmetic (1.15 times; 2.5
with four lanes per output over the whole triangular table)."""
import ctypes

import numpy as np
import pytest

import pointsets as ps
import wrappers as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-13, 1e-14])
def test_m2m(eps):
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    n, m = 1_000_000, 40
    src = ps.uniform(n, 1)
    q = np.random.default_rng(2).standard_normal(n) + 0j
    buf, times = ctypes.create_string_buffer(8192), {}
    L.fmm2d_b200_set_profiling(1)
    try:
        for _ in range(5):
            got, ier = W.call(L, "l", "s_c_p", eps, src, q)
            assert ier == 0
            L.fmm2d_b200_last_profile(buf, len(buf))
            for kv in buf.value.decode().split(";"):
                if "=" in kv:
                    k, v = kv.split("=")
                    times.setdefault(k, []).append(float(v))
    finally:
        L.fmm2d_b200_set_profiling(0)
    assert min(times["m2m"]) < 1.8 * min(times["l2l"])
    d = np.hypot(src[0, :m, None] - src[0], src[1, :m, None] - src[1])
    d[np.arange(m), np.arange(m)] = 1.0
    # (rounding of 1e6 terms of either sign)
    assert W.rel_err(got["pot"][:m], np.log(d) @ q) < 1e-11
