"""A batch's arrays in device memory that the one-launch copies do not take:
addresses that are no multiple of 8 bytes, and outputs that problems share
(the last problem's values stay)."""
import ctypes

import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu

SIZES = [300, 1, 777]


def _run(put, out):
    """Batch of Laplace charges; put(array, i) and out(n, i) give addresses."""
    import fmm2d_c_translation_b200 as fm
    import torch
    L = fm.lib()
    k = len(SIZES)
    rng = np.random.default_rng(4)
    src = [ps.uniform(n, 10 + i) for i, n in enumerate(SIZES)]
    q = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for n in SIZES]
    ptrs = lambda a: (ctypes.c_void_p * k)(*a)
    ins = [ptrs([put(np.ravel(a, order="F"), i) for i, a in enumerate(x)]) for x in (src, q)]
    pot = ptrs([out(n, i) for i, n in enumerate(SIZES)])
    torch.cuda.synchronize()
    ier = L.fmm2d_b200_fmm2d_batch(0, k, ctypes.c_double(1e-9), (ctypes.c_int * k)(*SIZES), ins[0],
                                   ins[1], None, None, 1, pot, None, None, None, None, 0, None,
                                   None, None)
    assert ier == 0, fm.last_error()
    torch.cuda.synchronize()


def _host():
    keep = []

    def put(a, i):
        keep.append(np.ascontiguousarray(a))
        return keep[-1].ctypes.data

    outs = [np.zeros(n, np.complex128) for n in SIZES]
    _run(put, lambda n, i: outs[i].ctypes.data)
    return outs


def test_addresses_at_4_bytes():
    torch = pytest.importorskip("torch")
    want, keep = _host(), []

    def put(a, i):
        b = np.frombuffer(np.ascontiguousarray(a).tobytes(), np.uint8)
        t = torch.zeros(b.size + 16, dtype=torch.uint8, device="cuda")
        t[4:4 + b.size] = torch.from_numpy(b.copy()).cuda()
        keep.append(t)
        return t.data_ptr() + 4

    outs = [torch.zeros(16 * n + 16, dtype=torch.uint8, device="cuda") for n in SIZES]
    _run(put, lambda n, i: outs[i].data_ptr() + 4)
    for o, w, n in zip(outs, want, SIZES):
        b = o.cpu().numpy()
        assert np.array_equal(b[4:4 + 16 * n].tobytes(), w.tobytes())
        assert not b[:4].any() and not b[4 + 16 * n:].any()


def test_shared_outputs_keep_the_last_problem():
    torch = pytest.importorskip("torch")
    want, keep = _host(), []

    def put(a, i):
        keep.append(torch.from_numpy(np.ascontiguousarray(a)).cuda())
        return keep[-1].data_ptr()

    out = torch.zeros(max(SIZES), dtype=torch.complex128, device="cuda")
    _run(put, lambda n, i: out.data_ptr())
    assert np.array_equal(out.cpu().numpy()[:SIZES[-1]], want[-1])
