"""A batch's inputs and outputs in host memory and in device memory, at
addresses that are multiples of 16 bytes and of 8 only, give the same bits."""
import ctypes

import numpy as np
import pytest

import pointsets as ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("place", ["device", "device8", "mixed"])
@pytest.mark.parametrize("with_targets", [False, True])
def test_batch_places(place, with_targets):
    torch = pytest.importorskip("torch")
    import fmm2d_c_translation_b200 as fm
    L = fm.lib()
    rng = np.random.default_rng(4)
    sizes = [1, 37, 500, 3001, 1200]
    k = len(sizes)
    src = [ps.uniform(n, 10 + i) for i, n in enumerate(sizes)]
    q = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for n in sizes]
    d = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for n in sizes]
    v = [rng.standard_normal((2, n)) for n in sizes]
    nt = [0 if i % 2 else n + 3 for i, n in enumerate(sizes)]
    trg = [ps.uniform(max(n, 1), 30 + i) for i, n in enumerate(nt)]
    flat = lambda a: np.ravel(a, order="F").view(np.float64) if np.iscomplexobj(a) \
        else np.ravel(a, order="F")

    def run(where):
        keep = []

        def put(a, i):
            """Address of a copy of the array of problem i."""
            a = np.ascontiguousarray(flat(a), dtype=np.float64)
            if where == "host" or (where == "mixed" and i % 2):
                keep.append((a, None))
                return a.ctypes.data
            off = 1 if where == "device8" else 0
            t = torch.zeros(a.size + 2, dtype=torch.float64, device="cuda")
            t[off:off + a.size] = torch.from_numpy(a).cuda()
            keep.append((t, (off, a.size)))
            return t.data_ptr() + 8 * off

        def ptrs(arrays):
            return (ctypes.c_void_p * k)(*[put(a, i) for i, a in enumerate(arrays)])

        ns = (ctypes.c_int * k)(*sizes)
        ins = [ptrs(x) for x in (src, q, d, v)]
        nts = (ctypes.c_int * k)(*nt) if with_targets else None
        tp = ptrs(trg) if with_targets else None
        first = len(keep)
        outs = [ptrs([np.zeros(2 * c * n) for n in sizes]) for c in (1, 2)]
        touts = [ptrs([np.zeros(2 * c * max(n, 1)) for n in nt]) for c in (1, 2)] \
            if with_targets else [None, None]
        torch.cuda.synchronize()
        ier = L.fmm2d_b200_fmm2d_batch(0, k, ctypes.c_double(1e-9), ns, *ins, 2, *outs, None,
                                       nts, tp, 2 if with_targets else 0, *touts, None)
        assert ier == 0
        torch.cuda.synchronize()
        return [a if o is None else a[o[0]:o[0] + o[1]].cpu().numpy() for a, o in keep[first:]]

    for a, b in zip(run("host"), run(place)):
        assert np.array_equal(a, b)
