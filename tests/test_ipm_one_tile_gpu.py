"""The one-CTA IPM for n <= 8, whose single tile one warp eliminates: the oracle's
result (src/ipm_mc_pk.c:28-359), the same bits as the general kernel (which a
batch with a larger problem uses), and less time."""
import ctypes as C

import numpy as np
import pytest

from helpers import O, instances, root_L
from parallel_biqbin_maxcut_b200 import _lib
from test_zz_no_alloc import _noalloc, _regular


def _L(n, seed):
    if n <= 2:
        return np.diag(np.arange(1.0, n + 1.0)) + seed
    return root_L(instances.gnp_int(n, 0.9, 10, seed))


def _batch(lib, Ls):
    m = len(Ls)
    ns = np.array([L.shape[0] for L in Ls], np.int32)
    host = [_lib.colmajor(L) for L in Ls]
    Xs = [np.zeros(n * n) for n in ns]
    phi, it, st = np.zeros(m), np.zeros(m, np.int32), np.zeros(m, np.int32)
    ptr = lambda a: (C.c_void_p * m)(*[x.ctypes.data for x in a])   # noqa: E731
    lib.bqb_ipm_batch(ptr(host), ptr(Xs), _lib.iptr(ns), m, _lib.dptr(phi), _lib.iptr(it), _lib.iptr(st))
    assert not st.any()
    return [_lib.from_colmajor(X, n) for X, n in zip(Xs, ns)], phi


@pytest.mark.gpu
@pytest.mark.parametrize("n", range(1, 9))
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_one_tile(lib, n, seed):
    L = _L(n, seed)
    X, phi = _regular(lib, L)
    Xn, out = _noalloc(lib, L)
    assert int(out[2]) == 0 and out[0] == phi and np.array_equal(X, Xn)
    for batch in ([L, L], [L, _L(20, seed)]):   # one tile each; the general kernel
        Xb, phib = _batch(lib, batch)
        assert phib[0] == phi and np.array_equal(Xb[0], X)
    if n > 2:
        r = O.ipm_mc_pk(L)
        assert abs(phi - r.phi) <= 1e-6 * max(1.0, abs(r.phi)) and np.max(np.abs(X - r.X)) <= 1e-6


def _us_per_iteration(lib, L):
    import torch
    n = L.shape[0]
    f = lib.bqb_ipm_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    dL = torch.from_numpy(_lib.colmajor(L)).to("cuda")
    dX = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    best = 1e9
    for _ in range(20):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        for _ in range(10):
            assert f(dL.data_ptr(), dX.data_ptr(), n, out.data_ptr(), s.cuda_stream) == 0
        b.record(s)
        s.synchronize()
        best = min(best, 100.0 * a.elapsed_time(b))
    return best / float(out[1])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 4, 8])
def test_one_tile_takes_less_time(lib, n):
    """An iteration takes at most 0.6 of one at n = 16, of two tile rows with
    their hand-overs (with those for one tile, too, it took 0.8)."""
    one, two = _us_per_iteration(lib, _L(n, 1)), _us_per_iteration(lib, _L(16, 1))
    assert one <= 0.6 * two, (one, two)
