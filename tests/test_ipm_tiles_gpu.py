"""The one-CTA IPM (n <= 128) on 8 x 8 tiles: sizes at the edges of a tile, of
a scheduler's share of the rows and of the shared-memory placements, against
the oracle (src/ipm_mc_pk.c:28-359).

Tolerances as in test_ipm_gpu.py: phi 1e-6 relative, X 1e-6 absolute (the
solves lose at most cond(M) eps, far below that at these sizes); the matrices
that do not fit in shared memory only change place, so a problem bounded alone,
in a batch of larger ones and by the allocation-free entry point returns the
same bits."""
import ctypes as C

import numpy as np
import pytest

from helpers import O, instances, root_L
from parallel_biqbin_maxcut_b200 import _lib

RTOL_PHI = 1e-6
ATOL_X = 1e-6


def _ipm(lib, L):
    n = L.shape[0]
    X = np.zeros(n * n)
    phi = C.c_double()
    lib.ipm_mc_pk(_lib.dptr(_lib.colmajor(L)), n, _lib.dptr(X), C.byref(phi), 0)
    return _lib.from_colmajor(X, n), phi.value


def _check(lib, L):
    X, phi = _ipm(lib, L)
    r = O.ipm_mc_pk(L)
    assert abs(phi - r.phi) <= RTOL_PHI * abs(r.phi), (phi, r.phi)
    assert np.max(np.abs(X - r.X)) <= ATOL_X
    assert np.array_equal(X, X.T)
    return X, phi


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 31, 96, 97, 104, 105, 112, 113, 120, 121, 127, 128])
def test_tile_edges(lib, n):
    _check(lib, root_L(instances.gnp_int(n, 0.9, 10, 300 + n)))


@pytest.mark.gpu
def test_one_vertex(lib):
    X, phi = _ipm(lib, np.array([[3.0]]))
    assert abs(X[0, 0] - 1.0) <= 1e-9 and abs(phi - 3.0) <= 1e-2   # (the gap the method stops at)


@pytest.mark.gpu
def test_placements_give_the_same_bits(lib):
    Ls = [root_L(instances.gnp_pm1(n, 0.5, 40 + n)) for n in (24, 100, 110, 128)]
    ns = np.array([L.shape[0] for L in Ls], np.int32)
    host = [_lib.colmajor(L) for L in Ls]
    Xs = [np.zeros(n * n) for n in ns]
    phi, it, st = np.zeros(4), np.zeros(4, np.int32), np.zeros(4, np.int32)
    ptr = lambda a: (C.c_void_p * 4)(*[x.ctypes.data for x in a])   # noqa: E731
    lib.bqb_ipm_batch(ptr(host), ptr(Xs), _lib.iptr(ns), 4, _lib.dptr(phi), _lib.iptr(it), _lib.iptr(st))
    assert not st.any()
    for L, X, p, n in zip(Ls, Xs, phi, ns):
        X1, p1 = _ipm(lib, L)
        assert p == p1 and np.array_equal(_lib.from_colmajor(X, n), X1)
