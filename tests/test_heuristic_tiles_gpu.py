"""The heuristic's tile Cholesky at its edges (n around a tile, and around 128
where the factorisation changes) against the oracle: values, cuts and the
rand() state are equal."""
import numpy as np
import pytest

from helpers import O, instances
from parallel_biqbin_maxcut_b200 import _lib
from test_heuristic_gpu import libc


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [8, 9, 17, 33, 64, 97, 120, 121, 128, 129])
def test_heuristic_at_the_edges(lib, lib_globals, nv):
    SPL = O.build_SP_L(instances.gnp_pm1(nv, 0.5, nv))
    N0 = SPL.shape[0]
    xf, sol = np.zeros(N0 - 1, np.int32), np.zeros(N0 - 1, np.int32)
    L = O.create_subproblem(SPL, xf, sol)
    n = L.shape[0]
    Xm = O.ipm_mc_pk(L).X
    lib_globals["X"][: n * n] = _lib.colmajor(Xm)
    x = np.zeros(N0 - 1, np.int32)
    libc.srand(77)
    v = lib.runHeuristic_unpacked(_lib.dptr(_lib.colmajor(SPL)), N0, _lib.dptr(_lib.colmajor(L)), n, _lib.iptr(xf),
                                  _lib.iptr(sol), _lib.iptr(x))
    after = libc.rand()
    libc.srand(77)
    xo = np.zeros(N0 - 1, np.int64)
    vo = O.runHeuristic_unpacked(SPL, L, xf, sol, xo, Xm)
    assert v == vo and np.array_equal(x, xo) and after == libc.rand()
