"""What a caller of the rounding sees besides its cut: a local search that stops
at its flip limit (an asymmetric P_L makes two vertices flip for ever; the
rounding then goes on with the cuts it has)."""
import ctypes as C

import numpy as np
import pytest

from helpers import O, instances
from parallel_biqbin_maxcut_b200 import _lib
from test_errors import hook  # noqa: F401
from test_heuristic_gpu import libc


def _round(lib, SPL, L):
    n = L.shape[0]
    N = SPL.shape[0] - 1
    x = np.zeros(N, np.int32)
    v = lib.runHeuristic_unpacked(_lib.dptr(_lib.colmajor(SPL)), N + 1, _lib.dptr(_lib.colmajor(L)), n,
                                  _lib.iptr(np.zeros(N, np.int32)), _lib.iptr(np.zeros(N, np.int32)), _lib.iptr(x))
    return v, x


def _problem(nv):
    SPL = O.build_SP_L(instances.gnp_unit(nv, 0.5, nv))
    return SPL, O.create_subproblem(SPL, np.zeros(nv - 1, int), np.zeros(nv - 1, int))


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [20, 140])
def test_local_search_at_its_limit_is_no_failed_factorisation(lib, lib_globals, hook, nv):  # noqa: F811
    SPL, L = _problem(nv)
    n = L.shape[0]
    lib_globals["X"][: n * n] = _lib.colmajor(0.9 * np.eye(n) + 0.1)
    P = L.copy()
    P[:2, :] = P[:, :2] = 0.0
    P[0, 1], P[1, 0] = 5.0, -5.0
    libc.srand(5)
    v, x = _round(lib, SPL, P)
    assert not hook, lib.bqb_last_error()
    assert v == O.evaluateSolution(SPL, x)
