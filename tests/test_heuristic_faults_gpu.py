"""What a caller of the rounding sees besides its cut: a local search that stops
at its flip limit (an asymmetric P_L makes two vertices flip for ever; the
rounding then goes on with the cuts it has), the rand() state after a failed
factorisation (src/heuristic.c:38-39, 68-74: only the random cut was drawn), and
the work left on the device at the return (none)."""
import ctypes as C
import os
import subprocess
import sys

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


def _at_the_limit(lib, X, nv):
    SPL, L = _problem(nv)
    n = L.shape[0]
    X[: n * n] = _lib.colmajor(0.9 * np.eye(n) + 0.1)
    P = L.copy()
    P[:2, :] = P[:, :2] = 0.0
    P[0, 1], P[1, 0] = 5.0, -5.0
    libc.srand(5)
    v, x = _round(lib, SPL, P)
    return v, O.evaluateSolution(SPL, x)


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [20, 140])
def test_local_search_at_its_limit_is_no_failed_factorisation(lib, lib_globals, hook, nv):  # noqa: F811
    v, value = _at_the_limit(lib, lib_globals["X"], nv)
    assert not hook, lib.bqb_last_error()
    assert v == value
    # without an abort hook (a failure would end the process) the host draws
    # while the device factors: the same cut
    prog = ("from test_heuristic_faults_gpu import _at_the_limit, _lib\n"
            "lib = _lib.load()\n"
            "lib.bqb_init(0)\n"
            "g = _lib.GlobalArrays(lib, 200)\n"
            "g.bind()\n"
            f"print(repr(_at_the_limit(lib, g['X'], {nv})))\n")
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == repr((v, value))


@pytest.mark.gpu
def test_failed_factorisation_leaves_the_random_numbers(lib, lib_globals, hook):  # noqa: F811
    SPL, L = _problem(20)
    n = L.shape[0]
    lib_globals["X"][: n * n] = _lib.colmajor(-np.eye(n))
    libc.srand(6)
    _round(lib, SPL, L)
    after = libc.rand()
    assert hook == [10]
    libc.srand(6)
    for _ in range(n):   # the random cut
        libc.rand()
    assert after == libc.rand()


@pytest.mark.gpu
def test_nothing_is_launched_after_the_last_round(lib, lib_globals):
    SPL, L = _problem(40)
    n = L.shape[0]
    lib_globals["X"][: n * n] = _lib.colmajor(O.ipm_mc_pk(L).X)
    libc.srand(7)
    before = lib.bqb_kernel_launches()
    v, x = _round(lib, SPL, L)
    launches = lib.bqb_kernel_launches() - before
    # the random cut's value; a round: factor, project, 1-opt, evaluate, select;
    # a re-mix of Z between two rounds
    assert launches % 6 == 0 and launches >= 12
    assert v == O.evaluateSolution(SPL, x)
