"""The triangle separation's replay with equal values (src/cutting_planes.c:
70-116: a cut replaces the list's first-found minimum when it is strictly
larger): few and many distinct values, in random and rising order, lists around
a chunk (512 cuts), the longest whose two lists fit in shared memory and the
next one.  Always more candidates than the list holds; the list equals the
oracle's, slot for slot."""
import ctypes as C
import time

import numpy as np
import pytest

from helpers import O
from parallel_biqbin_maxcut_b200 import _lib
from test_trisep_gpu import gpu_sep


def _X(n, levels, rising):
    rng = np.random.default_rng(n + levels)
    X = rng.uniform(-1.0, 1.0, (n, n))
    if rising:   # larger violations for later vertices
        X = -0.2 - 0.8 * np.add.outer(np.arange(n), np.arange(n)) / (2.0 * n) + 0.05 * X
    if levels:
        X = np.round(levels * X) / levels
    X = np.tril(X, -1)
    X = X + X.T
    np.fill_diagonal(X, 1.0)
    return X


def _boundary():
    """The longest list of the CTA-wide replay: two lists of 16 bytes a cut, 60
    bytes a thread of 512, 256 bytes."""
    import torch
    return (torch.cuda.get_device_properties(0).shared_memory_per_block_optin - 512 * 60 - 256) // 32


@pytest.mark.gpu
@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("levels", [0, 1, 2, 8, 100, 2000, 50000])
@pytest.mark.parametrize("T", [1, 2, 33, 511, 512, 513, 1500, "longest", "next"])
def test_equal_values(lib, rising, levels, T):
    X = _X(60, levels, rising)
    if isinstance(T, str):
        T = _boundary() + (T == "next")
    got, mx = gpu_sep(lib, X, T, 0.05)
    want, mx_ref = O.getViolated_TriangleInequalities(X, T, 0.05)
    assert mx == mx_ref
    assert got == want
    more, _ = O.getViolated_TriangleInequalities(X, T + 1, 0.05)
    assert len(got) == T and len(more) == T + 1   # (there were more candidates than places)


@pytest.mark.gpu
@pytest.mark.parametrize("levels", [0, 8])
@pytest.mark.parametrize("n", [6, 10, 16, 20, 22, 24, 30])
@pytest.mark.parametrize("T", [1, 2, 7, 8, 9])
def test_short_lists(lib, n, levels, T):
    X = _X(n, levels, False)
    got, mx = gpu_sep(lib, X, T, 0.05)
    want, mx_ref = O.getViolated_TriangleInequalities(X, T, 0.05)
    assert mx == mx_ref
    assert got == want


@pytest.mark.gpu
def test_equal_values_cost_no_replay_by_single_cuts(lib):
    """A list too long for shared memory is replayed one cut at a time; equal
    values in a shorter one take less than half of that."""
    n = 100
    ms = []
    for levels, T in ((0, 7000), (1000, 5000)):
        x = _lib.colmajor(_X(n, levels, False))
        _lib.set_params(lib, _lib.make_params(TriIneq=T, violated_TriIneq=0.05))
        lst = (_lib.TriIneq * T)()
        size = C.c_int()
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            lib.getViolated_TriangleInequalities(_lib.dptr(x), n, lst, C.byref(size))
            best = min(best, time.perf_counter() - t)
        assert size.value == T
        ms.append(1e3 * best)
    assert ms[1] <= 0.5 * ms[0], ms
