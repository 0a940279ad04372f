"""The grid that the multi-CTA IPM (n > 128) uses without a schedule's entry is
the fastest: no other, of the autotuner's candidates or a CTA for half a pair of
32 x 32 tiles, is faster by more than the timing's spread (1.5 %; the best of
24 calls of one grid, taken in turn with the others', repeats to 0.3 %)."""
import ctypes as C
import time

import numpy as np
import pytest

from helpers import instances, root_L
from parallel_biqbin_maxcut_b200 import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("n", [160, 208, 343])
def test_default_grid_is_the_fastest(lib, n):
    L = _lib.colmajor(root_L(instances.gnp_int(n, 0.9, 10, n)))
    X, phi = np.zeros(n * n), C.c_double()
    T = (n + 31) // 32
    best = {g: 1e9 for g in (0, 148, T * T, T * (T + 1), (T * T + 1) // 2)}   # (0: no entry)
    try:
        for _ in range(24):
            for g in best:
                lib.bqb_ipm_schedule_set(n, g)
                t = time.perf_counter()
                lib.ipm_mc_pk(_lib.dptr(L), n, _lib.dptr(X), C.byref(phi), 0)
                best[g] = min(best[g], time.perf_counter() - t)
    finally:
        lib.bqb_ipm_schedule_set(n, 0)
    assert best[0] <= 1.015 * min(best.values()), best
