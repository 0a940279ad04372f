"""The multi-CTA IPM's autotuner (n > 128) times the grid that it would replace."""
import ctypes as C

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [150, 200, 256])
def test_autotuner_times_the_default(lib, n):
    """Six grids, one warm-up and at least three calls each: the default T (T + 1),
    T^2 and its fractions, the SM count (all different at these sizes)."""
    g, ms = C.c_int(), C.c_double()
    T = (n + 31) // 32
    try:
        before = lib.bqb_kernel_launches()
        assert lib.bqb_ipm_autotune(n, 1, C.byref(g), C.byref(ms)) == 0
        assert lib.bqb_kernel_launches() - before == 6 * (1 + 3)
    finally:
        lib.bqb_ipm_schedule_set(n, 0)
    assert g.value in {T * (T + 1), T * T, (T * T + 1) // 2, (T * T + 3) // 4, (T * T + 7) // 8, 148}
    assert ms.value > 0
