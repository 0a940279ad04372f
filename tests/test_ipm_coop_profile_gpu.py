"""The multi-CTA IPM's time by parts (bqb_ipm_coop_profile): every part is
counted, the panel blocks' loads are a part of the panel factorisations, and
reset and disable work."""
import ctypes as C

import numpy as np
import pytest

from helpers import instances, root_L
from parallel_biqbin_maxcut_b200 import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("n", [130, 343])
def test_every_part_is_counted(lib, n):
    L = _lib.colmajor(root_L(instances.gnp_pm1(n, 0.5, n)))
    X, phi, out = np.zeros(n * n), C.c_double(), (C.c_double * 8)()
    lib.bqb_ipm_coop_profile_enable(1)
    try:
        lib.ipm_mc_pk(_lib.dptr(L), n, _lib.dptr(X), C.byref(phi), 0)
        lib.bqb_ipm_coop_profile(out, 1)
        profiled = phi.value, X.copy()
        lib.bqb_ipm_coop_profile_enable(0)
        lib.ipm_mc_pk(_lib.dptr(L), n, _lib.dptr(X), C.byref(phi), 0)
        barrier, factor, tiles, products, call, barriers, phases, loads = out
        assert min(out) > 0, list(out)
        assert loads < factor and barrier + factor + tiles + products < call, list(out)
        assert barriers > phases
        assert profiled[0] == phi.value and np.array_equal(profiled[1], X)
        lib.bqb_ipm_coop_profile(out, 1)
        assert not any(out)
    finally:
        lib.bqb_ipm_coop_profile_enable(0)
