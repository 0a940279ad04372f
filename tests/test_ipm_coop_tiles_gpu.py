"""The multi-CTA IPM (n > 128): sizes at the edges of its 32 x 32 tiles (a last
panel of 1, 31 and 32 columns, of whole and ragged 8 x 8 fragments) against the
oracle (src/ipm_mc_pk.c:28-359).  Tolerances as in test_ipm_gpu.py."""
import ctypes as C

import numpy as np
import pytest

from helpers import O, instances, root_L
from parallel_biqbin_maxcut_b200 import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 136, 152, 159, 160, 161, 191, 193, 225])
def test_tile_edges(lib, n):
    L = root_L(instances.gnp_int(n, 0.6, 10, 700 + n))
    n = L.shape[0]
    X = np.zeros(n * n)
    phi = C.c_double()
    lib.ipm_mc_pk(_lib.dptr(_lib.colmajor(L)), n, _lib.dptr(X), C.byref(phi), 0)
    X = _lib.from_colmajor(X, n)
    r = O.ipm_mc_pk(L)
    assert abs(phi.value - r.phi) <= 1e-6 * abs(r.phi), (phi.value, r.phi)
    assert np.max(np.abs(X - r.X)) <= 1e-6
    assert np.array_equal(X, X.T)
