"""The one-CTA IPM's results do not depend on the form of its parts: the tile
inverse (n <= 120) gives the same bits as the sweep by single columns (n > 120)
and fails for the same matrices, and the allocation-free entry point gives the
same bits as ipm_mc_pk."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from helpers import instances, root_L
from parallel_biqbin_maxcut_b200 import _lib, build
from test_zz_no_alloc import _noalloc, _regular


@pytest.fixture(scope="module")
def inverse(lib, tmp_path_factory):
    try:
        build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc to build tests/inverse_bits.cu with")
    so = str(tmp_path_factory.mktemp("inverse") / "inverse_bits.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "inverse_bits.cu")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I" + build.CSRC, "-shared", "-o", so, src], check=True)
    f = C.CDLL(so).inverse
    f.argtypes = [C.POINTER(C.c_double), C.c_int, C.c_int, C.POINTER(C.c_double)]

    def run(A, form):
        n = A.shape[0]
        out = np.zeros(n * n)
        return f(_lib.dptr(_lib.colmajor(A)), n, form, _lib.dptr(out)), out

    return run


def _matrix(n, kind):
    rng = np.random.default_rng(1000 * n + len(kind))
    G = rng.standard_normal((n, n))
    A = G @ G.T / n + 0.1 * np.eye(n)
    if kind == "graded":   # entries over ten decades
        d = 10.0 ** rng.uniform(-5, 5, n)
        A = d[:, None] * A * d[None, :]
    elif kind == "nearly singular":
        A = G[:, : n // 2 + 1] @ G[:, : n // 2 + 1].T / n + 1e-10 * np.eye(n)
    elif kind == "indefinite":   # the pivot of the last third turns negative
        A[(2 * n) // 3, (2 * n) // 3] = -1.0
    return 0.5 * (A + A.T)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "graded", "nearly singular", "indefinite"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 24, 60, 100, 113, 119, 120])
def test_tile_inverse_is_the_column_sweep(inverse, n, kind):
    A = _matrix(n, kind)
    ok0, out0 = inverse(A, 0)
    ok1, out1 = inverse(A, 1)
    assert ok0 == ok1 == (0 if kind == "indefinite" else 1)
    if ok0:
        assert np.array_equal(out0, out1)
        if kind == "plain":
            # the sweep's error is at most a small multiple of n eps cond(A)
            want = np.linalg.inv(A)
            tol = 10 * n * np.finfo(float).eps * np.linalg.cond(A)
            assert np.max(np.abs(_lib.from_colmajor(out0, n) - want)) <= tol * np.max(np.abs(want))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [24, 88, 89, 104, 105, 120, 121, 128])
def test_noalloc_gives_the_same_bits(lib, n):
    L = root_L(instances.gnp_pm1(n, 0.5, 60 + n))
    X, out = _noalloc(lib, L)
    X_ref, phi_ref = _regular(lib, L)
    assert int(out[2]) == 0 and out[0] == phi_ref and np.array_equal(X, X_ref)
