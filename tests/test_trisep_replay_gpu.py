"""The chunked replay of the triangle separation (src/cutting_planes.c:70-116):
list lengths around a chunk (512 cuts), the longest whose two lists fit in
shared memory and one that does not, candidates in random and in rising order
(every candidate of a chunk taken), and equal values.  The list equals the
oracle's, slot for slot."""
import numpy as np
import pytest

from helpers import O
from test_trisep_gpu import gpu_sep


def _X(kind, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-1.0, 1.0, (n, n))
    if kind == "rising":   # larger violations for later vertices
        X = -0.2 - 0.8 * (np.add.outer(np.arange(n), np.arange(n)) / (2.0 * n)) + 1e-6 * X
    elif kind == "ties":
        X = np.round(8.0 * X) / 8.0
    X = np.tril(X, -1)
    X = X + X.T
    np.fill_diagonal(X, 1.0)
    return X


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n", [("random", 40), ("rising", 40), ("ties", 30)])
@pytest.mark.parametrize("T", [1, 2, 511, 512, 513, 5000, 7000])
def test_replay_is_the_reference_order(lib, kind, n, T):
    X = _X(kind, n)
    got, mx = gpu_sep(lib, X, T, 0.05)
    want, mx_ref = O.getViolated_TriangleInequalities(X, T, 0.05)
    assert mx == mx_ref
    assert got == want
