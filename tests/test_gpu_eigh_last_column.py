"""The last diagonal element of the tridiagonal matrix: the cluster panel's last
column is written by one thread and stored by another. A matrix diag(B, x) with a
decoupled last row has x itself as an eigenvalue, so a lost or stale last element
shows as a wrong eigenvalue of order |x|. Panels whose last column is alone
(n mod 32 = 1), full, and in between; one CTA and clusters.

Tolerance: a backward-stable solver moves an eigenvalue by a modest multiple of
n eps max|lambda|: 1e-12 relative up to n = 616 (n eps = 1.4e-13)."""
import numpy as np
import pytest

import tinyscf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 33, 34, 47, 64, 65, 66, 260, 511, 616])
def test_decoupled_last_row(n):
    rng = np.random.default_rng(n)
    B = rng.normal(size=(n - 1, n - 1))
    for x in (-3.7 * n, 2.9 * n):
        A = np.zeros((n, n))
        A[:-1, :-1] = B + B.T
        A[-1, -1] = x
        w, V = tinyscf.eigh(A)
        ref = np.linalg.eigvalsh(A)
        assert np.abs(w - ref).max() < 1e-12 * np.abs(ref).max()
        k = np.abs(w - x).argmin()
        assert abs(w[k] - x) < 1e-12 * abs(x)
        assert abs(abs(V[k, -1]) - 1.0) < 1e-12
