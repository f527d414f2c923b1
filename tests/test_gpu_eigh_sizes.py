"""The eigensolver at the sizes where its panels change form: one CTA up to 64
rows, clusters of 2 to 16 CTAs, segments of 256 columns, trailing matrices of
616 rows (the most a cluster keeps in shared memory) and 1024 rows (the most it
owns), panels of 32 columns with and without a remainder.

Tolerances: a backward-stable solver's eigenvalues move by a modest multiple of
n eps max|lambda|, its residual and orthogonality likewise: 1e-12 relative up to
n = 1025 (n eps = 2.3e-13)."""
import numpy as np
import pytest

import tinyscf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 256, 257, 384, 385, 512, 513, 616, 648, 768, 769, 1024, 1025])
def test_sizes(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n))
    A = A + A.T
    w, V = tinyscf.eigh(A)
    ref = np.linalg.eigvalsh(A)
    scale = np.abs(ref).max()
    assert np.abs(w - ref).max() < 1e-12 * scale
    assert np.abs(A @ V.T - V.T * w).max() < 1e-12 * scale
    assert np.abs(V @ V.T - np.eye(n)).max() < 1e-12
