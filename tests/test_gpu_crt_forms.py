"""The integer rank-k product's CRT has two forms: ranges of K added up in groups
before it, and an element a thread where a range alone is too long to share a
group (512 and more of its 1023 chunks of 128). Integer-valued operands are exact
in every step, so both sides of the line must give the exact product."""
import numpy as np
import pytest

import tinyscf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [511, 512])   # 45 tiles of 256 x 256 leave all of K in one range
def test_exact_on_both_sides_of_the_line(chunks):
    rng = np.random.default_rng(chunks)
    T = rng.integers(-64, 65, size=(2049, 128 * chunks)).astype(np.float64)
    T[7] = 0.0
    K = tinyscf.syrk_int8(T)
    assert np.array_equal(K, T @ T.T)   # |sums| < 2^53: exact
