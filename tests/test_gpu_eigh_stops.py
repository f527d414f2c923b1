"""The eigensolver's two stopping rules of the roots in divide and conquer, each
on its own: the bracketed one (X, (P|Q)^-1/2, the accelerated form's eigenbases)
and the one at noise level (the plain form's density). Both against LAPACK, at
the sizes where merges change kernel (64 positions) and panels change form.

Tolerances: a backward-stable solver's errors are a few n eps max|A|: 1e-12 of
max|A| up to n = 1010 (n eps = 2.2e-13)."""
import numpy as np
import pytest

import tinyscf

pytestmark = pytest.mark.gpu
STOPS = [tinyscf.EIG_BRACKET, tinyscf.EIG_NOISE]


def _check(A, stop):
    n = A.shape[0]
    w, V = tinyscf.eigh(A, stop=stop)
    scale = np.abs(A).max()
    assert np.all(np.diff(w) >= 0)
    assert np.abs(w - np.linalg.eigvalsh(A)).max() < 1e-12 * scale
    assert np.abs(V @ A - w[:, None] * V).max() < 1e-12 * scale
    assert np.abs(V @ V.T - np.eye(n)).max() < 1e-12
    return w, V


@pytest.mark.parametrize("stop", STOPS)
@pytest.mark.parametrize("n", [2, 33, 64, 65, 127, 128, 129, 260, 385, 616, 1010])
def test_random(n, stop):
    X = np.random.default_rng(n).standard_normal((n, n))
    _check(X + X.T, stop)


@pytest.mark.parametrize("stop", STOPS)
def test_clustered(stop):
    rng = np.random.default_rng(7)
    n = 400
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    w = np.r_[np.full(40, -11.2) + 1e-10 * rng.standard_normal(40), np.full(30, -0.5), np.linspace(-1, 3, n - 70)]
    A = (Q * w) @ Q.T
    _check(0.5 * (A + A.T), stop)


@pytest.mark.parametrize("stop", STOPS)
def test_metric_inverse_sqrt(stop):
    """The spectrum of the C40H82 DF metric (condition 6e10), whose inverse square root takes the bracketed rule."""
    rng = np.random.default_rng(11)
    n = 600
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * np.logspace(np.log10(4.5e-8), np.log10(2.8e3), n)) @ Q.T
    A = 0.5 * (A + A.T)
    wg, V = _check(A, stop)
    X = V.T @ (V / np.sqrt(wg)[:, None])
    wl, Vl = np.linalg.eigh(A)
    Xl = Vl @ (Vl.T / np.sqrt(wl)[:, None])
    err = lambda Y: np.abs(Y @ A @ Y - np.eye(n)).max()
    assert err(X) < 10 * max(err(Xl), 1e-10)


def test_other_rules_are_refused():
    with pytest.raises(tinyscf.TinySCFError):
        tinyscf.eigh(np.eye(3), stop=2)
