"""Eigenvalues and eigenvectors of tridiagonal matrices (jn_tridiagonal, the solves' own kernels) against 40-digit
values: to the last bits, also the small ones of graded matrices, whose entries determine them to as many digits."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

mp = pytest.importorskip("mpmath")
pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _graded(n, step, coupling, seed):
    """Diagonal 2^-(step i), couplings 2^-(step i + coupling): diagonally dominant, so every eigenvalue is determined to
    a few roundings of itself."""
    i = np.arange(n)
    return 2.0 ** -(step * i) * np.random.default_rng(seed).uniform(0.5, 1, n), 2.0 ** -(step * i[:-1] + coupling)


def _exact(a, b):
    n = len(a)
    t = mp.matrix(n)
    for i in range(n):
        t[i, i] = mp.mpf(float(a[i]))
        if i + 1 < n:
            t[i, i + 1] = t[i + 1, i] = mp.mpf(float(b[i]))
    with mp.workdps(60):
        return sorted(mp.eigsy(t, eigvals_only=True))


@pytest.mark.parametrize("n,step,coupling", [(24, 1, 3), (16, 2, 3), (14, 5, 8), (14, 4, 40), (14, 4, 2000), (1, 1, 1), (2, 3, 3)])
@pytest.mark.parametrize("up", [False, True])
def test_graded(n, step, coupling, up):
    a, b = _graded(n, step, coupling, n)
    if up:
        a, b = a[::-1], b[::-1]
    values, vectors = jn.tridiagonal(a, b, num_vectors=n)
    with mp.workdps(60):
        want = _exact(a, b)
        # every step of a count perturbs an entry by a few roundings, relatively, and an eigenvalue moves by as much
        assert max(abs((mp.mpf(float(v)) - w) / w) for v, w in zip(values, want)) <= 8 * EPS
    t = np.diag(a) + np.diag(b, 1) + np.diag(b, -1)
    assert np.abs(vectors @ vectors.T - np.eye(n)).max() <= 64 * EPS
    # the residual of the k-th vector: n roundings of the span
    assert np.abs(t @ vectors.T - vectors.T * values).max() <= 4 * n * EPS * np.abs(values).max()


@pytest.mark.parametrize("n", [3, 33, 64, 100])
def test_random(n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n - 1)
    k = min(n, 12)
    values, vectors = jn.tridiagonal(a, b, num_values=k, num_vectors=k)
    want = np.array([float(v) for v in _exact(a, b)])
    scale = np.abs(want).max()
    # two counts of n / 2 steps that each perturb an entry by a few roundings of the span
    assert np.abs(values - want[:k]).max() <= 4 * EPS * scale
    t = np.diag(a) + np.diag(b, 1) + np.diag(b, -1)
    assert np.abs(vectors @ vectors.T - np.eye(k)).max() <= 64 * EPS
    assert np.abs(t @ vectors.T - vectors.T * values).max() <= 4 * n * EPS * scale
    assert (vectors[:, 0] >= 0).all()


def test_all_values_of_many_rows():
    """More rows than shared memory holds: the 1-2-1 matrix, whose eigenvalues are known."""
    n = 3300
    values, _ = jn.tridiagonal(np.full(n, 2.0), np.full(n - 1, -1.0))
    want = 4 * np.sin(np.pi * np.arange(1, n + 1) / (2 * (n + 1))) ** 2
    assert np.abs(values - want).max() <= 64 * EPS * 4


def test_refuses():
    for args in [([1.0], [], 0, 0), ([1.0, 2.0], [1.0], 3, 0), ([1.0, 2.0], [1.0], 1, 2)]:
        with pytest.raises(jn.JnError):
            jn.tridiagonal(np.array(args[0]), np.array(args[1]), num_values=args[2], num_vectors=args[3])
