"""The Lanczos step and its convergence check where their layouts change: bases smaller than a warp, Krylov spaces
up to the whole basis (every number of vectors, couplings down to rounding), and T_n above the rows that the
tridiagonal kernels keep in shared memory."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Z,N,nmax,M2,nbody", [(3, 3, 0, 2, 3), (1, 2, 2, 1, 2), (2, 2, 2, 0, 3), (3, 4, 2, 1, 3)])
def test_whole_basis(tmp_path, Z, N, nmax, M2, nbody):
    d = str(tmp_path)
    jn.generate(d, Z=Z, N=N, nmax=nmax, M2=M2, nbody=nbody, basis_files=False)
    p = oracle.Port(d)
    D = p.dimension
    dense = np.column_stack([p.matvec(np.eye(D)[j]) for j in range(D)])
    p.close()
    w = np.linalg.eigvalsh(0.5 * (dense + dense.T))
    H = jn.Hamiltonian.from_dir(d, Z, N)
    n = min(6, D)
    # a tolerance that nothing meets: the solve runs until the Krylov space is the basis
    r = H.lanczos(max_iterations=D, num_eigenvalues=n, tolerance=1e-300, allow_unconverged=True,
                  start_vector=np.random.default_rng(5).standard_normal(D))
    rv = H.ritz_values()
    scale = np.abs(w).max()
    # backward error of D orthonormal steps and of the tridiagonal values: a few D eps |H|
    tol = 8 * D * 2.3e-16 * scale
    assert r["iterations"] == D and len(rv) == D
    assert np.abs(rv - w).max() <= tol
    assert np.abs(r["ritz_values"] - w[:n]).max() <= tol
    assert np.abs(r["eigenvalues"] - w[:n]).max() <= tol
    # a Ritz vector's residual: rounding of the basis, amplified by the closest eigenvalue
    assert r["residual_norms"].max() <= 1e-9 * scale
    H.close()


def test_more_rows_than_shared_memory_holds(problem):
    d, Z, N, *_ = problem("he4_n6_3b")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    start = np.random.default_rng(6).standard_normal(H.dimension)
    want = H.lanczos(max_iterations=400, num_eigenvalues=10, tolerance=1e-10, start_vector=start, check_every=20)
    r = H.lanczos(max_iterations=3300, num_eigenvalues=10, tolerance=1e-300, start_vector=start, check_every=3300,
                  allow_unconverged=True)
    rv = H.ritz_values()
    assert r["iterations"] == 3300 and len(rv) == 3300 and np.all(np.diff(rv) >= 0)
    scale = np.abs(rv).max()
    assert np.abs(r["ritz_values"] - rv[:10]).max() <= 1e-14 * scale
    # want is converged to 1e-10 MeV by its bound, r beyond rounding
    assert np.abs(r["eigenvalues"] - want["eigenvalues"]).max() <= 1e-9
    assert np.abs(r["ritz_values"] - want["eigenvalues"]).max() <= 1e-9
    assert r["residual_norms"].max() <= 1e-9 * scale
    H.close()
