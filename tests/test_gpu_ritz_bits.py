"""The Ritz values that a solve reports are those of its tridiagonal matrix alone: the same bits however often
convergence was tested on the way, and the first of jn_lanczos_ritz_values."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,steps,bits", [("he4_n2_3b", 40, 64), ("he4_n4_2b", 60, 64), ("he4_n4_2b", 61, 32), ("li6_n2_3b", 90, 64)])
def test_single(problem, name, steps, bits):
    d, Z, N, *_ = problem(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_precision(bits)
    start = np.random.default_rng(3).standard_normal(H.dimension)
    seen = []
    for every in (1, 2, 7, steps):
        r = H.lanczos(max_iterations=steps, num_eigenvalues=10, tolerance=1e-300, start_vector=start, check_every=every,
                      allow_unconverged=True)
        assert r["iterations"] == steps
        assert np.array_equal(r["ritz_values"], H.ritz_values()[:10])
        seen.append(r["ritz_values"])
    for s in seen[1:]:
        assert np.array_equal(s, seen[0])
    H.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_batch(problem, precision):
    d, Z, N, *_ = problem("he4_n4_2b")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    me = H.read_matrix_elements(d + "/matrix_elements")
    seen = []
    for every in (1, 6, 60):
        rows = H.lanczos_batch([me, 1.1 * me], max_iterations=60, num_eigenvalues=8, tolerance=1e-300, check_every=every,
                               precision=precision)
        assert [r["iterations"] for r in rows] == [60, 60]
        seen.append(np.concatenate([r["ritz_values"] for r in rows]))
    for s in seen[1:]:
        assert np.array_equal(s, seen[0])
    H.close()
