"""Contexts of one process do not change each other's kernels: a large basis, opened before a small one, still runs."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [("he4_n4_2b", "he4_n2_2b"), ("he4_n6_3b", "he4_n2_3b"), ("li6_n2_3b", "he4_n2_2b")])
@pytest.mark.parametrize("bits", [32, 64])
def test_block_tiles_of_the_larger_basis(problem, large, small, bits):
    def opened(name):
        d, Z, N, *_ = problem(name)
        H = jn.Hamiltonian.from_dir(d, Z, N)
        H.set_engine(3)
        H.set_precision(bits)
        return H, d

    H, d = opened(large)
    x = np.random.default_rng(1).standard_normal(H.dimension)
    me = [H.read_matrix_elements(d + "/matrix_elements")]
    solve = lambda: H.lanczos_batch(me, max_iterations=30, num_eigenvalues=3, tolerance=1e-300, precision=bits)[0]["eigenvalues"]
    want, low = H.matvec(x), solve()
    other, _ = opened(small)
    assert np.array_equal(H.matvec(x), want)
    assert np.array_equal(solve(), low)
    other.matvec(np.ones(other.dimension))
    other.close()
    H.close()
