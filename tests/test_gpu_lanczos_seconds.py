"""What a solve's times count: steps that were already on their way when convergence was read belong to the iteration,
not to the refinement, and a solve of long steps runs one of them at most."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu


def _times(H, runs, **options):
    """The smallest times of `runs` solves, and the steps taken."""
    r = [H.lanczos(num_eigenvalues=10, start_vector=np.random.default_rng(3).standard_normal(H.dimension), allow_unconverged=True,
                   **options) for _ in range(runs + 1)][1:]
    return min(q["iteration_seconds"] for q in r), min(q["refinement_seconds"] for q in r), r[0]["iterations"]


def test_refinement_leaves_the_steps_out(problem):
    d, Z, N, *_ = problem("he4_n6_3b")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    _, after, k = _times(H, 10, max_iterations=300, tolerance=1e-6)
    # the same solve, ended by its limit: no step is under way when it refines
    _, alone, same = _times(H, 10, max_iterations=k, tolerance=1e-300)
    assert same == k
    # two steps of 130 us are a quarter of the refinement's time
    assert after < 1.12 * alone
    H.close()


@pytest.mark.slow
def test_long_steps_past_convergence(problem):
    d, Z, N, *_ = problem("li6_n6_3b")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    for every in (1, 10):
        t, _, k = _times(H, 3, max_iterations=300, tolerance=1e-4, check_every=every)
        limit, _, same = _times(H, 3, max_iterations=k, tolerance=1e-300, check_every=every)
        assert same == k
        assert t - limit < 1.5 * limit / k
    H.close()
