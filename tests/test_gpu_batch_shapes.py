"""The batched solver where its launches change shape: small accumulators (three CTAs an SM), accumulators that fill an
SM with and without x beside them, instances that converge long before others (the CTAs are shared out anew), Krylov
spaces that close (a second Gram-Schmidt pass), and instances of very uneven dimension."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn
import oracle

pytestmark = pytest.mark.gpu
EIG_TOL = 1e-6          # MeV, the solves' tolerance

SYSTEMS = {
    "li6_n0": (3, 3, 0, 2),     # D = 8
    "h3_n2": (1, 2, 2, 1),      # 41
    "he4_n4": (2, 2, 4, 0),     # 952
    "li6_n4": (3, 3, 4, 2),     # 15 764: x beside the accumulator
    "h4_n8": (1, 3, 8, 4),      # the accumulator alone fills an SM
}
_dirs = {}


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    def get(name):
        if name not in _dirs:
            Z, N, nmax, M2 = SYSTEMS[name]
            d = str(tmp_path_factory.mktemp(name))
            jn.generate(d, Z=Z, N=N, nmax=nmax, M2=M2, nbody=2, basis_files=False)
            jn.generate(d + "_1", Z=Z, N=N, nmax=nmax, M2=M2, nbody=2, seed=5, hbar_omega=0.0, basis_files=False)
            _dirs[name] = (d, Z, N)
        return _dirs[name]
    return get


def _open(system, name, count, seed):
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    h0, h1 = (H.read_matrix_elements(f"{q}/matrix_elements") for q in (d, d + "_1"))
    rng = np.random.default_rng(seed)
    # different spectra, so that the instances converge at different steps
    return H, [h0 + c * h1 for c in [0.0, *rng.uniform(-1, 1, count - 1)]]


def _plain(H, me, n):
    H.set_matrix_elements(me)
    return H.lanczos(max_iterations=min(400, H.dimension), num_eigenvalues=n, tolerance=1e-8, check_every=10,
                     start_vector=np.random.default_rng(1).standard_normal(H.dimension), allow_unconverged=True)["eigenvalues"]


@pytest.mark.parametrize("names,count,precision", [
    (["h3_n2"], 1, 32), (["he4_n4"], 3, 32), (["li6_n4"], 3, 32), (["h4_n8"], 2, 32), (["he4_n4"], 2, 64),
    (["li6_n0", "h3_n2", "he4_n4", "li6_n4"], 4, 32), (["h3_n2", "h4_n8"], 2, 32), (["li6_n0", "he4_n4"], 3, 64)])
def test_against_single_solves(system, names, count, precision):
    n = 4
    bases = [_open(system, name, count, 7 + i) for i, name in enumerate(names)]
    got = jn.lanczos_batch_bases(bases, max_iterations=300, num_eigenvalues=n, tolerance=1e-7, precision=precision)
    for (H, mes), rows in zip(bases, got):
        for me, r in zip(mes, rows):
            want = _plain(H, me, n)
            assert len(r["eigenvalues"]) == len(want)
            assert np.abs(r["eigenvalues"] - want).max() < EIG_TOL
        if len(names) == 1:
            for a, r in zip(H.lanczos_batch(mes, max_iterations=300, num_eigenvalues=n, tolerance=1e-7, precision=precision), rows):
                assert np.abs(a["eigenvalues"] - r["eigenvalues"]).max() < EIG_TOL
    for H, _ in bases:
        H.close()


@pytest.mark.parametrize("name", ["li6_n0", "h3_n2"])
def test_krylov_space_closes(system, name):
    """More steps than the basis has states: the solve ends at the whole basis, with every eigenvalue asked for."""
    d, _, _ = system(name)
    p = oracle.Port(d)
    D = p.dimension
    dense = np.column_stack([p.matvec(np.eye(D)[j]) for j in range(D)])
    p.close()
    w = np.linalg.eigvalsh(0.5 * (dense + dense.T))
    H, mes = _open(system, name, 1, 3)
    r = H.lanczos_batch(mes, max_iterations=100, num_eigenvalues=min(8, D), tolerance=1e-300, precision=64)[0]
    assert r["iterations"] <= D
    assert np.abs(r["eigenvalues"] - w[:len(r["eigenvalues"])]).max() < 1e-9 * np.abs(w).max()
    H.close()
