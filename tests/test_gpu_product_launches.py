"""The products' launches at the sizes where they change: up to 12 288 states one kernel takes max|x| and makes the
views of x (one CTA, a last CTA that is nearly empty, many CTAs), above it two do; and products that follow one another
on a stream, each reading what the one before it wrote while its own kernels are already resident.  Results are the
CPU model's, bit for bit."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn
from .test_gpu_matvec import emu4
from .test_gpu_walk import emu5, set_mode

pytestmark = pytest.mark.gpu

SYSTEMS = {             # Z, N, Nmax, 2M, dimension
    "li6_n0": (3, 3, 0, 2, 8),
    "he4_n4": (2, 2, 4, 0, 952),
    "li7_n4": (3, 4, 4, 1, 10817),
    "li6_n4": (3, 3, 4, 2, 15764),
}
_dirs = {}


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    def get(name):
        if name not in _dirs:
            Z, N, nmax, M2, _ = SYSTEMS[name]
            d = str(tmp_path_factory.mktemp(name))
            jn.generate(d, Z=Z, N=N, nmax=nmax, M2=M2, nbody=2, basis_files=False)
            _dirs[name] = (d, Z, N)
        return _dirs[name]
    return get


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("mode", [1, 64, 32])
def test_walk_launches(system, name, mode):
    import torch
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_engine(5)
    set_mode(H, mode)
    D = H.dimension
    x = np.random.default_rng(5).standard_normal(D)
    for at in (0, D // 2, D - 1):           # the largest state in the first, a middle and the last CTA
        v = x.copy()
        v[at] = -77.0
        assert np.array_equal(H.matvec(v).view(np.uint64), emu5(d, Z, N, v, mode).view(np.uint64))
    assert not H.matvec(np.zeros(D)).any()
    # a chain on one stream: every product reads the previous one's result, scaled back into range
    st = torch.cuda.Stream()
    a, b = torch.from_numpy(x).cuda(), torch.zeros(D, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(6):
            H.matvec_device(a.data_ptr(), b.data_ptr(), False, st.cuda_stream)
            H.matvec_device(b.data_ptr(), a.data_ptr(), False, st.cuda_stream)
            a.mul_(2.0 ** -12)
    st.synchronize()
    want = x
    for _ in range(6):
        want = emu5(d, Z, N, emu5(d, Z, N, want, mode), mode) * 2.0 ** -12
    assert np.array_equal(a.cpu().numpy().view(np.uint64), want.view(np.uint64))
    H.close()


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("mode,n", [(1, 2), (1, 32), (1, 33), (64, 9), (32, 9), (1, 1)])
def test_many_vectors(system, name, mode, n):
    """The products of one subspace call share launches (32 vectors at most): rows and columns of unit vectors show the
    components of H v, which are the single products', bit for bit."""
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_engine(5)
    set_mode(H, mode)
    D = H.dimension
    rng = np.random.default_rng(n)
    at = sorted({0, D // 3, D - 1})
    vs = [rng.standard_normal(D) * 10.0 ** rng.uniform(-4, 4) for _ in range(max(n - len(at), 0))]
    units = [np.eye(1, D, k)[0] for k in at][:n]
    _, op = H.subspace_matrices(vs + units)
    for i, v in enumerate(vs + units):
        hv = H.matvec(v)
        for j in range(max(i, len(vs)), len(vs) + len(units)):
            assert op[i, j] == hv[at[j - len(vs)]]
    H.close()


def test_subspace_workspace(system):
    """The workspace that stays between calls: calls that fit it, outgrow it, and are too large to be kept (68 MB)."""
    d, Z, N = system("li6_n4")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    v = np.random.default_rng(8).standard_normal((270, H.dimension))
    norm, op = H.subspace_matrices(list(v[:5]))
    for n in (40, 5, 270, 3, 5):
        more = H.subspace_matrices(list(v[:n]))
        m = min(n, 5)
        assert np.array_equal(more[0][:m, :m], norm[:m, :m]) and np.array_equal(more[1][:m, :m], op[:m, :m])
    H.close()


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("bits", [32, 64])
def test_panel_launches(system, name, bits):
    """The panel product changes at the same dimension: every CTA takes the maximum below it, one cluster above."""
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_engine(4)
    H.set_precision(bits)
    if H.active_engine() != 4:
        pytest.skip("the FP64 accumulators do not fit")
    D = H.dimension
    x = np.random.default_rng(6).standard_normal(D)
    for at in (0, D // 2, D - 1):
        v = x.copy()
        v[at] = 77.0
        assert np.array_equal(H.matvec(v).view(np.uint64), emu4(d, Z, N, v, bits == 32).view(np.uint64))
    assert not H.matvec(np.zeros(D)).any()
    H.close()


@pytest.mark.parametrize("engine,bits", [(5, 64), (5, 32), (4, 32), (3, 64)])
def test_refused_x_leaves_y(system, engine, bits):
    """x is checked while the product already runs: out of range, y is untouched and the next product is right."""
    d, Z, N = system("he4_n4")
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_engine(engine)
    H.set_precision(bits)
    x = np.random.default_rng(9).standard_normal(H.dimension)
    want = H.matvec(x)
    for bad in (1e300, np.inf, np.nan, 1e-200):
        y = np.arange(H.dimension, dtype=np.float64)
        with pytest.raises(jn.JnError):
            H.matvec(np.full(H.dimension, bad), y)
        assert np.array_equal(y, np.arange(H.dimension))
        assert np.array_equal(H.matvec(x).view(np.uint64), want.view(np.uint64))
    H.close()


@pytest.mark.parametrize("name", ["he4_n4", "li6_n4"])
@pytest.mark.parametrize("engine,bits", [(5, 64), (5, 32), (4, 32)])
def test_products_in_a_caller_graph(system, name, engine, bits):
    """A caller's graph of a copy, two products and a scaling: the products' own overlapped launches join the capture."""
    import torch
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    H.set_engine(engine)
    H.set_precision(bits)
    D = H.dimension
    src = torch.from_numpy(np.random.default_rng(10).standard_normal(D)).cuda()
    a, b, c = (torch.zeros_like(src) for _ in range(3))
    st = torch.cuda.Stream()

    def work():
        a.copy_(src)
        H.matvec_device(a.data_ptr(), b.data_ptr(), False, st.cuda_stream)
        b.mul_(2.0 ** -6)
        H.matvec_device(b.data_ptr(), c.data_ptr(), False, st.cuda_stream)

    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        work()
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        work()
    for k in range(3):
        src.copy_(torch.from_numpy(np.random.default_rng(11 + k).standard_normal(D)))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        want = H.matvec(H.matvec(src.cpu().numpy()) * 2.0 ** -6)
        assert np.array_equal(c.cpu().numpy().view(np.uint64), want.view(np.uint64))
    del g
    H.close()
