"""The number of kernels that the library says a product launches, against the kernel nodes of a captured product."""
import ctypes

import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu
# below and above the dimension (12 288) from which max|x| and the copies of x are kernels of their own; one kind of
# particle (no proton walks, so no transposed view of x)
SYSTEMS = {"he4_n4": (2, 2, 4, 0, 2), "li6_n4": (3, 3, 4, 2, 2), "h3_n8": (1, 2, 8, 1, 2), "n3_n4": (0, 3, 4, 1, 2),
           "n4_n8": (0, 4, 8, 0, 2)}
KERNEL_NODE = 0


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    dirs = {}

    def get(name):
        if name not in dirs:
            Z, N, nmax, M2, nbody = SYSTEMS[name]
            dirs[name] = str(tmp_path_factory.mktemp(name))
            jn.generate(dirs[name], Z=Z, N=N, nmax=nmax, M2=M2, nbody=nbody, basis_files=False)
        return dirs[name], SYSTEMS[name][0], SYSTEMS[name][1]
    return get


def _captured_kernels(H, x, y, stream):
    import torch
    cuda = ctypes.CDLL("libcuda.so.1")
    cuda.cuStreamBeginCapture_v2.argtypes = [ctypes.c_void_p, ctypes.c_int]
    cuda.cuStreamEndCapture.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    cuda.cuGraphGetNodes.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.POINTER(ctypes.c_size_t)]
    cuda.cuGraphNodeGetType.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_int)]
    cuda.cuGraphDestroy.argtypes = [ctypes.c_void_p]
    H.matvec_device(x.data_ptr(), y.data_ptr(), False, stream.cuda_stream)      # plans and copies are made
    torch.cuda.synchronize()
    graph, n, kind = ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_int()
    assert cuda.cuStreamBeginCapture_v2(stream.cuda_stream, 1) == 0
    H.matvec_device(x.data_ptr(), y.data_ptr(), False, stream.cuda_stream)
    assert cuda.cuStreamEndCapture(stream.cuda_stream, ctypes.byref(graph)) == 0
    assert cuda.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cuda.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    count = 0
    for node in nodes:
        assert cuda.cuGraphNodeGetType(node, ctypes.byref(kind)) == 0
        count += kind.value == KERNEL_NODE
    cuda.cuGraphDestroy(graph)
    return count


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("engine,bits,fp64_fma", [(5, 64, False), (5, 64, True), (5, 32, False), (4, 64, False), (4, 32, False),
                                                  (3, 64, False), (3, 32, False), (2, 64, False), (2, 32, False)])
def test_kernels_of_a_product(system, name, engine, bits, fp64_fma):
    import torch
    d, Z, N = system(name)
    H = jn.Hamiltonian.from_dir(d, Z, N)
    try:
        H.set_engine(engine)
    except jn.JnError:
        H.close()
        pytest.skip("the basis is too large for this engine")
    H.set_precision(bits)
    if engine == 5:
        H.set_walk_arithmetic(fp64_fma)
    x = torch.from_numpy(np.random.default_rng(2).standard_normal(H.dimension)).cuda()
    y = torch.zeros_like(x)
    st = torch.cuda.Stream()
    assert H.product_kernels() == _captured_kernels(H, x, y, st)
    H.close()
