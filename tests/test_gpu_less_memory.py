"""Solves on a machine with less memory (native/failing_allocations.cpp, preloaded into a child process)."""
import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = os.path.join(ROOT, "tests", "_build", "libfailing_allocations.so")
pytestmark = pytest.mark.gpu


def _child(body, *args):
    head = """
        import ctypes, sys
        import numpy as np
        sys.path.insert(0, sys.argv[1])
        import jupiterncsm_gb300 as jn
        fa = ctypes.CDLL(None)
        fa.fa_budget.argtypes = [ctypes.c_size_t]
        fa.fa_peak.restype = ctypes.c_size_t
        fa.fa_refused.restype = fa.fa_calls.restype = ctypes.c_long
        fa.fa_new.argtypes = [ctypes.c_char_p, ctypes.c_long]
        ALL = ctypes.c_size_t(-1).value
    """
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(head) + textwrap.dedent(body), ROOT, *map(str, args)],
                       env=dict(os.environ, LD_PRELOAD=SHIM), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("precision", [32, 64])
def test_refinement_takes_the_memory_there_is(problem, precision):
    """The refinement multiplies as many vectors at a time as fit beside the solve's own: with memory for half of them,
    and for one, the bits are the same; with memory for none it fails, and the next solve is right."""
    d, Z, N, *_ = problem("he4_n4_2b")
    _child("""
        d, Z, N, precision = sys.argv[2], int(sys.argv[3]), int(sys.argv[4]), int(sys.argv[5])
        H = jn.Hamiltonian.from_dir(d, Z, N)
        me = H.read_matrix_elements(d + "/matrix_elements")
        B, r = 8, 14
        mes = [(1 + 0.01 * i) * me for i in range(B)]
        run = lambda: H.lanczos_batch(mes, max_iterations=40, num_eigenvalues=10, tolerance=1e-300, precision=precision)
        bits = lambda rows: np.concatenate([np.concatenate([q["eigenvalues"], q["residual_norms"]]) for q in rows])
        want = bits(run())
        fa.fa_budget(ALL)
        assert np.array_equal(bits(run()), want)
        peak, vector = fa.fa_peak(), 16 * B * H.dimension      # of the refinement, with all r vectors at a time
        for vectors in (r // 2, 1):
            fa.fa_budget(peak - (r - vectors) * vector + 4096)
            assert np.array_equal(bits(run()), want)
            assert fa.fa_refused() > 0
        fa.fa_budget(peak - r * vector)
        try:
            run()
            raise SystemExit("a solve without memory for a vector succeeded")
        except jn.JnError as e:
            assert e.status == 5, e
        fa.fa_budget(ALL)
        assert np.array_equal(bits(run()), want)
    """, d, Z, N, precision)


def test_no_host_memory_is_an_error(problem):
    """An allocation of the library's C++ containers fails: the call returns an error, and the next one is right."""
    d, Z, N, *_ = problem("he4_n4_2b")
    d2, Z2, N2, *_ = problem("he4_n2_2b")
    _child("""
        d, Z, N, d2, Z2, N2 = sys.argv[2], int(sys.argv[3]), int(sys.argv[4]), sys.argv[5], int(sys.argv[6]), int(sys.argv[7])
        bases = []
        for q, z, n in ((d, Z, N), (d2, Z2, N2)):
            H = jn.Hamiltonian.from_dir(q, z, n)
            me = H.read_matrix_elements(q + "/matrix_elements")
            bases.append((H, [me, 1.5 * me, 2.0 * me]))
        H, mes = bases[0]
        net = jn.MLP(3, 10, 4)
        x, t = np.ones((5, 3), np.float32), np.ones((5, 4), np.float32)

        def lanczos():
            r = H.lanczos(max_iterations=40, num_eigenvalues=4, mode=jn.LANCZOS_REFERENCE, tolerance=1e-3,
                          converge_eigenvectors=True, allow_unconverged=True)
            return r["eigenvalues"]

        def batch(precision, bases):
            def call():
                # uneven convergence: the instances' CTAs are shared out anew on the way
                res = jn.lanczos_batch_bases(bases, max_iterations=200, num_eigenvalues=4, tolerance=1e-6, precision=precision,
                                             check_every=5)
                return np.concatenate([r["eigenvalues"] for rows in res for r in rows])
            return call

        def one_basis():
            return np.concatenate([r["eigenvalues"] for r in H.lanczos_batch(mes, max_iterations=200, num_eigenvalues=4, tolerance=1e-6)])

        def train():
            net.set_params(np.linspace(-1, 1, net.num_params, dtype=np.float32))
            return net.loss_and_gradient(x, t)[1], net.train(x, t, 0)

        for call, some in ((lanczos, 1), (batch(32, bases), 10), (batch(64, bases), 2), (one_basis, 10), (train, 0)):
            want = call()
            fa.fa_new(b"libjncsm_gpu.so", 0)
            call()
            total = fa.fa_calls()
            assert total >= some, total
            # the first twenty, the last, and some between
            for n in sorted({*range(1, min(20, total) + 1), *(int(v) for v in np.geomspace(1, max(total, 1), 20)), total} - {0}):
                if n > total:
                    continue
                fa.fa_new(b"libjncsm_gpu.so", n)
                try:
                    call()
                    raise SystemExit(f"allocation {n} of {total} did not fail the call")
                except jn.JnError as e:
                    assert e.status == 5, e
                fa.fa_new(b"", 0)
                assert all(np.array_equal(a, b) for a, b in zip(call(), want))
            fa.fa_new(b"", 0)
    """, d, Z, N, d2, Z2, N2)
