"""What a user of this library runs, as cases to time and to compare.

A program that uses the library opens the files of a Hamiltonian (index lists, matrix elements) and multiplies
vectors by it, one at a time or inside a Lanczos solve; solves many Hamiltonians H(c) = H0 + sum_i c_i H_i of several
bases together; projects the Hamiltonian onto training vectors; turns J-scheme interactions into M-scheme matrix
elements; and fits the small network of the learned warm start.  The cases are those calls, through the public entry
points, on the bases of this repository's tests and benchmark and on others of the same range: dimension 8 to
186 894, two- and two- plus three-body forces, both precisions, odd and even particle numbers.

The problems are synthetic (the library's generator, in the reference's file formats) and are written once per
machine; what changes with the seed is what a program's calls differ in: vectors, couplings, interactions, samples.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import jupiterncsm_gb300 as jn

# A basis and its forces: protons, neutrons, excitation limit, 2 M, two-body (2) or two- plus three-body (3) forces.
SYSTEMS = {
    "li6_nmax0_3nf": (3, 3, 0, 2, 3),       # D = 8
    "h3_nmax2_2nf": (1, 2, 2, 1, 2),        # 41
    "he4_nmax2_2nf": (2, 2, 2, 0, 2),       # 59
    "he4_nmax2_3nf": (2, 2, 2, 0, 3),       # 59
    "li7_nmax2_3nf": (3, 4, 2, 1, 3),       # 264
    "h3_nmax4_3nf": (1, 2, 4, 1, 3),        # 388
    "he6_nmax2_3nf": (2, 4, 2, 0, 3),       # 511
    "li6_nmax2_2nf": (3, 3, 2, 2, 2),       # 711
    "li6_nmax2_3nf": (3, 3, 2, 2, 3),       # 711
    "he4_nmax4_2nf": (2, 2, 4, 0, 2),       # 952
    "he4_nmax4_3nf": (2, 2, 4, 0, 3),       # 952
    "he4_nmax6_2nf": (2, 2, 6, 0, 2),       # 7 916
    "he4_nmax6_3nf": (2, 2, 6, 0, 3),       # 7 916
    "h3_nmax8_2nf": (1, 2, 8, 1, 2),        # 8 294
    "li7_nmax4_2nf": (3, 4, 4, 1, 2),       # 10 817
    "li7_nmax4_3nf": (3, 4, 4, 1, 3),       # 10 817
    "he6_nmax4_3nf": (2, 4, 4, 0, 3),       # 11 658
    "he5_nmax6_2nf": (2, 3, 6, 1, 2),       # 13 162
    "li6_nmax4_2nf": (3, 3, 4, 2, 2),       # 15 764
    "li6_nmax4_3nf": (3, 3, 4, 2, 3),       # 15 764
    "li6_nmax6_3nf": (3, 3, 6, 2, 3),       # 186 894
}
COUPLINGS = 4           # H(c) = H0 + c_1 H_1 + ... + c_4 H_4
OPERATOR_SEED = 20261203


def listed():
    return [
        # One product y = H x on device vectors, as every Lanczos step of a user's own solver takes it.
        # The smallest call: launches and latency are all of it.
        {"name": "product_he4_nmax2_2nf_f64", "kind": "product", "system": "he4_nmax2_2nf", "precision": 64},
        # Ordinary two-body product in 32 bits, of a mixed-precision solve.
        {"name": "product_he4_nmax4_2nf_f32", "kind": "product", "system": "he4_nmax4_2nf", "precision": 32},
        # Ordinary two- plus three-body product in 32 bits (the benchmark's panel workload).
        {"name": "product_he4_nmax6_3nf_f32", "kind": "product", "system": "he4_nmax6_3nf", "precision": 32},
        # The same size in FP64-grade arithmetic, on an odd nucleus: ragged blocks of uneven proton and neutron sides.
        {"name": "product_li7_nmax4_3nf_f64", "kind": "product", "system": "li7_nmax4_3nf", "precision": 64},
        # The largest: the benchmark's headline product.
        {"name": "product_li6_nmax6_3nf_f64", "kind": "product", "system": "li6_nmax6_3nf", "precision": 64},
        # The operator seam of the reference: y += H x on host arrays.
        {"name": "host_product_li6_nmax4_3nf_f64", "kind": "host_product", "system": "li6_nmax4_3nf", "precision": 64},
        # A whole solve: the ten lowest eigenvalues to 1e-6 MeV, convergence tested after every step (the default).
        {"name": "lanczos_he4_nmax6_3nf", "kind": "lanczos", "system": "he4_nmax6_3nf", "precision": 64, "check_every": 1},
        # A whole batch: 64 Hamiltonians on four bases of uneven sizes in one mixed-precision solve.
        {"name": "batch_64_on_four_bases", "kind": "batch", "per_basis": 16, "precision": 32,
         "systems": "he4_nmax2_2nf he4_nmax4_2nf he4_nmax6_2nf li6_nmax4_2nf"},
        # Projection onto 32 training vectors (norm and operator matrices).
        {"name": "subspace_32_li6_nmax4_2nf", "kind": "subspace", "system": "li6_nmax4_2nf", "vectors": 32, "precision": 64},
        # J-scheme to M-scheme, two-body: every block of 6Li Nmax 6 from one interaction.
        {"name": "transform2_li6_nmax6", "kind": "transform2", "Z": 3, "N": 3, "nmax": 6, "M2": 2},
        # J-scheme to M-scheme, three-body: every block of 6Li Nmax 4.
        {"name": "transform3_li6_nmax4", "kind": "transform3", "Z": 3, "N": 3, "nmax": 4, "M2": 0},
        # The warm start's network: created, trained on 256 solves' couplings and coordinates, run on 64 others.
        {"name": "mlp_fit_256", "kind": "mlp", "inputs": 4, "hidden": 128, "outputs": 32, "samples": 256, "held_out": 64,
         "steps": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "host_product", "lanczos", "batch", "subspace", "transform2",
                       "transform3", "mlp"])
    names = [s for s in SYSTEMS if s != "li6_nmax6_3nf"]
    if kind in ("product", "host_product"):
        return {"kind": kind, "system": rng.choice(names if kind == "host_product" else list(SYSTEMS)),
                "precision": rng.choice([64, 32])}
    if kind == "lanczos":
        return {"kind": kind, "system": rng.choice([s for s in names if s.endswith(("4_2nf", "4_3nf", "6_2nf", "2_3nf"))
                                                    and s != "he4_nmax2_3nf"]),
                "precision": rng.choice([64, 32]), "check_every": rng.choice([1, 5, 10])}
    if kind == "batch":
        # smallest basis first, as in the listed batch
        two = ["he4_nmax2_2nf", "li6_nmax2_2nf", "he4_nmax4_2nf", "he4_nmax6_2nf", "li7_nmax4_2nf", "li6_nmax4_2nf"]
        return {"kind": kind, "per_basis": _log_int(rng, 1, 16), "precision": rng.choice([32, 32, 64]),
                "systems": " ".join(two[i] for i in sorted(rng.sample(range(len(two)), rng.randint(1, 3))))}
    if kind == "subspace":
        return {"kind": kind, "system": rng.choice([s for s in names if s.endswith("_2nf")]),
                "vectors": _log_int(rng, 2, 48), "precision": rng.choice([64, 32])}
    if kind in ("transform2", "transform3"):
        Z, N, M2, most = rng.choice([(2, 2, 0, 6), (3, 3, 2, 6), (3, 4, 1, 4), (2, 3, 1, 4)])
        most = min(most, 4) if kind == "transform3" else most
        return {"kind": kind, "Z": Z, "N": N, "nmax": rng.choice(range(2, most + 1, 2)), "M2": M2}
    return {"kind": kind, "inputs": rng.randint(1, 8), "hidden": rng.randint(16, 160), "outputs": rng.randint(4, 40),
            "samples": _log_int(rng, 16, 300), "held_out": _log_int(rng, 1, 100), "steps": _log_int(rng, 50, 800)}


# ---------------------------------------------------------------------------------------------- problems on disk
def _once(name, make):
    """The directory of a generated problem, written once: make(dir) fills it; returns what make returned (texts)."""
    base = os.path.join(tempfile.gettempdir(), f"jupiterncsm_cases_{os.getuid()}")
    d = os.path.join(base, name)
    if not os.path.exists(os.path.join(d, "complete")):
        os.makedirs(base, exist_ok=True)
        part = tempfile.mkdtemp(dir=base)
        with open(os.path.join(part, "complete"), "w") as f:
            f.write(make(part) or "")
        try:
            os.rename(part, d)
        except OSError:                 # another process was first
            shutil.rmtree(part)
    with open(os.path.join(d, "complete")) as f:
        return d, f.read().split()


def _problem(system):
    Z, N, nmax, M2, nbody = SYSTEMS[system]

    def make(d):
        jn.generate(d, Z=Z, N=N, nmax=nmax, M2=M2, nbody=nbody, basis_files=False)
        s = jn.inspect(d, Z, N)
        return " ".join(str(int(s[k])) for k in ("dimension", "list_entries", "me_referenced", "multiply_adds"))

    d, said = _once(system, make)
    return d, Z, N, dict(zip(("D", "entries", "referenced", "multiply_adds"), map(int, said)))


def _family(system):
    """The problem of H0 and the matrix-element directories of H_1 .. H_4 on the same lists."""
    Z, N, nmax, M2, nbody = SYSTEMS[system]
    d, _, _, n = _problem(system)
    more = []
    for i in range(1, COUPLINGS + 1):
        def make(to, i=i):
            jn.generate(to, Z=Z, N=N, nmax=nmax, M2=M2, nbody=nbody, seed=OPERATOR_SEED + 1000 * i, hbar_omega=0.0,
                        basis_files=False)
        more.append(os.path.join(_once(f"{system}_operator{i}", make)[0], "matrix_elements"))
    return d, Z, N, n, more


def _jscheme(case):
    """A combination table with basis files for the J -> M transform of `case`, and its energy limits."""
    three = case["kind"] == "transform3"

    def make(d):
        s = jn.generate(d, Z=case["Z"], N=case["N"], nmax=case["nmax"], M2=case["M2"], nbody=3 if three else 2,
                        antoine=True)
        e3 = jn.three_body_energy(os.path.join(d, "comb.txt")) if three else 0
        return f"{s['emax_single']} {s['emax_pair']} {e3}"

    d, said = _once(f"{case['kind']}_{case['Z']}_{case['N']}_{case['nmax']}_{case['M2']}", make)
    return (d, *map(int, said))


_stream = None


def _one_stream():
    """The stream a program enqueues its products on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _unit(rng, n):
    v = rng.standard_normal(n)
    return v / np.linalg.norm(v)


def _couplings(case, seed):
    """Per basis of a batch: the couplings c of its instances."""
    rng = np.random.default_rng(seed)
    return [rng.uniform(-1.0, 1.0, size=(case["per_basis"], COUPLINGS)) for _ in case["systems"].split()]


def _samples(case, seed):
    """Couplings and smooth coordinates of them, as the snapshots' reduced-basis coordinates are."""
    rng = np.random.default_rng(seed)
    n, k = case["inputs"], case["outputs"]
    x = rng.uniform(-1.7, 1.7, size=(case["samples"] + case["held_out"], n)).astype(np.float32)
    a, b = rng.standard_normal((n, k)) / math.sqrt(n), rng.uniform(-1, 1, size=k)
    t = np.sin(x @ a + b) / np.sqrt(1.0 + np.arange(k))
    return x[:case["samples"]], t[:case["samples"]].astype(np.float32), x[case["samples"]:]


# ---------------------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind in ("product", "host_product", "lanczos", "subspace"):
        d, Z, N, n = _problem(case["system"])
        H = jn.Hamiltonian.from_dir(d, Z, N)
        H.set_precision(case["precision"])
        s = {"case": case, "H": H}
        if kind == "subspace":
            return s | {"vectors": [_unit(rng, H.dimension) for _ in range(case["vectors"])]}
        x = _unit(rng, H.dimension)
        if kind == "lanczos":
            return s | {"start": x}
        H.matvec(np.ones(H.dimension))          # the handle is in use: its plan is laid out
        if kind == "host_product":
            return s | {"x": x, "y": rng.standard_normal(H.dimension)}
        return s | {"x": torch.from_numpy(x).cuda(), "y": torch.empty(H.dimension, dtype=torch.float64, device="cuda"),
                    "stream": _one_stream()}
    if kind == "batch":
        bases = []
        for system, cs in zip(case["systems"].split(), _couplings(case, seed)):
            d, Z, N, _, more = _family(system)
            H = jn.Hamiltonian.from_dir(d, Z, N)
            H.set_precision(case["precision"])
            parts = [H.read_matrix_elements(os.path.join(d, "matrix_elements"))] + [H.read_matrix_elements(m) for m in more]
            bases.append((H, [parts[0] + sum(c[i] * parts[i + 1] for i in range(COUPLINGS)) for c in cs]))
        return {"case": case, "bases": bases}
    if kind == "transform2":
        d, e1, e2, _ = _jscheme(case)
        f = os.path.join(d, f"interaction_{os.getpid()}.bin")
        jn.write_antoine(f, e1, e2, case["Z"] + case["N"], seed=int(seed) + 1)
        T = jn.Transform(os.path.join(d, "comb.txt"), os.path.join(d, "anicr"), case["Z"], case["N"], e1, e2, f)
        os.unlink(f)
        return {"case": case, "T": T, "blocks": _block_ids(T.block, d)}
    if kind == "transform3":
        d, e1, _, e3 = _jscheme(case)
        f = tempfile.mkdtemp(dir=d)
        jn.write_jjj(f, e1, e3, seed=int(seed) + 1)
        T = jn.Transform3(os.path.join(d, "comb.txt"), os.path.join(d, "anicr"), case["Z"], case["N"], e1, f)
        shutil.rmtree(f)
        return {"case": case, "T": T, "blocks": _block_ids(T.block, d)}
    x, t, held_out = _samples(case, seed)
    return {"case": case, "x": x, "t": t, "held_out": held_out, "seed": int(seed)}


def _block_ids(block, d):
    """The ids of a combination table's matrix-element blocks that the transform computes."""
    ids, section = [], ""
    with open(os.path.join(d, "comb.txt")) as f:
        for row in f:
            if "***" in row:
                section = row
            elif "Matrix-elements" in section and "ARRAY:" in row:
                i = int(row.split("ARRAY:")[1].replace("=", " ").split()[0])
                try:
                    block(i)
                    ids.append(i)
                except jn.JnError:
                    pass                # a one-body block, or one of the other transform
    return ids


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product":
        state["H"].matvec_device(state["x"].data_ptr(), state["y"].data_ptr(), stream=state["stream"].cuda_stream)
        return state["y"]
    if kind == "host_product":
        return state["H"].matvec(state["x"], state["y"].copy())
    if kind == "lanczos":
        r = state["H"].lanczos(max_iterations=300, num_eigenvalues=10, tolerance=1e-6, check_every=case["check_every"],
                               start_vector=state["start"], allow_unconverged=True)
        return {"eigenvalues": r["eigenvalues"], "ritz_values": _ritz(case, r["ritz_values"]), "iterations": r["iterations"]}
    if kind == "batch":
        res = jn.lanczos_batch_bases(state["bases"], max_iterations=300, num_eigenvalues=10, tolerance=1e-6,
                                     precision=case["precision"], check_every=10)
        return [{"eigenvalues": np.concatenate([r["eigenvalues"] for r in basis]),
                 "ritz_values": _ritz(case, np.concatenate([r["ritz_values"] for r in basis])),
                 "iterations": np.array([r["iterations"] for r in basis])} for basis in res]
    if kind == "subspace":
        return state["H"].subspace_matrices(state["vectors"])
    if kind in ("transform2", "transform3"):
        state["T"].run()
        return np.concatenate([state["T"].block(i) for i in state["blocks"]])
    m = jn.MLP(case["inputs"], case["hidden"], case["outputs"], seed=state["seed"])
    loss = m.train(state["x"], state["t"], case["steps"])
    out = {"loss": np.float32(loss), "params": m.params(), "predictions": m.predict(state["held_out"])}
    m.close()
    return out


def _ritz(case, values):
    """Ritz values are those of the products' own operator: 32-bit numbers where its elements and vectors are.  (The
    eigenvalues are refined with FP64-grade products at either precision.)"""
    return values.astype(np.float32) if case["precision"] == 32 else values


def _product_work(n, precision, products=1):
    """One product: each index list (12-byte records) and each referenced element once, x in and y out."""
    size = 8 if precision == 64 else 4
    return {"bytes": products * (12.0 * n["entries"] + size * n["referenced"] + 16.0 * n["D"]),
            "flops": products * 2.0 * n["multiply_adds"]}


def work(case):
    kind = case["kind"]
    if kind == "product":
        return _product_work(_problem(case["system"])[3], case["precision"])
    if kind == "host_product":
        n = _problem(case["system"])[3]
        w = _product_work(n, case["precision"])
        return {"bytes": w["bytes"] + 8.0 * n["D"], "flops": w["flops"]}
    if kind in ("lanczos", "batch"):
        bytes_, flops = 0.0, 0.0
        for system in case.get("systems", case.get("system", "")).split():
            n = _problem(system)[3]
            instances = case.get("per_basis", 1)
            # Ten eigenvalues of these operators to 1e-6 MeV take about 110 steps; a step multiplies once (the lists
            # serve all instances of a basis) and orthogonalises against the vectors so far, twice.
            steps = min(n["D"], 110)
            w = _product_work(n, case["precision"])
            lists = 12.0 * n["entries"]
            bytes_ += steps * (lists + instances * (w["bytes"] - lists)) + instances * 8.0 * n["D"] * steps * steps
            flops += instances * (steps * w["flops"] + 4.0 * n["D"] * steps * steps)
        return {"bytes": bytes_, "flops": flops}
    if kind == "subspace":
        n, m = _problem(case["system"])[3], case["vectors"]
        w = _product_work(n, case["precision"], 1)
        return {"bytes": w["bytes"] + 8.0 * n["D"] * m + 16.0 * m * m, "flops": m * w["flops"] + 4.0 * n["D"] * m * m}
    if kind in ("transform2", "transform3"):
        T = prepare(case, 0)["T"]
        st = T.stats()
        T.close()
        # every element is at least one product of a coupled element and a bra coefficient
        return {"bytes": float(st["algorithmic_bytes"]), "flops": 2.0 * st["num_elements"]}
    i, h, o, n = case["inputs"], case["hidden"], case["outputs"], case["samples"]
    weights = i * h + h + h * h + h + h * o + o
    return {"bytes": 4.0 * (n * (i + o) + weights + case["held_out"] * (i + o)),
            "flops": 6.0 * weights * n * case["steps"] + 2.0 * weights * case["held_out"]}


# ---------------------------------------------------------------------------------------------- 64-bit results
class _Exact:
    """The Hamiltonian of a problem directory, read from its files: products and the dense matrix in 64 bits."""

    def __init__(self, d, me_dirs=None, weights=(1.0,)):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        me_dirs = me_dirs or [os.path.join(d, "matrix_elements")]
        self.np, self.nn, self.off, self.type, D, section = {}, {}, {}, {}, 0, ""
        with open(os.path.join(d, "comb.txt")) as f:
            for row in f:
                if "***" in row:
                    section = row
                elif "mp-states" in section and "ARRAYMP:" in row:
                    w = row.split()
                    b = int(row.split("ARRAYMP:")[1].split("=")[0])
                    self.np[b], self.nn[b], self.off[b] = int(w[4]), int(w[5]), D
                    D += int(w[4]) * int(w[5])
                elif "Conn lists" in section and "ARRAY:" in row:
                    self.type[int(row.split("ARRAY:")[1].split("=")[0])] = row.split()[0][0]
        self.D, self.rows, lists, self.me = D, [], {}, {}
        with open(os.path.join(d, "evaluation_order.txt")) as f:
            for row in f:
                if "BLOCK:" in row and "UNLOAD_" not in row:
                    w = [int(v) for v in row.split("BLOCK:")[1].split()]
                    self.rows.append((w[0], w[1], w[2:-1], w[-1]))
        for _, _, ls, me in self.rows:
            for i in ls:
                if i not in lists:
                    e = np.fromfile(os.path.join(d, "index_lists", f"index_list_{i}"), dtype=np.int32).reshape(-1, 3)
                    lists[i] = (e[:, 0].astype(np.int64), e[:, 1].astype(np.int64),
                                (e[:, 2] & 0x7FFFFFFF).astype(np.int64), np.where(e[:, 2] < 0, -1.0, 1.0))
            if me not in self.me:
                total, nd = 0.0, 0
                for c, m in zip(weights, me_dirs):
                    raw = np.fromfile(os.path.join(m, f"{me}_matrix_elements"), dtype=np.int64, count=1)
                    nd = int(raw[0])
                    total = total + c * np.fromfile(os.path.join(m, f"{me}_matrix_elements"), dtype=np.float64, offset=16)
                self.me[me] = (nd, torch.from_numpy(total).to(self.dev))
        self.lists = {i: tuple(torch.from_numpy(v).to(self.dev) for v in e) for i, e in lists.items()}

    def terms(self):
        """Per instruction: element values, their (output, input) positions in the full vector, and whether diagonal."""
        for bi, bo, ls, me in self.rows:
            nd, M = self.me[me]
            if len(ls) == 2:
                ln, lp = (ls[0], ls[1]) if self.type[ls[0]] == "n" else (ls[1], ls[0])
                n_in, n_out, kn, sn = self.lists[ln]
                p_in, p_out, kp, sp = self.lists[lp]
                v = M[(kp * nd)[:, None] + kn[None, :]] * (sp[:, None] * sn[None, :])
                i = (p_in * self.nn[bi])[:, None] + n_in[None, :]
                o = (p_out * self.nn[bo])[:, None] + n_out[None, :]
            else:
                s_in, s_out, k, sg = self.lists[ls[0]]
                m = M[k]
                m = torch.where(m.abs() < 1e-12, torch.zeros_like(m), m) * sg
                if self.type[ls[0]] == "n":
                    q = torch.arange(self.np[bi], device=self.dev)
                    i = s_in[:, None] + (q * self.nn[bi])[None, :]
                    o = s_out[:, None] + (q * self.nn[bo])[None, :]
                else:
                    q = torch.arange(self.nn[bi], device=self.dev)
                    i = (s_in * self.nn[bi])[:, None] + q[None, :]
                    o = (s_out * self.nn[bo])[:, None] + q[None, :]
                v = m[:, None].expand_as(i)
            yield v.reshape(-1), (o + self.off[bo]).reshape(-1), (i + self.off[bi]).reshape(-1), bi == bo

    def matvec(self, x):
        """H X for the columns of x (D x n)."""
        x = torch.as_tensor(x, dtype=torch.float64, device=self.dev)
        y = torch.zeros_like(x)
        for v, o, i, diag in self.terms():
            y.index_add_(0, o, v[:, None] * x[i])
            if not diag:
                y.index_add_(0, i, v[:, None] * x[o])
        return y

    def dense(self):
        h = torch.zeros(self.D * self.D, dtype=torch.float64, device=self.dev)
        for v, o, i, diag in self.terms():
            h.index_add_(0, o * self.D + i, v)
            if not diag:
                h.index_add_(0, i * self.D + o, v)
        return h.reshape(self.D, self.D)

    def lowest(self, n):
        return torch.linalg.eigvalsh(self.dense())[:n].cpu().numpy()


def _exact_mlp(case, seed):
    """The fit in 64 bits: the seeded initial weights, full-batch Adam, the predictions."""
    n_in, h, n_out = case["inputs"], case["hidden"], case["outputs"]
    mask, z = (1 << 64) - 1, int(seed) & ((1 << 64) - 1)

    def uniform(count, fan_in):
        nonlocal z
        out = np.empty(count, dtype=np.float32)
        for k in range(count):
            z = (z + 0x9E3779B97F4A7C15) & mask
            v = z
            v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & mask
            v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & mask
            v ^= v >> 31
            out[k] = ((v >> 11) * 2.0 ** -53 * 2.0 - 1.0) / math.sqrt(fan_in)
        return torch.from_numpy(out.astype(np.float64))

    w1, w2 = uniform(h * n_in, n_in).reshape(h, n_in), uniform(h * h, h).reshape(h, h)
    w3 = uniform(n_out * h, h).reshape(n_out, h)
    p = [w1, torch.zeros(h, dtype=torch.float64), w2, torch.zeros(h, dtype=torch.float64), w3,
         torch.zeros(n_out, dtype=torch.float64)]
    p = [t.clone().requires_grad_() for t in p]
    x, t, held_out = (torch.from_numpy(a.astype(np.float64)) for a in _samples(case, seed))

    def forward(a):
        a = torch.nn.functional.gelu(a @ p[0].T + p[1])
        a = torch.nn.functional.gelu(a @ p[2].T + p[3])
        return a @ p[4].T + p[5]

    opt = torch.optim.Adam(p, lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
    for _ in range(case["steps"]):
        opt.zero_grad()
        (((forward(x) - t) ** 2).sum() / (2 * len(x))).backward()
        opt.step()
    with torch.no_grad():
        loss = float(((forward(x) - t) ** 2).sum() / (2 * len(x)))
        return {"loss": np.float64(loss), "params": torch.cat([q.reshape(-1) for q in p]).numpy(),
                "predictions": forward(held_out).numpy()}


def exact(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind in ("product", "host_product", "subspace"):
        e = _Exact(_problem(case["system"])[0])
        if kind == "subspace":
            v = torch.from_numpy(np.stack([_unit(rng, e.D) for _ in range(case["vectors"])])).to(e.dev)
            norm, op = v @ v.T, torch.cat([e.matvec(c.T) for c in v.split(4)], 1).T @ v.T
            return norm.cpu().numpy(), ((op + op.T) / 2).cpu().numpy()
        y = e.matvec(_unit(rng, e.D)[:, None])[:, 0].cpu().numpy()
        return y if kind == "product" else y + rng.standard_normal(e.D)
    if kind == "lanczos":
        e = _Exact(_problem(case["system"])[0])
        return {"eigenvalues": e.lowest(10), "ritz_values": None, "iterations": None} if e.D <= 8000 else None
    if kind == "batch":
        out = []
        for system, cs in zip(case["systems"].split(), _couplings(case, seed)):
            d, _, _, n, more = _family(system)
            low = None
            if n["D"] <= 1000:          # larger ones would take minutes
                dirs = [os.path.join(d, "matrix_elements")] + more
                low = np.concatenate([_Exact(d, dirs, (1.0, *c)).lowest(10) for c in cs])
            out.append({"eigenvalues": low, "ritz_values": None, "iterations": None})
        return out
    if kind in ("transform2", "transform3"):
        return None                     # the dense transform of these takes minutes in numpy
    return _exact_mlp(case, seed)
