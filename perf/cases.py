"""Workloads whose time is tracked: the calls a user of the framework makes.

The framework's work is y = H x, matrix-free, on one vector or on a block of
vectors, and the Krylov solvers around it.  The cases are therefore H x over
the model families, sector sizes and vector types (the inner call of every
user-written Krylov or time-evolution loop), the block form (batched FTLM,
coupling sweeps, block fractions), and two whole solver calls.

Kinds of case
  apply    MatrixFreeHamiltonian.apply_device on vectors in GPU memory
  block    MatrixFreeHamiltonian.apply_block_device on row-interleaved blocks
           (float64: with the column dots, as the recurrences use it)
  ftlm     ftlm_block, the whole batched finite-temperature Lanczos
  lanczos  lanczos_ground_state from a start vector, the reference's solver

Models: "heisenberg" (periodic or open chain, any Sz), "j1j2" (periodic
chain), "tfim" (transverse-field Ising chain, full basis), "tj" (periodic t-J
chain), "hubbard" (periodic lx x ly lattice; ly = 1 is a chain).
"""
import functools
import math

import numpy as np
import torch

import qkrylov_b200 as qk

DTYPES = {
    "complex128": (torch.complex128, qk.DTYPE_C128, 16),
    "complex64": (torch.complex64, qk.DTYPE_C64, 8),
    "float64": (torch.float64, qk.DTYPE_F64, 8),
    "float32": (torch.float32, qk.DTYPE_F32, 4),
}


def listed():
    return [
        # the smallest call: tutorials, tests and small-sector scans; launch latency
        dict(name="hx heisenberg n16 c128", kind="apply", model="heisenberg", n=16, sz2=0, periodic=True,
             dtype="complex128"),
        # an ordinary single-precision sector, next-nearest bonds (coupling scans)
        dict(name="hx j1j2 n24 f32", kind="apply", model="j1j2", n=24, sz2=0, j2=0.4, dtype="float32"),
        # odd chain, open ends, Sz = 1/2: ragged blocks
        dict(name="hx open n25 f64", kind="apply", model="heisenberg", n=25, sz2=1, periodic=False, dtype="float64"),
        # the headline workload: complex128 Heisenberg ring at half filling
        dict(name="hx heisenberg n28 c128", kind="apply", model="heisenberg", n=28, sz2=0, periodic=True,
             dtype="complex128"),
        # doped t-J ring: the two-part tables
        dict(name="hx tj n20 f64", kind="apply", model="tj", n=20, nup=9, ndn=9, dtype="float64"),
        # odd Hubbard ring, unequal spin counts, complex vectors (dynamics of a doped chain)
        dict(name="hx hubbard n13 c64", kind="apply", model="hubbard", lx=13, ly=1, nup=6, ndn=7, dtype="complex64"),
        # the largest sector in use: the 4x4 Hubbard torus at half filling
        dict(name="hx hubbard 4x4 f64", kind="apply", model="hubbard", lx=4, ly=4, nup=8, ndn=8, dtype="float64"),
        # an operator without a conserved charge, in the reference's default type
        dict(name="hx tfim n20 c64", kind="apply", model="tfim", n=20, dtype="complex64"),
        # block apply of the batched FTLM (single-precision vectors)
        dict(name="block tj n18 r64 f32", kind="block", model="tj", n=18, nup=8, ndn=8, R=64, dtype="float32"),
        # block apply of the coupling sweep (double precision, fused dots)
        dict(name="block j1j2 n24 r32 f64", kind="block", model="j1j2", n=24, sz2=0, j2=0.4, R=32, dtype="float64"),
        # a whole finite-temperature run
        dict(name="ftlm tj n14 r64", kind="ftlm", model="tj", n=14, nup=6, ndn=6, R=64, steps=100, temps=200),
        # a whole ground-state run through the reference's API, host vectors
        dict(name="lanczos heisenberg n22", kind="lanczos", model="heisenberg", n=22, sz2=0, periodic=True, steps=40),
    ]


def draw(rng):
    """One more case of the same ranges.  Sector dimensions grow
    exponentially with the sites, so drawing the sites evenly spreads the
    sizes evenly over their logarithm."""
    kind = rng.choice(["apply"] * 7 + ["block"] * 3 + ["ftlm", "lanczos"])
    dtype = rng.choice(sorted(DTYPES))
    if kind == "apply":
        model = rng.choice(["heisenberg", "heisenberg", "j1j2", "tj", "hubbard", "tfim"])
        if model == "heisenberg":
            n = rng.randint(14, 28)
            return dict(kind=kind, model=model, n=n, sz2=n % 2 + 2 * rng.randint(0, 2), periodic=rng.random() < 0.7,
                        dtype=dtype)
        if model == "j1j2":
            n = rng.randint(14, 26)
            return dict(kind=kind, model=model, n=n, sz2=n % 2 + 2 * rng.randint(0, 1),
                        j2=round(rng.uniform(0.1, 0.9), 3), dtype=dtype)
        if model == "tj":
            n, holes = rng.randint(10, 20), rng.randint(1, 3)
            nup = (n - holes) // 2
            return dict(kind=kind, model=model, n=n, nup=nup, ndn=n - holes - nup, dtype=dtype)
        if model == "hubbard":
            lx, ly = rng.choice([(7, 1), (8, 1), (9, 1), (10, 1), (11, 1), (12, 1), (13, 1), (14, 1), (4, 2), (5, 2),
                                 (3, 3), (4, 3), (7, 2)])
            n = lx * ly
            return dict(kind=kind, model=model, lx=lx, ly=ly, nup=n // 2, ndn=n // 2 - rng.randint(0, 1), dtype=dtype)
        return dict(kind=kind, model=model, n=rng.randint(11, 22), dtype=dtype)
    if kind == "block":
        dtype = rng.choice(["float32", "float64"])
        R = rng.choice([32, 64, 128])
        if rng.random() < 0.5:
            n, holes = rng.randint(10, 17), rng.randint(1, 3)
            nup = (n - holes) // 2
            return dict(kind=kind, model="tj", n=n, nup=nup, ndn=n - holes - nup, R=R, dtype=dtype)
        n = rng.randint(14, 23)
        return dict(kind=kind, model="j1j2", n=n, sz2=n % 2, j2=round(rng.uniform(0.1, 0.9), 3), R=R, dtype=dtype)
    if kind == "ftlm":
        n = rng.randint(10, 13)
        nup = (n - 2) // 2
        return dict(kind=kind, model="tj", n=n, nup=nup, ndn=n - 2 - nup, R=rng.choice([32, 64]),
                    steps=rng.randint(30, 100), temps=rng.randint(20, 200))
    n = rng.randint(15, 22)
    return dict(kind=kind, model="heisenberg", n=n, sz2=n % 2, periodic=rng.random() < 0.7, steps=rng.randint(15, 32))


# ------------------------------------------------------------------- models
def bonds(c):
    """(i, j, J) of a spin chain's exchange bonds, or (i, j, 1) of a lattice's."""
    m = c["model"]
    if m == "hubbard":
        lx, ly = c["lx"], c["ly"]
        out = []
        for y in range(ly):
            for x in range(lx):
                i = x + lx * y
                for j in sorted({(x + 1) % lx + lx * y, x + lx * ((y + 1) % ly)} - {i}):
                    out.append((i, j, 1.0))
        return out
    n = c["n"]
    if m == "j1j2":
        return [(i, (i + d) % n, J) for d, J in ((1, 1.0), (2, c["j2"])) for i in range(n)]
    return [(i, (i + 1) % n, 1.0) for i in range(n if c.get("periodic", True) else n - 1)]


HOP, EXCHANGE, REPULSION, FIELD = 1.0, 0.4, 4.0, 0.7


def operator_key(c):
    return tuple(sorted((k, v) for k, v in c.items() if k in ("model", "n", "sz2", "periodic", "j2", "nup", "ndn",
                                                              "lx", "ly")))


@functools.lru_cache(maxsize=2)
def hamiltonian(key):
    """The operator handle a program builds once and applies many times."""
    c = dict(key)
    m = c["model"]
    ops = qk.OpSum(dtype=np.float64)
    if m in ("heisenberg", "j1j2"):
        for i, j, J in bonds(c):
            ops.add_term(J, "Sz", i, "Sz", j)
            ops.add_term(0.5 * J, "Sp", i, "Sm", j)
            ops.add_term(0.5 * J, "Sm", i, "Sp", j)
        basis, site = qk.SpinHalfBasis(c["n"], sz=c["sz2"] / 2, dtype=np.float64), qk.SpinHalfSite()
    elif m == "tfim":
        for i, j, _ in bonds(c):
            ops.add_term(1.0, "Sz", i, "Sz", j)
        for i in range(c["n"]):
            ops.add_term(FIELD, "Sx", i)
        basis, site = qk.SpinHalfBasis(c["n"], dtype=np.float64), qk.SpinHalfSite()
    else:
        for i, j, _ in bonds(c):
            for a, b in ((i, j), (j, i)):
                ops.add_term(-HOP, "CUp", b, "CdagUp", a)
                ops.add_term(-HOP, "CDn", b, "CdagDn", a)
        if m == "hubbard":
            for i in range(c["lx"] * c["ly"]):
                ops.add_term(REPULSION, "Nupdn", i)
            basis, site = qk.HubbardBasis(c["lx"] * c["ly"], nup=c["nup"], ndn=c["ndn"]), qk.HubbardSite()
        else:
            for i, j, _ in bonds(c):
                ops.add_term(-0.5 * EXCHANGE, "Nup", i, "Ndn", j)
                ops.add_term(-0.5 * EXCHANGE, "Ndn", i, "Nup", j)
                ops.add_term(0.5 * EXCHANGE, "CUp", j, "CdagDn", j, "CDn", i, "CdagUp", i)
                ops.add_term(0.5 * EXCHANGE, "CUp", i, "CdagDn", i, "CDn", j, "CdagUp", j)
            basis, site = qk.TJBasis(c["n"], nup=c["nup"], ndn=c["ndn"]), qk.TJSite()
    return qk.MatrixFreeHamiltonian(basis, site, ops, dtype=np.float64)


def dimension(c):
    m = c["model"]
    if m in ("heisenberg", "j1j2"):
        return math.comb(c["n"], (c["n"] + c["sz2"]) // 2)
    if m == "tfim":
        return 1 << c["n"]
    if m == "hubbard":
        return math.comb(c["lx"] * c["ly"], c["nup"]) * math.comb(c["lx"] * c["ly"], c["ndn"])
    return math.comb(c["n"], c["nup"]) * math.comb(c["n"] - c["nup"], c["ndn"])


# ------------------------------------------------------------ prepare and run
def vectors(c, seed, dim):
    """Random vectors of unit norm (the Krylov vectors of a solver), (dim,) or (dim, R)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (dim, c["R"]) if c["kind"] == "block" else (dim,)
    x = torch.randn(shape, dtype=DTYPES[c["dtype"]][0], device="cuda", generator=g)
    return x.div_(math.sqrt(dim))


def prepare(case, seed):
    H = hamiltonian(operator_key(case))
    s = dict(case=case, H=H)
    if case["kind"] in ("apply", "block"):
        s["x"] = vectors(case, seed, H.dimension)
        s["y"] = torch.empty_like(s["x"])
    elif case["kind"] == "ftlm":
        s["T"] = np.geomspace(0.1, 20.0, case["temps"])
        s["seed"] = seed
    else:
        s["start"] = lanczos_start(H.dimension, seed)
    return s


def lanczos_start(dim, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(dim) + 1j * r.standard_normal(dim)


def run(state):
    c, H = state["case"], state["H"]
    if c["kind"] == "apply":
        H.apply_device(state["x"].data_ptr(), state["y"].data_ptr(), DTYPES[c["dtype"]][1])
        return state["y"]
    if c["kind"] == "block":
        dots = H.apply_block_device(state["x"].data_ptr(), state["y"].data_ptr(), DTYPES[c["dtype"]][1], c["R"],
                                    dots=c["dtype"] == "float64")
        return [state["y"], dots]
    if c["kind"] == "ftlm":
        r = qk.ftlm_block(H, state["T"], n_random=c["R"], n_steps=c["steps"], seed=state["seed"], precision=64)
        return [r.logZ, r.U, r.Cv]
    r = qk.lanczos_ground_state(H, maxiter=c["steps"], start=state["start"])
    return [r.energy, r.eigenvector, r.alphas, r.betas]


def work(case):
    """Bytes: every vector a pass reads once plus every vector it writes once
    (a solver's steps depend on one another, so each streams its vectors).
    Flops: two per real component and nonzero of H."""
    dim, m = dimension(case), case["model"]
    per_row = {"heisenberg": 0.5, "j1j2": 0.5, "tfim": 0.0, "tj": 1.0, "hubbard": 1.0}[m] * len(bonds(case)) + 1
    if m == "tfim":
        per_row += case["n"]
    if case["kind"] in ("apply", "block"):
        R, es = case.get("R", 1), DTYPES[case["dtype"]][2]
        comp = 2 if case["dtype"].startswith("complex") else 1
        return {"bytes": 2.0 * dim * R * es, "flops": 2.0 * dim * R * comp * per_row}
    if case["kind"] == "ftlm":
        n = dim * case["R"] * case["steps"]
        return {"bytes": 3.0 * n * 8, "flops": 2.0 * n * per_row}
    k = case["steps"]  # step j reads its j + 1 stored vectors twice (projections, then update) and writes one
    return {"bytes": 16.0 * dim * (k * (k + 1) + 2 * k), "flops": 4.0 * dim * (k * per_row + 2 * k * (k + 1))}


# --------------------------------------------------------------------- exact
def popcount(v):
    c = torch.zeros_like(v)
    for b in range(44):
        c += (v >> b) & 1
    return c


def spread(v, n):
    out = torch.zeros_like(v)
    for b in range(n):
        out |= ((v >> b) & 1) << (2 * b)
    return out


def basis_states(c, dev):
    """The sector's states in ascending order."""
    def subsets(n, k):
        parts = []
        for lo in range(0, 1 << n, 1 << 24):
            v = torch.arange(lo, min(lo + (1 << 24), 1 << n), dtype=torch.int64, device=dev)
            parts.append(v[popcount(v) == k])
        return torch.cat(parts)

    m = c["model"]
    if m == "tfim":
        return torch.arange(1 << c["n"], dtype=torch.int64, device=dev)
    if m in ("heisenberg", "j1j2"):
        return subsets(c["n"], (c["n"] + c["sz2"]) // 2)
    n = c["n"] if m == "tj" else c["lx"] * c["ly"]
    u, d = subsets(n, c["nup"]), subsets(n, c["ndn"])
    parts = []
    for k in range(0, len(u), 2048):
        w = u[k:k + 2048, None]
        s = spread(w, n) | (spread(d, n) << 1)[None, :]
        parts.append(s[(w & d[None, :]) == 0] if m == "tj" else s.reshape(-1))
    return torch.cat(parts).sort().values


class Plain:
    """H X by its definition: masks and ranks of the sorted states, 64-bit sums."""

    def __init__(self, c, dev):
        self.c, self.s = c, basis_states(c, dev)
        n = c.get("n") or c["lx"] * c["ly"]
        bits = n if c["model"] in ("heisenberg", "j1j2", "tfim") else 2 * n
        self.table = None
        if bits <= 32:  # the rank of every state by one lookup
            self.table = torch.zeros(1 << bits, dtype=torch.int32, device=dev)
            self.table[self.s] = torch.arange(len(self.s), dtype=torch.int32, device=dev)

    def rank(self, t):
        return self.table[t].long() if self.table is not None else torch.searchsorted(self.s, t)

    def __call__(self, X):
        Y = torch.empty_like(X)
        step = max(1, (1 << 24) // (X.shape[1] if X.dim() > 1 else 1))
        for lo in range(0, len(self.s), step):
            Y[lo:lo + step] = self.rows(self.s[lo:lo + step], X, lo)
        return Y

    def rows(self, s, X, lo):
        c, m = self.c, self.c["model"]
        x0 = X[lo:lo + len(s)]
        shape = (-1,) + (1,) * (X.dim() - 1)

        def bit(b):
            return (s >> b) & 1

        diag = torch.zeros(len(s), dtype=torch.float64, device=s.device)
        acc = torch.zeros_like(x0)

        def add(on, target, value):
            at = on.nonzero().squeeze(1)
            v = value[at] if torch.is_tensor(value) else torch.full((len(at),), value, dtype=torch.float64, device=s.device)
            acc.index_add_(0, at, v.reshape(shape).to(X.dtype) * X[self.rank(target[at])])

        for i, j, J in bonds(c):
            if m in ("heisenberg", "j1j2", "tfim"):
                anti = bit(i) != bit(j)
                diag += (0.25 - 0.5 * anti.double()) * J
                if m != "tfim":
                    add(anti, s ^ ((1 << i) | (1 << j)), 0.5 * J)
                continue
            for sp in (0, 1):
                a, b = 2 * i + sp, 2 * j + sp
                on = bit(a) != bit(b)
                if m == "tj":  # the site hopped to is empty
                    on = on & ((bit(a ^ 1) + bit(b ^ 1)) == 0)
                p, q = min(a, b), max(a, b)
                between = ((1 << q) - 1) & ~((1 << (p + 1)) - 1)
                sign = 1.0 - 2.0 * (popcount(s & between) & 1).double()
                add(on, s ^ ((1 << a) | (1 << b)), -HOP * sign)
            if m == "tj":
                ui, di, uj, dj = (bit(k) for k in (2 * i, 2 * i + 1, 2 * j, 2 * j + 1))
                anti = ((ui & dj) | (di & uj)) == 1
                diag -= (0.5 * EXCHANGE) * anti.double()
                add(anti, s ^ ((3 << (2 * i)) | (3 << (2 * j))), 0.5 * EXCHANGE)
        if m == "hubbard":
            for i in range(c["lx"] * c["ly"]):
                diag += REPULSION * (bit(2 * i) & bit(2 * i + 1)).double()
        if m == "tfim":
            everywhere = torch.ones(len(s), dtype=torch.bool, device=s.device)
            for i in range(c["n"]):
                add(everywhere, s ^ (1 << i), 0.5 * FIELD)
        return acc + diag.reshape(shape).to(X.dtype) * x0


def exact(case, seed):
    if case["kind"] == "ftlm":
        return None  # its random vectors come from the framework's own generator
    P = Plain(case, "cuda" if torch.cuda.is_available() else "cpu")
    dim = dimension(case)
    if case["kind"] in ("apply", "block"):
        x = vectors(case, seed, dim)
        x = x.to(torch.complex128 if x.is_complex() else torch.float64)
        y = P(x)
        if case["kind"] == "apply":
            return y
        if case["dtype"] != "float64":
            return [y, None]
        dots = np.zeros(2 * case["R"])
        dots[0::2] = (x * y).sum(0).cpu().numpy()
        return [y, dots]
    # Lanczos with full reorthogonalisation; the Ritz vector's sign is free, so it has no exact value
    v = torch.from_numpy(lanczos_start(dim, seed)).to(P.s.device)
    V, alphas, betas = [v / v.norm()], [], []
    for k in range(case["steps"]):
        w = P(V[-1])
        alphas.append(float(torch.vdot(V[-1], w).real))
        for _ in range(2):
            B = torch.stack(V)
            w = w - (B.conj() @ w) @ B
        if k + 1 < case["steps"]:
            betas.append(float(w.norm()))
            V.append(w / betas[-1])
    T = np.diag(alphas) + np.diag(betas, 1) + np.diag(betas, -1)
    return [float(np.linalg.eigvalsh(T)[0]), None, np.array(alphas), np.array(betas)]
