"""Row lists of small sectors (kernels/hx_list.cu) and the flips of complete
bases (kernels/hx_flip.cu) against the row kernels, the generic kernel and
the CPU oracle, for every vector type: sectors below one 32-row slice, exact
multiples of it and ragged ones, operators without a diagonal, one with more
coefficient values than the class table holds; flips of one tile and of four,
with state-dependent coefficients, some of them zero."""
import numpy as np
import pytest

import oracle as O
import qkrylov_b200 as qk
from test_gpu_hx import ham, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def all_pairs(n):
    """Distinct couplings on every pair: n (n - 1) / 2 coefficient values."""
    r = np.random.default_rng(n)
    t = []
    for i in range(n):
        for j in range(i + 1, n):
            w = float(r.uniform(0.2, 1.0))
            t += [(w, [("Sz", i), ("Sz", j)]), (0.5 * w, [("Sp", i), ("Sm", j)]), (0.5 * w, [("Sm", i), ("Sp", j)])]
    return t


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 4, dict(use_sz=1, sz2=0), O.heisenberg_chain(4)),                      # 6 rows: part of one slice
    ("spin", 6, {}, O.heisenberg_chain(6)),                                         # 64 rows: two whole slices
    ("spin", 11, dict(use_sz=1, sz2=1), O.heisenberg_chain(11, periodic=False)),    # 462 rows: ragged last slice
    ("spin", 10, {}, [(0.5, [("Sz", i), ("Sz", (i + 1) % 10)]) for i in range(10)] + [(0.7, [("Sx", i)]) for i in range(10)]),
    ("spin", 9, {}, [(0.7, [("Sx", i)]) for i in range(9)]),                        # no diagonal
    ("spin", 12, dict(use_sz=1, sz2=0), all_pairs(12)),                             # 66 values: no lists, row kernel
    ("spin", 11, {}, [(0.5, [("Sz", i), ("Sz", (i + 1) % 11)]) for i in range(11)] + [(0.7, [("Sx", i)]) for i in range(11)]),
    ("spin", 13, {}, [(0.7 + 0.1 * i, [("Sx", i)]) for i in range(13)]),            # flips, no diagonal
    ("spin", 13, {}, [(w, [(o, i), (o, (i + 1) % 13)]) for i in range(13) for o, w in (("Sx", 0.4), ("Sy", 0.4), ("Sz", 0.3))]
     + [(0.2, [("Sx", 3)])]),                                                       # coefficients zero for parallel spins
    ("fermion", 9, dict(use_n=1, n=4), [(-1.0, [("C", (i + 1) % 9), ("Cdag", i)]) for i in range(9)] +
     [(-1.0, [("C", i), ("Cdag", (i + 1) % 9)]) for i in range(9)]),
    ("hubbard", 6, dict(use_nup=1, nup=3, use_ndn=1, ndn=2), O.hubbard_square(3, 2)),
    ("tj", 9, dict(use_nup=1, nup=4, use_ndn=1, ndn=3), O.tj_chain(9)),
])
def test_small_sector_kernels_match_the_others(kind, N, sec, terms):
    H = ham(kind, N, sec, terms)
    ref = O.port().hamiltonian(kind, N, sec, terms)
    rng = np.random.default_rng(N)
    xc = rng.standard_normal(H.dimension) + 1j * rng.standard_normal(H.dimension)
    for code, tdt, tol in [(qk.DTYPE_C128, torch.complex128, 1e-13), (qk.DTYPE_C64, torch.complex64, 2e-6),
                           (qk.DTYPE_F64, torch.float64, 1e-13), (qk.DTYPE_F32, torch.float32, 2e-6)]:
        x = torch.tensor(xc if tdt.is_complex else xc.real, dtype=tdt, device="cuda")
        want = ref.apply(x.cpu().numpy().astype(np.complex128))
        try:
            for pol in ("auto", "no-spin-product", "generic"):
                qk.set_kernel_policy(pol)
                y = torch.full_like(x, float("nan"))
                torch.cuda.synchronize()
                H.apply_device(x.data_ptr(), y.data_ptr(), code)
                torch.cuda.synchronize()
                assert rel(y.cpu().numpy().astype(np.complex128), want) < tol, (pol, code)
        finally:
            qk.set_kernel_policy("auto")


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 7, {}, O.heisenberg_chain(7)),                                         # 128 rows: one whole tile
    ("spin", 9, dict(use_sz=1, sz2=1), O.j1j2_chain(9, 1.0, 0.5)),                  # 126 rows: one ragged tile
    ("spin", 9, {}, [(0.7, [("Sx", i)]) for i in range(9)]),                        # no diagonal; 9 targets a row
    ("tj", 8, dict(use_nup=1, nup=3, use_ndn=1, ndn=3), O.tj_chain(8)),             # 560 rows, 0 to 12 targets
])
@pytest.mark.parametrize("R", [32, 64, 128])
def test_tuned_block_apply_on_small_tiles(kind, N, sec, terms, R):
    """The shape the tuner picks (the packed lists among its candidates) for
    every vector type, with column dots that repeat bit for bit."""
    H = ham(kind, N, sec, terms)
    ref = O.port().hamiltonian(kind, N, sec, terms)
    rng = np.random.default_rng(R + N)
    Xc = rng.standard_normal((H.dimension, R)) + 1j * rng.standard_normal((H.dimension, R))
    for code, tdt, tol in [(qk.DTYPE_C128, torch.complex128, 1e-12), (qk.DTYPE_C64, torch.complex64, 2e-5),
                           (qk.DTYPE_F64, torch.float64, 1e-12), (qk.DTYPE_F32, torch.float32, 2e-5)]:
        X = torch.tensor(Xc if tdt.is_complex else Xc.real, dtype=tdt, device="cuda").contiguous()
        Xh = X.cpu().numpy().astype(np.complex128)
        want = np.stack([ref.apply(np.ascontiguousarray(Xh[:, r])) for r in range(R)], axis=1)
        Y = torch.full_like(X, float("nan"))
        torch.cuda.synchronize()
        H.apply_block_device(X.data_ptr(), Y.data_ptr(), code, R)
        dots = [H.apply_block_device(X.data_ptr(), Y.data_ptr(), code, R, dots=True) for _ in range(2)]
        torch.cuda.synchronize()
        assert rel(Y.cpu().numpy().astype(np.complex128), want) < tol, code
        d = np.einsum("ir,ir->r", Xh.conj(), want)
        got = dots[0][0::2] + 1j * dots[0][1::2]
        assert np.abs(got - d).max() <= 10 * tol * np.abs(d).max() + 1e-300, code
        assert np.array_equal(dots[0], dots[1]), code


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 9, {}, [(0.7, [("Sx", i)]) for i in range(9)]),                        # one warp tile per slice
    ("fermion", 20, dict(use_n=1, n=10), [(-1.0, [(a, (i + 1) % 20), (b, i)]) for i in range(20)
                                          for a, b in (("C", "Cdag"), ("Cdag", "C"))]),  # whole slices
    ("spin", 13, {}, [(0.7, [("Sx", i)]) for i in range(13)]),                      # flips
])
def test_no_diagonal_leaves_infinities_to_the_rows_they_couple_to(kind, N, sec, terms):
    """An operator without a diagonal does not touch a row's own element, as the
    generic kernel does not: an infinite one stays out of that row."""
    H = ham(kind, N, sec, terms)
    for code, tdt in [(qk.DTYPE_F64, torch.float64), (qk.DTYPE_F32, torch.float32), (qk.DTYPE_C128, torch.complex128)]:
        x = torch.ones(H.dimension, dtype=tdt, device="cuda")
        j = H.dimension // 3
        x[j] = float("inf")
        got = {}
        try:
            for pol in ("auto", "generic"):
                qk.set_kernel_policy(pol)
                y = torch.empty_like(x)
                H.apply_device(x.data_ptr(), y.data_ptr(), code)
                torch.cuda.synchronize()
                got[pol] = torch.isfinite(torch.view_as_real(y).sum(-1) if tdt.is_complex else y)
        finally:
            qk.set_kernel_policy("auto")
        assert got["auto"][j] and torch.equal(got["auto"], got["generic"]), (kind, code)
    X = torch.ones(H.dimension, 32, dtype=torch.float64, device="cuda")
    X[j] = float("inf")
    Y = torch.empty_like(X)
    H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F64, 32)
    torch.cuda.synchronize()
    assert torch.equal(torch.isfinite(Y), got["generic"][:, None].expand(-1, 32))


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 7, {}, O.heisenberg_chain(7)),                                         # 128 rows: four whole tiles
    ("spin", 9, dict(use_sz=1, sz2=1), O.j1j2_chain(9, 1.0, 0.5)),                  # 126 rows: ragged last tile
    ("spin", 9, {}, [(0.7, [("Sx", i)]) for i in range(9)]),                        # no diagonal
    ("tj", 8, dict(use_nup=1, nup=3, use_ndn=1, ndn=3), O.tj_chain(8)),             # rows of 0 to 12 targets
])
def test_every_shape_of_the_packed_lists(kind, N, sec, terms):
    H = ham(kind, N, sec, terms)
    ref = O.port().hamiltonian(kind, N, sec, terms)
    rng = np.random.default_rng(N)
    Xc = rng.standard_normal((H.dimension, 128)) + 1j * rng.standard_normal((H.dimension, 128))
    for code, tdt, tol in [(qk.DTYPE_C128, torch.complex128, 1e-12), (qk.DTYPE_C64, torch.complex64, 2e-5),
                           (qk.DTYPE_F64, torch.float64, 1e-12), (qk.DTYPE_F32, torch.float32, 2e-5)]:
        for R in (32, 64, 128):
            X = torch.tensor((Xc if tdt.is_complex else Xc.real)[:, :R], dtype=tdt, device="cuda").contiguous()
            Xh = X.cpu().numpy().astype(np.complex128)
            want = np.stack([ref.apply(np.ascontiguousarray(Xh[:, r])) for r in range(R)], axis=1)
            d = np.einsum("ir,ir->r", Xh.conj(), want)
            for lanes in (32, 16, 8):
                if R // lanes > 8:
                    continue
                Y = torch.full_like(X, float("nan"))
                torch.cuda.synchronize()
                qk.set_kernel_policy("packed-shapes")
                try:
                    dots = H.apply_block_device(X.data_ptr(), Y.data_ptr(), code, R, lanes_per_row=lanes, dots=True)
                finally:
                    qk.set_kernel_policy("auto")
                assert rel(Y.cpu().numpy().astype(np.complex128), want) < tol, (code, R, lanes)
                assert np.abs(dots[0::2] + 1j * dots[1::2] - d).max() <= 10 * tol * np.abs(d).max() + 1e-300, (code, R, lanes)


def test_block_results_do_not_depend_on_what_was_applied_before():
    """Which block kernel runs follows from sizes alone: the same bits from an
    operator whose packed lists another block size has built already."""
    n = 20
    sec, terms = dict(use_sz=1, sz2=0), O.j1j2_chain(n, 1.0, 0.4)
    Hs = [ham("spin", n, sec, terms) for _ in range(3)]
    D = Hs[0].dimension
    X = torch.randn(D, 64, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    x = X[:, :32].float().contiguous()
    ys = []
    for k, H in enumerate(Hs):
        Y, y = torch.empty_like(X), torch.empty_like(x)
        torch.cuda.synchronize()
        if k:
            H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F64, 64)
        H.apply_block_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F32, 32)
        if not k:
            H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F64, 64)
        torch.cuda.synchronize()
        ys.append((Y, y))
    for Y, y in ys[1:]:
        assert torch.equal(Y, ys[0][0]) and torch.equal(y, ys[0][1])


def test_refused_packed_lists_keep_nothing():
    """A sector beyond the lists' 24-bit ranks: tuning its block apply must not
    leave a diagonal (8 bytes per row) behind."""
    n = 27
    H = ham("spin", n, dict(use_sz=1, sz2=1), O.heisenberg_chain(n))
    assert H.dimension > 1 << 24
    before = qk.lib().qkrylov_hamiltonian_device_bytes(H._h)
    X = torch.zeros(H.dimension, 32, dtype=torch.float32, device="cuda")
    Y = torch.empty_like(X)
    torch.cuda.synchronize()
    H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F32, 32)
    torch.cuda.synchronize()
    assert qk.lib().qkrylov_hamiltonian_device_bytes(H._h) == before
