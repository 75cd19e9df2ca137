"""Kernels behind the sizes that reach them by default: operators created under
the 'no-spin-product' policy build no row lists, so small sectors run on the
grouped row kernel (kernels/hx_group.cu), with and without the per-die queues,
whole and by row ranges; larger lists (kernels/hx_list.cu, more slices than are
resident at once) against the CPU oracle; complex operators on the generic one."""
import ctypes

import numpy as np
import pytest

import oracle as O
import qkrylov_b200 as qk
from test_gpu_grouped_rows import HOPS
from test_gpu_hx import ham, rel
from test_sector_tables import make_basis

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TYPES = [(qk.DTYPE_C128, torch.complex128, 1e-13), (qk.DTYPE_C64, torch.complex64, 2e-6),
         (qk.DTYPE_F64, torch.float64, 1e-13), (qk.DTYPE_F32, torch.float32, 2e-6)]


def ham_without_lists(kind, N, sec, terms):
    qk.set_kernel_policy("no-spin-product")
    try:
        return ham(kind, N, sec, terms)
    finally:
        qk.set_kernel_policy("auto")


def vectors(H, tdt):
    g = torch.Generator("cuda").manual_seed(H.dimension % 1000)
    x = torch.randn(H.dimension, dtype=tdt, device="cuda", generator=g)
    return x, torch.full_like(x, float("nan"))


def apply(H, x, y, code, policy="auto"):
    torch.cuda.synchronize()
    qk.set_kernel_policy(policy)
    try:
        H.apply_device(x.data_ptr(), y.data_ptr(), code)
    finally:
        qk.set_kernel_policy("auto")
    torch.cuda.synchronize()
    return y


def shards(H, basis, x, code, n):
    b = np.zeros(n + 1, np.uint64)
    assert qk.lib().qkrylov_b200_basis_shard_bounds(basis._h, n, b.ctypes.data_as(ctypes.c_void_p)) == 0
    y = torch.full_like(x, float("nan"))
    for k in range(n):
        assert qk.lib().qkrylov_hamiltonian_apply_range_device(
            H._h, code, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()), int(b[k]), int(b[k + 1]), None) == 0
    torch.cuda.synchronize()
    return y


SMALL = [
    ("spin", 5, dict(use_sz=1, sz2=1), O.heisenberg_chain(5)),                       # 10 rows
    ("spin", 13, dict(use_sz=1, sz2=1), O.heisenberg_chain(13, periodic=False)),     # one crossing bond, ragged classes
    ("spin", 14, dict(use_sz=1, sz2=4), O.j1j2_chain(14, 1.0, 0.3)),                 # two coefficients, six crossing bonds
    ("spin", 12, {}, O.heisenberg_chain(12)),                                        # complete basis: one class
    ("spin", 10, dict(use_sz=1, sz2=0), [(1.0, [("Sp", 0), ("Sm", 1)]), (1.0, [("Sm", 0), ("Sp", 1)])]),  # low bonds only
    ("spin", 10, dict(use_sz=1, sz2=0), [(0.5, [("Sp", 8), ("Sm", 9)]), (0.5, [("Sm", 8), ("Sp", 9)])]),  # high bonds only
    ("fermion", 13, dict(use_n=1, n=6), HOPS),
    ("tj", 10, dict(use_nup=1, nup=4, use_ndn=1, ndn=4), O.tj_chain(10)),
    ("tj", 6, {}, O.tj_chain(6)),
]


@pytest.mark.parametrize("kind,N,sec,terms", SMALL)
def test_grouped_rows_on_small_sectors(kind, N, sec, terms):
    """Against the oracle; the queue order, the grid-stride order and shards of
    the rows give the same bits, also on repeated launches (the queues reset)."""
    H, basis = ham_without_lists(kind, N, sec, terms), make_basis(kind, N, sec)
    ref = O.port().hamiltonian(kind, N, sec, terms)
    for code, tdt, tol in TYPES:
        x, y = vectors(H, tdt)
        apply(H, x, y, code)
        want = ref.apply(x.cpu().numpy().astype(np.complex128))
        assert rel(y.cpu().numpy().astype(np.complex128), want) < tol, tdt
        for policy in ("auto", "no-die-queues", "auto"):
            assert torch.equal(apply(H, x, torch.full_like(x, float("nan")), code, policy), y), (tdt, policy)
        for n in (2, 5):
            assert torch.equal(shards(H, basis, x, code, n), y), (tdt, n)


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 24, dict(use_sz=1, sz2=0), O.heisenberg_chain(24)),
    ("tj", 18, dict(use_nup=1, nup=8, use_ndn=1, ndn=8), O.tj_chain(18)),
])
def test_per_die_queues_and_shards_above_the_lists(kind, N, sec, terms):
    H, basis = ham(kind, N, sec, terms), make_basis(kind, N, sec)
    for code, tdt, tol in TYPES:
        x, y = vectors(H, tdt)
        apply(H, x, y, code)
        for policy in ("no-die-queues", "auto"):
            assert torch.equal(apply(H, x, torch.full_like(x, float("nan")), code, policy), y), (tdt, policy)
        assert torch.equal(shards(H, basis, x, code, 3), y), tdt
        g = apply(H, x, torch.empty_like(x), code, "generic")
        assert float((g - y).abs().max() / g.abs().max()) < tol, tdt


def test_shards_of_a_complex_operator():
    """A complex coefficient: the generic kernel, whole and by ranges."""
    sec, terms = dict(use_sz=1, sz2=0), O.heisenberg_chain(14) + [(0.3j, [("Sp", 0), ("Sm", 2)]), (-0.3j, [("Sm", 0), ("Sp", 2)])]
    H, basis = ham("spin", 14, sec, terms), make_basis("spin", 14, sec)
    ref = O.port().hamiltonian("spin", 14, sec, terms)
    for code, tdt, tol in TYPES[:2]:
        x, y = vectors(H, tdt)
        apply(H, x, y, code)
        assert rel(y.cpu().numpy().astype(np.complex128), ref.apply(x.cpu().numpy().astype(np.complex128))) < tol, tdt
        assert torch.equal(shards(H, basis, x, code, 4), y), tdt


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 19, dict(use_sz=1, sz2=1), O.j1j2_chain(19, 1.0, 0.3)),                 # 92,378 rows: ragged last slice
    ("tj", 14, dict(use_nup=1, nup=6, use_ndn=1, ndn=6), O.tj_chain(14)),
    ("hubbard", 9, dict(use_nup=1, nup=4, use_ndn=1, ndn=5), O.hubbard_square(3, 3)),  # 15,876 rows: resident at once
    ("hubbard", 11, dict(use_nup=1, nup=5, use_ndn=1, ndn=5), O.hubbard_square(11, 1)),
])
def test_larger_row_lists(kind, N, sec, terms):
    H, basis = ham(kind, N, sec, terms), make_basis(kind, N, sec)
    ref = O.port().hamiltonian(kind, N, sec, terms)
    for code, tdt, tol in TYPES:
        x, y = vectors(H, tdt)
        apply(H, x, y, code)
        want = ref.apply(x.cpu().numpy().astype(np.complex128))
        assert rel(y.cpu().numpy().astype(np.complex128), want) < tol, tdt
        assert torch.equal(shards(H, basis, x, code, 3), y), tdt
