"""The grouped row kernel (kernels/hx_group.cu) against the CPU oracle for
every vector type, through apply_operator (one-shot operators keep no row
lists, so small sectors reach it): groups of one to four blocks, classes of
fewer and more than 32 positions, several coefficient classes, no and many
crossing bonds, blocks without high bonds, fused dots, and row ranges."""
import ctypes

import numpy as np
import pytest

import oracle as O
import qkrylov_b200 as qk
from test_compiler import SITES, opsum
from test_gpu_hx import ham, rel
from test_sector_tables import make_basis

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HOPS = [(-1.0, [("C", (i + 1) % 13), ("Cdag", i)]) for i in range(13)] + \
       [(-1.0, [("C", i), ("Cdag", (i + 1) % 13)]) for i in range(13)]


@pytest.mark.parametrize("kind,N,sec,terms", [
    ("spin", 5, dict(use_sz=1, sz2=1), O.heisenberg_chain(5)),                       # 10 rows
    ("spin", 13, dict(use_sz=1, sz2=1), O.heisenberg_chain(13, periodic=False)),     # one crossing bond, ragged classes
    ("spin", 14, dict(use_sz=1, sz2=4), O.j1j2_chain(14, 1.0, 0.3)),                 # two coefficients, six crossing bonds
    ("spin", 12, {}, O.heisenberg_chain(12)),                                        # complete basis: one class
    ("spin", 10, dict(use_sz=1, sz2=0), [(1.0, [("Sp", 0), ("Sm", 1)]), (1.0, [("Sm", 0), ("Sp", 1)])]),  # low bonds only
    ("spin", 10, dict(use_sz=1, sz2=0), [(0.5, [("Sp", 8), ("Sm", 9)]), (0.5, [("Sm", 8), ("Sp", 9)])]),  # high bonds only
    ("fermion", 13, dict(use_n=1, n=6), HOPS),
    ("tj", 10, dict(use_nup=1, nup=4, use_ndn=1, ndn=4), O.tj_chain(10)),
    ("tj", 6, {}, O.tj_chain(6)),
])
def test_grouped_rows_match_the_oracle(kind, N, sec, terms):
    ref = O.port().hamiltonian(kind, N, sec, terms)
    basis, site, ops = make_basis(kind, N, sec), SITES[kind](), opsum(terms)
    rng = np.random.default_rng(N)
    xc = rng.standard_normal(ref.dim) + 1j * rng.standard_normal(ref.dim)
    for tdt, tol in [(torch.complex128, 1e-13), (torch.complex64, 2e-6), (torch.float64, 1e-13), (torch.float32, 2e-6)]:
        x = torch.tensor(xc if tdt.is_complex else xc.real, dtype=tdt, device="cuda")
        xh = x.cpu().numpy().astype(np.complex128)
        want = ref.apply(xh)
        torch.cuda.synchronize()
        y = qk.apply_operator(basis, site, ops, x)
        assert rel(y.cpu().numpy().astype(np.complex128), want) < tol, tdt
        y, e = qk.apply_operator(basis, site, ops, x, expectation=True)
        assert rel(y.cpu().numpy().astype(np.complex128), want) < tol, tdt
        assert abs(e - np.vdot(xh, want)) < 10 * tol * np.linalg.norm(xh) * np.linalg.norm(want), tdt


def test_grouped_rows_ignore_infinities_they_do_not_couple_to():
    """Loads beyond a block's entries and of invalid crossing rows are not
    added: an infinite element of x reaches only the rows H couples it to and
    its own (whose diagonal, zero included, is always applied)."""
    terms, sec = O.j1j2_chain(12, 1.0, 0.3), dict(use_sz=1, sz2=0)
    ref = O.port().hamiltonian("spin", 12, sec, terms)
    basis, site, ops = make_basis("spin", 12, sec), SITES["spin"](), opsum(terms)
    for j in (0, 17, 401, ref.dim - 1):
        unit = np.zeros(ref.dim, np.complex128)
        unit[j] = 1.0
        coupled = np.abs(ref.apply(unit)) > 0
        coupled[j] = True
        for tdt in (torch.float64, torch.float32):
            x = torch.ones(ref.dim, dtype=tdt, device="cuda")
            x[j] = float("inf")
            torch.cuda.synchronize()
            y = qk.apply_operator(basis, site, ops, x).cpu().numpy()
            assert np.isfinite(y[~coupled]).all(), (j, tdt)


def test_grouped_rows_ranges_reassemble():
    """Shards of a sector above the row lists' size equal the whole apply."""
    B = make_basis("spin", 24, dict(use_sz=1, sz2=0))
    H = ham("spin", 24, dict(use_sz=1, sz2=0), O.heisenberg_chain(24))
    x = torch.randn(H.dimension, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    whole = torch.empty_like(x)
    torch.cuda.synchronize()
    H.apply_device(x.data_ptr(), whole.data_ptr(), qk.DTYPE_F64)
    b = np.zeros(4, np.uint64)
    assert qk.lib().qkrylov_b200_basis_shard_bounds(B._h, 3, b.ctypes.data_as(ctypes.c_void_p)) == 0
    y = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    for k in range(3):
        assert qk.lib().qkrylov_hamiltonian_apply_range_device(
            H._h, qk.DTYPE_F64, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()), int(b[k]), int(b[k + 1]), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(y, whole)
