"""The spin-product kernels (kernels/hx_pair.cu) against the CPU oracle for
every vector type, through apply_operator (one-shot operators keep no row
lists, so small sectors reach these kernels): sectors below one 32-row tile,
odd row lengths (rows not 16-byte aligned), one species empty or full, rows
that fill tiles exactly, unequal counts, and hops of one, few and many
amplitudes."""
import numpy as np
import pytest

import oracle as O
import qkrylov_b200 as qk
from test_compiler import SITES, opsum
from test_gpu_hx import rel
from test_sector_tables import make_basis

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def magnitudes(n, k):
    """A ring whose bond (i, i + 1) hops with the (i mod k)-th of k amplitudes."""
    t = []
    for i in range(n):
        j = (i + 1) % n
        w = -(1.0 + 0.25 * (i % k))
        for a, b in ((i, j), (j, i)):
            t += [(w, [("CUp", b), ("CdagUp", a)]), (w, [("CDn", b), ("CdagDn", a)])]
    return t + [(3.0, [("Nupdn", i)]) for i in range(n)]


@pytest.mark.parametrize("N,nup,ndn,terms", [
    (7, 3, 4, O.hubbard_square(7, 1, 1.0, 4.0)),     # 35 x 35
    (9, 4, 5, O.hubbard_square(3, 3, 1.0, 4.0)),     # 126 x 126, signs within a species
    (8, 4, 2, O.hubbard_square(4, 2, 1.0, 4.0)),     # 70 x 28
    (6, 0, 3, O.hubbard_square(3, 2, 1.0, 4.0)),     # 1 x 20
    (6, 6, 5, O.hubbard_square(3, 2, 1.0, 4.0)),     # 1 x 6
    (9, 2, 7, O.hubbard_square(9, 1, 1.0, 4.0)),     # 36 x 36
    (11, 5, 6, O.hubbard_square(11, 1, 1.0, 4.0)),   # 462 x 462
    (8, 4, 4, magnitudes(8, 3)),                     # three hop amplitudes
    (9, 5, 4, magnitudes(9, 9)),                     # nine: more than the slot tables hold
    (8, 3, 4, O.hubbard_square(2, 4, 1.0, 4.0)),     # doubled bonds: two amplitudes
])
def test_spin_product_kernels_match_the_oracle(N, nup, ndn, terms):
    sec = dict(use_nup=1, nup=nup, use_ndn=1, ndn=ndn)
    ref = O.port().hamiltonian("hubbard", N, sec, terms)
    basis, site, ops = make_basis("hubbard", N, sec), SITES["hubbard"](), opsum(terms)
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
