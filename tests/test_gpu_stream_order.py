"""Ordering of device-pointer calls with other streams: every call without a
stream starts after what the default stream holds (not only the first of its
vector type), for each entry point, and leaves a capture on another stream
alone."""
import ctypes

import numpy as np
import pytest

import oracle as O
import qkrylov_b200 as qk
from qkrylov_b200 import sharded
from test_gpu_hx import ham, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N, SEC, TERMS = 14, dict(use_sz=1, sz2=0), O.heisenberg_chain(14)


@pytest.fixture(scope="module")
def case():
    H = ham("spin", N, SEC, TERMS)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(H.dimension)
    return H, x, O.port().hamiltonian("spin", N, SEC, TERMS).apply(x.astype(np.complex128)).real


def busy():
    """Some milliseconds of work on the current stream."""
    a = torch.ones(4096, 4096, device="cuda")
    for _ in range(8):
        a = a @ a * 1e-4
    return a


@pytest.mark.parametrize("entry", ["apply", "range", "block", "diagonal", "multi_dot"])
def test_calls_without_a_stream_follow_the_default_stream(case, entry):
    H, xh, want = case
    src = torch.tensor(xh, device="cuda")
    D = H.dimension
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    if entry == "block":
        X, Y = (torch.zeros(D, 32, dtype=torch.float64, device="cuda") for _ in range(2))
        H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F64, 32)  # tunes
    for _ in range(4):
        shape = (D, 32) if entry == "block" else (D,)
        x = torch.full(shape, 9.0, dtype=torch.float64, device="cuda")
        y = torch.full(shape, 9.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        keep = busy()
        x.copy_(src[:, None].expand(D, 32) if entry == "block" else src)
        y.fill_(float("nan"))
        if entry == "apply":
            H.apply_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F64)
        elif entry == "range":
            assert qk.lib().qkrylov_hamiltonian_apply_range_device(H._h, qk.DTYPE_F64, ptr(x), ptr(y), 0, D, None) == 0
        elif entry == "block":
            H.apply_block_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F64, 32)
        elif entry == "diagonal":
            assert qk.lib().qkrylov_hamiltonian_diagonal_device(H._h, qk.DTYPE_F64, ptr(y), None) == 0
        else:
            out = np.zeros(2)
            V = (ctypes.c_void_p * 1)(x.data_ptr())
            assert qk.lib().qkrylov_b200_multi_dot(0, qk.DTYPE_F64, D, 1, V, ptr(x), out.ctypes.data) == 0
            assert abs(out[0] - xh @ xh) < 1e-12 * (xh @ xh)
        torch.cuda.synchronize()
        del keep
        got = y.cpu().numpy()
        if entry == "diagonal":
            assert np.array_equal(got, H.diagonal().real)
        elif entry == "block":
            assert rel(got, np.repeat(want[:, None], 32, axis=1)) < 1e-13
        elif entry != "multi_dot":
            assert rel(got, want) < 1e-13


def test_device_start_vectors_follow_the_default_stream(case):
    """Solvers whose start vectors are the caller's device memory."""
    H, xh, _ = case
    src = torch.tensor(xh, device="cuda")
    blk = torch.randn(H.dimension, 32, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    torch.cuda.synchronize()
    x, X = src.clone(), blk.clone()
    torch.cuda.synchronize()
    want = qk.lanczos_fp64(H, start_device=x.data_ptr(), maxiter=5, tol=1e-3)
    cf = qk.cf_block(H, X.data_ptr(), 6, n_vectors=32)
    for _ in range(2):
        x, X = torch.zeros_like(src), torch.zeros_like(blk)
        torch.cuda.synchronize()
        keep = busy()
        x.copy_(src)
        got = qk.lanczos_fp64(H, start_device=x.data_ptr(), maxiter=5, tol=1e-3)
        assert got.energy == want.energy
        keep = busy()
        X.copy_(blk)
        r = qk.cf_block(H, X.data_ptr(), 6, n_vectors=32)
        torch.cuda.synchronize()
        del keep
        assert all(np.array_equal(p.alphas, q.alphas) for p, q in zip(r, cf))


def test_range_hook_follows_the_current_stream(case):
    """The sharded Lanczos' range apply on a stream other than the default one."""
    H, xh, want = case
    src = torch.tensor(xh, device="cuda")
    apply_rows = sharded.gpu_apply_rows(H, qk.DTYPE_F64)
    x = torch.empty_like(src)
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(torch.cuda.Stream()):
        for k in (1.0, 2.0, 3.0):
            keep = busy()
            torch.mul(src, k, out=x)
            got.append(apply_rows(x, 0, H.dimension).clone())
    torch.cuda.synchronize()
    del keep
    for k, y in zip((1.0, 2.0, 3.0), got):
        assert rel(y.cpu().numpy(), k * want) < 1e-13, k


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_a_capture_on_another_stream_survives(case, mode):
    """Calls without a stream, on an operator that has been applied before and
    on a new vector type, while another stream is in capture."""
    H, xh, want = case
    x = torch.tensor(xh, device="cuda")
    x32, y32 = x.float(), torch.empty(len(xh), dtype=torch.float32, device="cuda")
    y, z = torch.empty_like(x), torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        z.add_(1.0)
        H.apply_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F64)
        H.apply_device(x32.data_ptr(), y32.data_ptr(), qk.DTYPE_F32)
    g.replay()
    torch.cuda.synchronize()
    assert (z == 1.0).all() and rel(y.cpu().numpy(), want) < 1e-13 and rel(y32.cpu().numpy(), want) < 2e-6
    g.reset()


def test_a_capture_on_a_blocking_stream_survives(case):
    """The default stream cannot be named while a stream that synchronises with
    it is in capture: the call goes ahead and the capture stays valid."""
    H, xh, want = case
    x = torch.tensor(xh, device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    rt = ctypes.CDLL(f"libcudart.so.{torch.version.cuda.split('.')[0]}")
    s, g = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(s)) == 0
    assert rt.cudaStreamBeginCapture(s, 1) == 0
    H.apply_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F64)
    assert rt.cudaStreamEndCapture(s, ctypes.byref(g)) == 0 and g.value
    assert rt.cudaGraphDestroy(g) == 0 and rt.cudaStreamDestroy(s) == 0
    torch.cuda.synchronize()
    assert rel(y.cpu().numpy(), want) < 1e-13


@pytest.mark.parametrize("kind,n,sec,terms", [
    ("spin", 24, dict(use_sz=1, sz2=0), O.heisenberg_chain(24)),                    # grouped rows: work queues
    ("tj", 18, dict(use_nup=1, nup=8, use_ndn=1, ndn=8), O.tj_chain(18)),           # the same, two-part
    ("hubbard", 13, dict(use_nup=1, nup=6, use_ndn=1, ndn=7), O.hubbard_square(13, 1)),  # product-ordered scratch
])
def test_applies_of_one_operator_on_several_streams(kind, n, sec, terms):
    """Sectors above the row lists' size, whose kernels keep queues or scratch
    in the operator: applies issued in turn on three streams without waiting."""
    H = ham(kind, n, sec, terms)
    g = torch.Generator("cuda").manual_seed(n)
    xs = [torch.randn(H.dimension, dtype=torch.float64, device="cuda", generator=g) for _ in range(6)]
    want = [torch.empty_like(x) for x in xs]
    ys = [torch.full_like(x, float("nan")) for x in xs]
    for x, w in zip(xs, want):
        H.apply_device(x.data_ptr(), w.data_ptr(), qk.DTYPE_F64)
        torch.cuda.synchronize()
    streams = [0, torch.cuda.Stream().cuda_stream, torch.cuda.Stream().cuda_stream]
    for rep in range(3):
        for k, (x, y) in enumerate(zip(xs, ys)):
            H.apply_device(x.data_ptr(), y.data_ptr(), qk.DTYPE_F64, stream=streams[(k + rep) % 3])
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want)), rep
        for y in ys:
            y.fill_(float("nan"))
        torch.cuda.synchronize()


@pytest.mark.parametrize("kind,n,sec,terms", [
    ("tj", 14, dict(use_nup=1, nup=6, use_ndn=1, ndn=6), O.tj_chain(14)),
    ("spin", 16, {}, [(0.5, [("Sz", i), ("Sz", (i + 1) % 16)]) for i in range(16)] + [(0.7, [("Sx", i)]) for i in range(16)]),
])
def test_block_applies_of_one_operator_on_several_streams(kind, n, sec, terms):
    H = ham(kind, n, sec, terms)
    g = torch.Generator("cuda").manual_seed(n)
    Xs = [torch.randn(H.dimension, 64, dtype=torch.float64, device="cuda", generator=g) for _ in range(4)]
    want = [torch.empty_like(X) for X in Xs]
    Ys = [torch.full_like(X, float("nan")) for X in Xs]
    torch.cuda.synchronize()
    for X, W in zip(Xs, want):
        H.apply_block_device(X.data_ptr(), W.data_ptr(), qk.DTYPE_F64, 64)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream().cuda_stream, 0, torch.cuda.Stream().cuda_stream]
    for rep in range(3):
        for k, (X, Y) in enumerate(zip(Xs, Ys)):
            H.apply_block_device(X.data_ptr(), Y.data_ptr(), qk.DTYPE_F64, 64, stream=streams[(k + rep) % 3])
        torch.cuda.synchronize()
        assert all(torch.equal(Y, W) for Y, W in zip(Ys, want)), rep
        for Y in Ys:
            Y.fill_(float("nan"))
        torch.cuda.synchronize()


@pytest.mark.parametrize("route", ["lists", "groups", "flips", "spin-product", "block"])
def test_applies_can_be_captured_and_replayed(route):
    """One apply per kernel family captured on a caller's stream (after a first
    call outside the capture), replayed on new contents of x; calls without a
    stream go on beside the capture."""
    kind, n, sec, terms = {
        "lists": ("spin", 14, dict(use_sz=1, sz2=0), O.heisenberg_chain(14)),
        "groups": ("spin", 24, dict(use_sz=1, sz2=0), O.heisenberg_chain(24)),
        "flips": ("spin", 13, {}, [(0.7, [("Sx", i)]) for i in range(13)]),
        "spin-product": ("hubbard", 13, dict(use_nup=1, nup=6, use_ndn=1, ndn=6), O.hubbard_square(13, 1)),
        "block": ("tj", 12, dict(use_nup=1, nup=5, use_ndn=1, ndn=5), O.tj_chain(12)),
    }[route]
    H = ham(kind, n, sec, terms)
    shape = (H.dimension, 32) if route == "block" else (H.dimension,)
    g = torch.Generator("cuda").manual_seed(n)
    xs = [torch.randn(shape, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    x, y, z = xs[0].clone(), torch.empty(shape, dtype=torch.float64, device="cuda"), torch.empty(shape, dtype=torch.float64, device="cuda")

    def call(a, b, stream=0):
        if route == "block":
            H.apply_block_device(a.data_ptr(), b.data_ptr(), qk.DTYPE_F64, 32, stream=stream)
        else:
            H.apply_device(a.data_ptr(), b.data_ptr(), qk.DTYPE_F64, stream=stream)

    want = []
    for v in xs:
        call(v, z)
        torch.cuda.synchronize()
        want.append(z.clone())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(x, y, torch.cuda.current_stream().cuda_stream)
        call(xs[1], z)  # not part of the graph
    torch.cuda.synchronize()
    assert torch.equal(z, want[1])
    for v, w in zip(xs, want):
        x.copy_(v)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, w), route
    graph.reset()
