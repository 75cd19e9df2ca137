"""A Lanczos run that converges needs no more vectors than one stopped there."""
import ctypes

import pytest

import oracle as O
import qkrylov_b200 as qk
from test_gpu_hx import ham

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_converged_run_fits_where_a_stopped_one_does():
    """The next step's vector is made while the host checks for convergence:
    with the GPU's memory taken, a run that ends there must not fail for it."""
    n = 26
    H = ham("spin", n, dict(use_sz=1, sz2=0), O.heisenberg_chain(n))  # 83 MB per vector
    m = qk.lanczos_fp64(H, seed=1, tol=1e-4).iterations_high
    hold = []
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # the library's pool, emptied, keeps what the run stopped at step m needs ...
    rt = ctypes.CDLL(f"libcudart.so.{torch.version.cuda.split('.')[0]}")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
    stopped = qk.lanczos_fp64(H, seed=1, tol=1e-4, maxiter=m)
    # ... and everything else goes, but for less than a vector
    try:
        for size in (1 << 30, 1 << 28, 1 << 26, 1 << 24):
            while torch.cuda.mem_get_info()[0] > size + (24 << 20):
                try:
                    hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        assert torch.cuda.mem_get_info()[0] < 8 * H.dimension
        free = qk.lanczos_fp64(H, seed=1, tol=1e-4)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert free.iterations_high == stopped.iterations_high == m and free.energy == stopped.energy
