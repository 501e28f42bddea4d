"""Device memory of the library: freed memory is kept for the next allocation
up to a bound, and memory a caller borrowed from a handle is not handed to
anyone else before the caller's pending work on it is done."""
import ctypes
import gc
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


# 1 GiB arrays are the driver's own, 32 MiB ones cut from slabs, of which 1 GiB
# is kept
@pytest.mark.parametrize("log2n, kept", [(27, 0), (22, 1 << 30)])
def test_freed_memory_is_given_back_above_the_bound(log2n, kept):
    rb.ParVector(1)
    rb.synchronize()
    gc.collect()
    before = torch.cuda.mem_get_info()[0]
    big = [rb.ParVector(1 << log2n) for _ in range(6 << (27 - log2n))]   # 6 GiB
    rb.synchronize()
    assert torch.cuda.mem_get_info()[0] < before - (5 << 30)
    del big
    gc.collect()
    rb.synchronize()
    # (and the driver's own granularity)
    assert torch.cuda.mem_get_info()[0] > before - kept - (256 << 20)


def test_the_pool_keeps_at_most_2_gib():
    """Block matrices of 32 MiB (their addresses are not given out: pool
    memory), with a handle alive throughout, so that nothing else is given
    back."""
    b, nnz = 16, (4 << 20) // 256
    vals = np.ones((nnz, b, b))
    rowptr, cols = np.arange(nnz + 1, dtype=np.int32), np.zeros(nnz, np.int32)
    alive = rb.ParVector(1)
    rb.synchronize()
    gc.collect()
    before = torch.cuda.mem_get_info()[0]
    big = [rb.BSRMatrix.from_arrays(nnz, 1, b, b, rowptr, cols, vals) for _ in range(112)]   # 3.5 GiB
    assert torch.cuda.mem_get_info()[0] < before - (2 << 30)
    del big
    gc.collect()
    rb.synchronize()
    assert torch.cuda.mem_get_info()[0] > before - (2 << 30) - (256 << 20)
    del alive


def _ipc_capable(ptr):
    """Whether cudaIpcGetMemHandle takes the address (a query only)."""
    from cuda.bindings import driver

    attr = driver.CUpointer_attribute.CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE
    err, capable = driver.cuPointerGetAttribute(attr, int(ptr))
    assert err == driver.CUresult.CUDA_SUCCESS, err
    return bool(capable)


def test_addresses_given_out_can_be_shared_between_processes():
    """Vectors and matrices of every origin and of sizes on both sides of the
    pool's and the slabs' limits lie in memory of cudaMalloc, which other
    processes (CUDA IPC) and other devices (peer access) can be given."""
    for n in (1, 31, 1000, 1 << 16, (1 << 22) - 1, 1 << 22, 1 << 23):
        assert _ipc_capable(rb.ParVector(n).device_ptr()), n
    A = rb.par_stencil_grid(rb.diffusion_stencil_2d(0.1, 0.4), [40, 40])
    n = A.global_num_rows
    S = A.strength(rb.Classical, 0.25)
    ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, rb.Jacobi)
    ml.setup(A)
    blocks = rb.BSRMatrix.from_arrays(1, 1, 2, 2, [0, 1], [0], np.arange(1.0, 5.0).reshape(1, 2, 2))
    mats = {"grid": A, "strength": S, "transpose": A.transpose(), "product": A.mult_matrix(A),
            "level A": ml.level_matrix(1, "A"), "level P": ml.level_matrix(0, "P"),
            "blocks": blocks.to_CSR(),
            "arrays": rb.ParCSRMatrix.from_arrays(2, 2, [0, 1, 2], [0, 1], [1.0, 2.0])}
    for name, M in mats.items():
        ptrs = [ctypes.c_void_p() for _ in range(3)]
        rb.check(rb.lib().rb_csr_device_arrays(M.h, *map(ctypes.byref, ptrs)))
        for ptr in ptrs:
            assert _ipc_capable(ptr.value), name
    x = rb.ParVector(n, values=np.ones(n))
    y, z = rb.ParVector(n), rb.ParVector(n)
    A.mult(x, y)
    mats["transpose"].mult(x, z)     # (the square grid's operator is symmetric)
    np.testing.assert_allclose(y.numpy(), z.numpy(), rtol=0, atol=1e-13)


def test_a_new_vector_may_be_written_on_any_stream():
    """With work queued on the library's stream, a vector is created and at
    once filled through its view on another stream: its zeros are in place
    by then."""
    s, mine = torch.cuda.Stream(), torch.cuda.Stream()
    busy = torch.zeros(1 << 26, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    vs = []
    try:
        rb.set_stream(s.cuda_stream)
        for n in (5, 1 << 16, 1 << 22):
            with torch.cuda.stream(s):
                for _ in range(20):
                    busy += 1.0
            v = rb.ParVector(n)
            assert s.query()
            with torch.cuda.stream(mine):
                v.torch_view().fill_(3.0)
            vs.append(v)
        mine.synchronize()
        s.synchronize()
        for v in vs:
            assert torch.all(v.torch_view() == 3.0)
            assert v.inner_product(v) == 9.0 * v.local_n
    finally:
        rb.synchronize()
        rb.set_stream(0)


def test_workspaces_replaced_while_another_stream_uses_them():
    """A block cycle of 4 columns is pending on one stream when one of 8
    columns on another replaces the hierarchy's workspaces."""
    A = rb.par_stencil_grid(rb.diffusion_stencil_2d(0.1, 0.4), [300, 300])
    n = A.global_num_rows
    ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
    ml.setup(A)
    rng = np.random.default_rng(8)
    B = {k: rb.ParVector(n * k, values=rng.uniform(-1, 1, n * k)) for k in (4, 8)}
    want = {}
    for k in (8, 4):
        X = rb.ParVector(n * k)
        ml.cycle_block(X, B[k], k)
        want[k] = X.numpy()
    X = {k: rb.ParVector(n * k) for k in (4, 8)}
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    busy = torch.zeros(1 << 26, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    try:
        rb.set_stream(first.cuda_stream)
        with torch.cuda.stream(first):
            for _ in range(20):
                busy += 1.0
        ml.cycle_block(X[4], B[4], 4)
        rb.set_stream(second.cuda_stream)
        ml.cycle_block(X[8], B[8], 8)
        assert first.query()          # nothing is freed under a pending cycle
        first.synchronize()
        second.synchronize()
    finally:
        rb.synchronize()
        rb.set_stream(0)
    for k in (4, 8):
        np.testing.assert_allclose(X[k].numpy(), want[k], rtol=1e-12, atol=1e-14)


def test_memory_freed_in_a_capture_is_not_reused_under_pending_reads():
    """Waiting for the device is refused while a stream capture is in progress
    (a garbage collector may run in one): the memory stays taken until a
    later release could wait."""
    from cuda.bindings import runtime

    n = 1 << 22
    v = rb.ParVector(n, values=np.full(n, 3.0))
    t, at = v.torch_view(), v.device_ptr()
    acc = torch.zeros(n, dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    err, c = runtime.cudaStreamCreateWithFlags(runtime.cudaStreamNonBlocking)
    assert int(err) == 0
    with torch.cuda.stream(side):
        for _ in range(200):
            acc += t
    (err,) = runtime.cudaStreamBeginCapture(c, runtime.cudaStreamCaptureMode.cudaStreamCaptureModeGlobal)
    assert int(err) == 0
    del t, v
    gc.collect()
    runtime.cudaStreamEndCapture(c)      # (the wait that was tried ended it)
    runtime.cudaGetLastError()
    new = [rb.ParVector(n, values=np.full(n, -7.0)) for _ in range(4)]
    assert all(w.device_ptr() != at for w in new)
    side.synchronize()
    assert torch.all(acc == 600.0)
    del new                              # the late free happens here
    gc.collect()
    runtime.cudaStreamDestroy(c)
    # (more than the slabs keep free: one of them covers the place again)
    again = [rb.ParVector(n) for _ in range(40)]
    assert any(w.device_ptr() <= at < w.device_ptr() + 8 * n for w in again)


def test_memory_goes_back_once_the_last_handle_is_gone():
    """A hierarchy and vectors of 1.5 GiB: with every handle destroyed at most
    384 MiB stay with the library, and after rb.trim() nothing but the
    driver's granularity (and the two buffers of the process, made by a first
    small run)."""
    code = """
import gc, torch, raptor_b200 as rb
rb.init(0)
free = lambda: torch.cuda.mem_get_info()[0]
def work(m, count):
    A = rb.par_stencil_grid(rb.laplace_stencil_27pt(), [m, m, m])
    ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
    ml.setup(A)
    x, b = rb.ParVector(m ** 3), rb.ParVector(m ** 3)
    b.set_const_value(1.0)
    ml.cycle(x, b)
    many = [rb.ParVector(1 << 21) for _ in range(count)]   # 16 MiB each
    rb.synchronize()
    return free()
work(30, 1)
gc.collect()
rb.trim()
before = free()
held = work(64, 64)
assert held < before - (1200 << 20), (before, held)
gc.collect()
kept = before - free()
rb.trim()
left = before - free()
print(kept >> 20, left >> 20, flush=True)
assert kept <= (384 + 64) << 20, kept
assert left <= 64 << 20, left
x = rb.ParVector(1 << 21)
x.set_const_value(1.0)
assert abs(x.norm() - (1 << 21) ** 0.5) < 1e-9
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stdout + r.stderr


def test_process_exit_after_the_callers_stream_is_gone():
    code = """
import torch, raptor_b200 as rb
from cuda.bindings import runtime
rb.init(0)
err, s = runtime.cudaStreamCreate()
rb.set_stream(int(s))
x = rb.ParVector(1000)
x.set_const_value(2.0)
assert x.norm() == 2.0 * 1000 ** 0.5
rb.synchronize()
del x
(err,) = runtime.cudaStreamDestroy(s)
assert int(err) == 0
print("ended", flush=True)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stdout.strip() == "ended", r.stderr


def test_borrowed_memory_outlives_pending_reads():
    n = 1 << 22
    for rep in range(5):
        v = rb.ParVector(n, values=np.full(n, 1.0 + rep))
        t = v.torch_view()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            acc = torch.zeros(n, dtype=torch.float64, device="cuda")
            for _ in range(50):
                acc += t
        del t, v                     # the reads above may still be pending
        w = rb.ParVector(n)          # takes the freed memory and overwrites it
        w.set_const_value(-7.0)
        rb.synchronize()
        side.synchronize()
        assert torch.all(acc == 50.0 * (1.0 + rep))
        del w


def test_hierarchies_on_another_stream_than_their_setup():
    """A handle made on the library's stream is complete when the call
    returns: it works at once on a stream the caller sets, and its memory is
    freed after that stream is gone."""
    A = rb.par_stencil_grid(rb.laplace_stencil_27pt(), [20, 20, 20])
    n = A.global_num_rows
    bh = np.random.default_rng(3).uniform(-1, 1, n)
    got = []
    for own in (True, False):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
        ml.setup(A)
        s = None if own else torch.cuda.Stream()
        try:
            if s is not None:
                rb.set_stream(s.cuda_stream)
            b, x = rb.ParVector(n, values=bh), rb.ParVector(n)
            ml.cycle(x, b)
            got.append(x.numpy())
        finally:
            rb.synchronize()
            rb.set_stream(0)
        del s, ml, b, x
        gc.collect()
    np.testing.assert_allclose(got[0], got[1], rtol=1e-12, atol=1e-14)
