"""Device memory of the library: freed memory is kept for the next allocation
up to a bound, and memory a caller borrowed from a handle is not handed to
anyone else before the caller's pending work on it is done."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


# 1 GiB arrays are the driver's own, 32 MiB ones the pool's, which keeps 2 GiB
@pytest.mark.parametrize("log2n, kept", [(27, 0), (22, 2 << 30)])
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
