"""GPU tests of the products' row schedules at the sizes where they change:
rows and columns of 256 and 257 entries (a longer one has a block of its
own), of several thousand, empty ones, and the mean lengths at which the
transposed product changes its lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


def ragged(rng, n, m, lens):
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(lens)
    cols = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in lens]).astype(np.int32)
    return rowptr, cols, rng.uniform(-1.0, 1.0, len(cols))


@pytest.mark.parametrize("n,m,mean,special", [
    (5000, 4000, 5, [256, 257, 258, 3000]),      # rows on blocks of their own, 2 lanes
    (4000, 9000, 14, [0, 0, 255, 256, 257, 8999]),
    (9000, 4096, 12, []),                        # no long row, columns of about 26
    (300, 200, 3, [200, 0]),                     # below the timed sizes
    (20000, 3, 2, []),                           # columns of thousands of entries
])
def test_products_with_long_rows_and_columns(n, m, mean, special):
    rng = np.random.default_rng(n + m)
    lens = rng.integers(0, 2 * mean + 1, n)
    lens[rng.choice(n, len(special), replace=False)] = special
    lens = np.minimum(lens, m)
    rowptr, cols, vals = ragged(rng, n, m, lens)
    A = rb.ParCSRMatrix.from_arrays(n, m, rowptr, cols, vals)
    rows = np.repeat(np.arange(n), lens)
    xh, uh = rng.uniform(-1, 1, m), rng.uniform(-1, 1, n)
    x, u = rb.ParVector(m, values=xh), rb.ParVector(n, values=uh)
    b, r, t, a = rb.ParVector(n), rb.ParVector(n), rb.ParVector(m), rb.ParVector(n, values=uh)
    A.mult(x, b)
    A.residual(x, u, r)
    A.mult_append(x, a)
    A.mult_T(u, t)
    own = rb.ParVector(n, values=uh)
    A.residual(x, own, own)          # in place
    np.testing.assert_array_equal(own.numpy(), r.numpy())
    want = np.bincount(rows, vals * xh[cols], n)
    wantT = np.bincount(cols, vals * uh[rows], m)
    # |sum error| <= (terms) eps sum |terms|, for any order of the sum
    scale = np.bincount(rows, np.abs(vals * xh[cols]), n)
    scaleT = np.bincount(cols, np.abs(vals * uh[rows]), m)
    eps = np.finfo(np.float64).eps
    bound = eps * (lens + 2) * (scale + np.abs(uh)) + 1e-300
    assert np.all(np.abs(b.numpy() - want) <= bound)
    assert np.all(np.abs(r.numpy() - (uh - want)) <= 2 * bound)
    assert np.all(np.abs(a.numpy() - (uh + want)) <= 2 * bound)
    assert np.all(np.abs(t.numpy() - wantT) <= eps * (np.bincount(cols, minlength=m) + 2) * scaleT + 1e-300)


def test_transposed_product_is_complete_on_return():
    """Whatever was queued before it on the stream: the caller may read the
    result on another stream at once (the first call also builds the map)."""
    torch = pytest.importorskip("torch")
    A = rb.par_stencil_grid(rb.diffusion_stencil_2d(0.1, 0.4), [80, 80])
    n = A.global_num_rows
    uh = np.random.default_rng(5).uniform(-1, 1, n)
    u, t = rb.ParVector(n, values=uh), rb.ParVector(n)
    s, mine = torch.cuda.Stream(), torch.cuda.Stream()
    busy = torch.zeros(1 << 26, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    got = []
    try:
        rb.set_stream(s.cuda_stream)
        for rep in range(3):
            with torch.cuda.stream(s):
                for _ in range(20):
                    busy += 1.0      # about 3 ms of work ahead of the product
            A.mult_T(u, t)
            assert s.query()
            with torch.cuda.stream(mine):
                got.append(t.torch_view().clone())
            mine.synchronize()
            t.set_const_value(0.0)
    finally:
        rb.synchronize()
        rb.set_stream(0)
    b = rb.ParVector(n)
    A.mult(u, b)                     # the operator is symmetric (a square grid)
    for g in got:
        np.testing.assert_allclose(g.cpu().numpy(), b.numpy(), rtol=1e-13, atol=1e-13)


@pytest.mark.parametrize("prec", [rb.FP64, rb.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("k", [4, 8, 12, 16, 24])
def test_block_cycle_with_split_rows(prec, k):
    """Column groups of 16 bytes with a row's entries split over 1 to 8
    groups: levels above and below the size whose split is timed, against one
    single-vector cycle a column (the order of the sums is all that
    differs)."""
    m = 26
    st = [0.0] * 27
    st[13], st[12], st[14], st[10], st[16], st[4], st[22] = 4.02, -1, -1, -1, -1, -0.01, -0.01
    A = rb.par_stencil_grid(st, [m, m, m])
    n = A.global_num_rows
    ml = rb.ParSmoothedAggregationSolver(0.25, relax_type=rb.L1Jacobi)
    ml.precision = prec
    ml.setup(A)
    Bh = np.random.default_rng(k).uniform(-1, 1, (n, k))
    X = rb.ParVector(n * k)
    ml.cycle_block(X, rb.ParVector(n * k, values=Bh.reshape(-1)), k)
    got = X.numpy().reshape(n, k)
    tol = 1e-11 if prec == rb.FP64 else 1e-5
    for c in range(k):
        x = rb.ParVector(n)
        ml.cycle(x, rb.ParVector(n, values=Bh[:, c]))
        ref = x.numpy()
        assert np.linalg.norm(got[:, c] - ref) <= tol * np.linalg.norm(ref), c
