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
