"""The staged block CSR products (bsr.cu, k_bsr_staged) where their schedule
changes: block sizes from 1x1 to the largest that fits the staging area and
just past it, more scalar rows a block than a warp has lanes, block rows of
many blocks (several pieces), empty ones, and a last warp that is not full.
Results are those of the reference's order of operations bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


def in_order(n, rows, terms, start, sign=1.0):
    """start[r] + or - its terms one after another, for all rows at once."""
    out = start.copy()
    order = np.argsort(rows, kind="stable")
    rows, terms = rows[order], terms[order]
    pos = np.arange(len(rows)) - np.searchsorted(rows, rows)
    for p in range(pos.max() + 1 if len(pos) else 0):
        k = pos == p
        out[rows[k]] = out[rows[k]] + sign * terms[k]
    return out


@pytest.mark.parametrize("br,bc,nb,nc,long_row", [
    (1, 1, 700, 500, 600), (2, 2, 333, 333, 130), (3, 3, 257, 200, 60), (3, 2, 100, 150, 90),
    (2, 5, 90, 41, 40), (6, 6, 70, 70, 20), (16, 32, 5, 4, 3), (23, 23, 4, 4, 3), (33, 2, 9, 9, 4),
    (32, 16, 6, 6, 2), (7, 1, 50, 300, 200),
])
def test_products_bit_exact(br, bc, nb, nc, long_row):
    rng = np.random.default_rng(100 * br + bc)
    lens = rng.integers(0, 8, nb)
    lens[rng.integers(nb)] = long_row
    lens[-1] = 0
    rowptr = np.zeros(nb + 1, np.int32)
    rowptr[1:] = np.cumsum(lens)
    z = int(rowptr[-1])
    cols = rng.integers(0, nc, z).astype(np.int32)
    vals = rng.uniform(-1, 1, (z, br, bc))
    A = rb.BSRMatrix.from_arrays(nb, nc, br, bc, rowptr, cols, vals)
    xh, uh = rng.uniform(-1, 1, nc * bc), rng.uniform(-1, 1, nb * br)
    x, u = rb.ParVector(nc * bc, values=xh), rb.ParVector(nb * br, values=uh)
    b, r, a, t = (rb.ParVector(nb * br), rb.ParVector(nb * br), rb.ParVector(nb * br, values=uh),
                  rb.ParVector(nc * bc))
    A.mult(x, b)
    A.residual(x, u, r)
    A.mult_append(x, a)
    A.mult_T(u, t)
    brow = np.repeat(np.arange(nb), lens)
    # entries in storage order: block, row of the block, column of the block
    R = np.broadcast_to((brow[:, None] * br + np.arange(br))[:, :, None], vals.shape).reshape(-1)
    C = np.broadcast_to((cols.astype(np.int64)[:, None] * bc + np.arange(bc))[:, None, :], vals.shape).reshape(-1)
    v = vals.reshape(-1)
    zero = np.zeros(nb * br)
    np.testing.assert_array_equal(b.numpy(), in_order(nb * br, R, v * xh[C], zero))
    np.testing.assert_array_equal(r.numpy(), in_order(nb * br, R, v * xh[C], uh, -1.0))
    np.testing.assert_array_equal(a.numpy(), in_order(nb * br, R, v * xh[C], uh))
    np.testing.assert_array_equal(t.numpy(), in_order(nc * bc, C, v * uh[R], np.zeros(nc * bc)))
