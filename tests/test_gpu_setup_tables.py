"""Setup kernels at the sizes where their tables and lanes change: sparse
products whose rows overflow the first key table (192 and 768 distinct
columns), fill each table of the numeric pass (64, 128, 256, 2048 and more)
and have long rows of A or of B; row sorts at the staging area's capacity (96
and 384 entries a group, runs of 1536 for longer rows), with and without a
diagonal, and with repeated columns;
extended interpolation with sets of more than 64 and more than 256 points.
Products and interpolation are compared bit for bit with sums in the same
order."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_parity import assert_csr_equal, oc_tuple, rb_tuple

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


def matrix(rng, n, m, lens):
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(lens)
    cols = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in lens] + [[]]).astype(np.int32)
    return rowptr, cols, rng.uniform(-1.0, 1.0, len(cols))


@pytest.mark.parametrize("n,k,m,la,lb,long_a", [
    (600, 500, 400, 4, 3, [0, 60, 61, 62, 250]),       # 8 lanes a row, overflow of 192 keys
    (300, 400, 3000, 6, 20, [0, 30, 40, 50, 128]),     # 32 lanes a row, overflow of 768 keys
    (60, 200, 9000, 10, 60, [0, 1, 100, 199]),         # thousands of columns: 8192 keys, global
    (2000, 2000, 2000, 3, 2, []),
    (500, 300, 64, 20, 6, [299]),                      # every column met many times
])
def test_spgemm_tables(n, k, m, la, lb, long_a):
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 2 * la + 1, n)
    lens[rng.choice(n, len(long_a), replace=False)] = long_a
    arp, aci, acv = matrix(rng, n, k, np.minimum(lens, k))
    brp, bci, bcv = matrix(rng, k, m, rng.integers(0, 2 * lb + 1, k))
    C = rb.ParCSRMatrix.from_arrays(n, k, arp, aci, acv).mult_matrix(
        rb.ParCSRMatrix.from_arrays(k, m, brp, bci, bcv))
    rp, ci, cv = C.arrays()
    for i in range(n):
        acc = {}
        for j in range(arp[i], arp[i + 1]):
            for q in range(brp[aci[j]], brp[aci[j] + 1]):
                acc[bci[q]] = acc.get(bci[q], 0.0) + acv[j] * bcv[q]
        want = sorted((c, v) for c, v in acc.items() if abs(v) > 1e-16)
        assert list(ci[rp[i]:rp[i + 1]]) == [c for c, _ in want], i
        assert list(cv[rp[i]:rp[i + 1]]) == [v for _, v in want], i


@pytest.mark.parametrize("mean", [6, 40])
def test_row_sort(mean):
    rng = np.random.default_rng(mean)
    n = 700
    lens = rng.integers(0, 2 * mean + 1, n)
    lens[rng.choice(n, 14, replace=False)] = [0, 1, 95, 96, 97, 383, 384, 385,
                                              1535, 1536, 1537, 3072, 3073, 9001]
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(lens)
    cols = rng.integers(0, n, rowptr[-1]).astype(np.int32)      # repeated columns too
    rows = np.repeat(np.arange(n), lens)
    hit = rng.random(len(cols)) < 0.05
    cols[hit] = rows[hit]
    vals = rng.uniform(-1, 1, len(cols))
    A = rb.ParCSRMatrix.from_arrays(n, n, rowptr, cols, vals).sort_diag_first()
    rp, ci, cv = A.arrays()
    for i in range(n):
        s, e = rowptr[i], rowptr[i + 1]
        order = list(np.argsort(cols[s:e], kind="stable"))
        d = [q for q in order if cols[s + q] == i]
        if d:
            order.remove(d[0])
            order.insert(0, d[0])
        np.testing.assert_array_equal(ci[s:e], cols[s:e][order])
        np.testing.assert_array_equal(cv[s:e], vals[s:e][order])


@pytest.mark.parametrize("width", [12, 40, 140])
def test_extended_interpolation_with_large_sets(width):
    """A banded matrix whose rows reach 4 width coarse points: sets of about
    50, of more than 64 and of more than 256 entries (and neighbours of
    more than 32 entries)."""
    n = 900
    rng = np.random.default_rng(width)
    rows, cols, vals = [], [], []
    for i in range(n):
        js = [j for j in range(max(0, i - width), min(n, i + width + 1)) if j != i]
        v = -rng.uniform(0.8, 1.0, len(js))
        rows += [i] * (len(js) + 1)
        cols += [i] + js
        vals += [-v.sum() + 0.1] + list(v)
    rowptr = np.searchsorted(rows, np.arange(n + 1)).astype(np.int32)
    A = rb.ParCSRMatrix.from_arrays(n, n, rowptr, cols, vals).sort_diag_first()
    S = A.strength(rb.Classical, 0.25)
    states = (rng.random(n) < 0.5).astype(np.int32)
    P = rb.extended_interpolation(A, S, states, 0.0)
    Ao = O.CSR.from_arrays(n, n, *A.arrays())
    So = O.classical_strength(Ao, 0.25)
    Po = O.interpolation(Ao, So, states, "extended", 0.0)
    assert_csr_equal(rb_tuple(P), oc_tuple(Po))
