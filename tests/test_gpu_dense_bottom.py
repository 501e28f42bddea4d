"""The bottom of the V-cycle as one dense product (dense_bottom.cuh, the
default) against the level-by-level cycle (fuse_coarse = 0).  Both apply the
same linear operator; in FP64 they differ by the rounding of the levels they
replace, in FP32 by the rounding of single precision (the product is the more
exact of the two: its matrix is formed and kept in FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


LIMIT = 16 << 20     # bytes of the largest matrix, FP64, rows padded to 16 bytes


def start_level(ml):
    """(level, rows) at which the size rule starts the dense product."""
    sizes = [ml.level_info(l)[0] for l in range(ml.num_levels)]
    f = -1
    for l in range(len(sizes) - 2, 0, -1):
        if sizes[l] == 0 or sizes[l] * (sizes[l] + 1 & ~1) * 8 > LIMIT:
            break
        f = l
    return (f, sizes[f]) if f > 0 else (-1, 0)


def operator(name, m):
    if name == "lap27":
        return rb.par_stencil_grid(rb.laplace_stencil_27pt(), [m, m, m])
    return rb.par_stencil_grid(rb.diffusion_stencil_2d(0.1, 0.4), [m, m])


@pytest.mark.parametrize("prec", [rb.FP64, rb.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("relax,compat", [(rb.L1Jacobi, 0), (rb.Jacobi, 0), (rb.Jacobi, 1)],
                         ids=["l1_jacobi", "jacobi", "jacobi_noop"])
@pytest.mark.parametrize("name,m", [("lap27", 18), ("lap27", 31), ("rot2d", 61), ("rot2d", 140)])
def test_cycle_equals_level_by_level(name, m, relax, compat, prec):
    A = operator(name, m)
    n = A.global_num_rows
    b = rb.ParVector(n, values=np.random.default_rng(m).uniform(-1, 1, n))
    got = []
    for fuse in (0, 1):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, relax)
        ml.precision, ml.jacobi_compat, ml.fuse_coarse = prec, compat, fuse
        if relax == rb.Jacobi:
            ml.relax_weight = 2.0 / 3.0
        ml.setup(A)
        assert ml.num_levels >= 3
        assert ml.dense_info() == (start_level(ml) if fuse else (-1, 0))
        x = rb.ParVector(n)
        ml.cycle(x, b)
        got.append(x.numpy())
    assert ml.dense_info()[0] >= 1
    tol = 1e-11 if prec == rb.FP64 else 1e-4
    assert np.all(np.isfinite(got[1]))
    assert np.linalg.norm(got[1] - got[0]) <= tol * np.linalg.norm(got[0])


@pytest.mark.parametrize("sweeps,relax", [(2, rb.L1Jacobi), (1, rb.SOR)], ids=["two_sweeps", "sor"])
def test_other_smoothers_keep_the_levels(sweeps, relax):
    A = operator("rot2d", 100)
    n = A.global_num_rows
    b = rb.ParVector(n, values=np.random.default_rng(2).uniform(-1, 1, n))
    got = []
    for fuse in (0, 1):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, relax)
        ml.num_smooth_sweeps, ml.fuse_coarse = sweeps, fuse
        ml.setup(A)
        assert ml.dense_info() == (-1, 0)
        x = rb.ParVector(n)
        ml.cycle(x, b)
        got.append(x.numpy())
    np.testing.assert_array_equal(got[0], got[1])


@pytest.fixture(scope="module")
def paths():
    """Path operators (tridiagonal) whose level 1 has 1448 rows (a matrix of
    16 MB less 3 kB) and 1449 (16 MB and 31 kB)."""
    found = {}
    for n in range(2600, 4400):
        rowptr = np.concatenate([[0], np.cumsum(np.r_[2, np.full(n - 2, 3), 2])])
        cols = np.concatenate([[0, 1]] + [[i - 1, i, i + 1] for i in range(1, n - 1)] + [[n - 2, n - 1]])
        A = rb.ParCSRMatrix.from_arrays(n, n, rowptr.astype(np.int32), cols.astype(np.int32),
                                        np.where(cols == np.repeat(np.arange(n), np.diff(rowptr)), 2.0, -1.0))
        S = A.strength(rb.Classical, 0.25)
        coarse = int(np.sum(rb.split_pmis(S) == 1))
        if coarse in (1448, 1449):
            found.setdefault(coarse, A)
        if len(found) == 2:
            return found
    raise AssertionError("no path of that size")


@pytest.mark.parametrize("prec", [rb.FP64, rb.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("rows", [1448, 1449])
def test_largest_matrix(paths, rows, k, prec):
    """At the size limit and one row above it, one right-hand side and three."""
    A = paths[rows]
    n = A.global_num_rows
    B = np.random.default_rng(rows).uniform(-1, 1, n * k)
    got = []
    for fuse in (0, 1):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
        ml.precision, ml.fuse_coarse = prec, fuse
        ml.setup(A)
        assert ml.level_info(1)[0] == rows
        x, b = rb.ParVector(n * k), rb.ParVector(n * k, values=B)
        if k == 1:
            ml.cycle(x, b)
        else:
            ml.cycle_block(x, b, k)
        got.append(x.numpy())
    assert ml.dense_info() == start_level(ml) == ((1, 1448) if rows == 1448 else (2, ml.level_info(2)[0]))
    # x is nearly all the smoothest component, of which b, uniform, holds one
    # part in sqrt(n); 16 roundings of b and of the levels' vectors
    tol = 16 * 2.0 ** (-53 if prec == rb.FP64 else -24) * n ** 0.5
    assert np.linalg.norm(got[1] - got[0]) <= tol * np.linalg.norm(got[0])


def shifted_laplacian(m, d, shift):
    """Graph Laplacian of an m^d grid (its null vector is the constant) plus
    shift times the identity."""
    n = m ** d
    idx = np.arange(n).reshape((m,) * d)
    rows, cols = [], []
    for a in range(d):
        p = np.take(idx, np.arange(m - 1), axis=a).ravel()
        q = np.take(idx, np.arange(1, m), axis=a).ravel()
        rows += [p, q]
        cols += [q, p]
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    vals = np.concatenate([-np.ones(len(rows)), np.bincount(rows, minlength=n) + shift])
    rows, cols = np.concatenate([rows, np.arange(n)]), np.concatenate([cols, np.arange(n)])
    o = np.lexsort((cols, rows))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return n, rowptr.astype(np.int32), cols[o].astype(np.int32), vals[o]


# The matrix of the bottom holds 1 / shift times the constant's projector, and
# a right-hand side without a constant part must not see it: what it gets is
# what the FP32 vectors round, 2^-24 = 6e-8 an operation (1.3e-7 level by
# level).  Rounded to FP32 the matrix's entries were off by 6e-8 / shift of
# that: 5e-5 and 2e-4 here.  The bound is 16 roundings.
@pytest.mark.parametrize("m,d", [(100, 2), (40, 3)])
def test_fp32_cycle_of_a_nearly_singular_operator(m, d):
    n, *arrays = shifted_laplacian(m, d, 1e-7)
    A = rb.ParCSRMatrix.from_arrays(n, n, *arrays)
    bh = np.random.default_rng(1).uniform(-1, 1, n)
    b = rb.ParVector(n, values=bh - bh.mean())
    got = []
    for prec, fuse in ((rb.FP64, 0), (rb.FP32, 0), (rb.FP32, 1)):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
        ml.precision, ml.fuse_coarse = prec, fuse
        ml.setup(A)
        x = rb.ParVector(n)
        ml.cycle(x, b)
        z = x.numpy()
        got.append(z - z.mean())
    for z in got[1:]:
        assert np.linalg.norm(z - got[0]) <= 16 * 2.0 ** -24 * np.linalg.norm(got[0])
