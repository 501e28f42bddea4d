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
        x = rb.ParVector(n)
        ml.cycle(x, b)
        got.append(x.numpy())
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
        x = rb.ParVector(n)
        ml.cycle(x, b)
        got.append(x.numpy())
    np.testing.assert_array_equal(got[0], got[1])


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
