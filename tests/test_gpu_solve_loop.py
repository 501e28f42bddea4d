"""The stationary solve's device-side loop against the loop on the host
(use_graphs = 0): the same iterations, history and solution, over a launch
boundary of the loop (1024 iterations), with an iteration limit inside and
outside a launch, and when no iteration is needed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


@pytest.mark.parametrize("limit,tol,weight", [(1500, 1e-8, 0.05), (1024, 1e-30, 0.6), (1025, 1e-30, 0.6),
                                              (7, 1e-8, 0.6), (0, 1e-8, 0.6), (50, 2.0, 0.6)])
def test_solve_equals_host_loop(limit, tol, weight):
    A = rb.par_stencil_grid(rb.diffusion_stencil_2d(0.001, np.pi / 8), [40, 40])
    n = A.global_num_rows
    b = rb.ParVector(n, values=np.random.default_rng(1).uniform(-1, 1, n))
    got = []
    for graphs in (0, 1):
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, rb.Jacobi)
        ml.relax_weight, ml.max_iterations, ml.solve_tol, ml.use_graphs = weight, limit, tol, graphs
        ml.setup(A)
        x = rb.ParVector(n)
        its = ml.solve(x, b)
        got.append((its, np.array(ml.get_residuals()), x.numpy()))
    (i0, r0, x0), (i1, r1, x1) = got
    assert i0 == i1 and len(r0) == len(r1) == i0 + 1
    # the cycles are the same; the norms' sums differ in their order only, and
    # at the residual's round-off floor b - A x is all rounding
    np.testing.assert_allclose(r1, r0, rtol=1e-10, atol=1e-14)
    np.testing.assert_array_equal(x0, x1)
