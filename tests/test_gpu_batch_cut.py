"""The batch whose cycles end in a dense matrix (the level each system is cut
at is chosen by size, fewer rows when the matrices of all systems would not
fit) against the batch without it (fuse_coarse = 0) and against standalone
cycles; the reported levels are those of the whole hierarchies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rb = pytest.importorskip("raptor_b200")


@pytest.fixture(scope="module", autouse=True)
def _device():
    rb.init(0)


def make(prec, fuse, relax, compat=0):
    ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, relax)
    ml.precision, ml.fuse_coarse, ml.jacobi_compat = prec, fuse, compat
    return ml


# sides 5 and 7: no coarse level at all, and none above the coarsest; 40 systems
# of 60 x 60 and more: the cut falls to 512 and 256 rows
SETS = {"mixed": [5, 7, 13, 40, 90], "one": [64], "many": [60, 64, 68, 72] * 10}


def expected_cuts(mats, prec, fuse, relax, compat):
    """The size rule: down to the first level of at most 1024 rows, halved
    until the matrices (FP64, rows padded to 16 bytes) fit 32 MB."""
    sizes = []
    for A in mats:
        ml = make(prec, 0, relax, compat)
        ml.setup(A)
        sizes.append([ml.level_info(l)[0] for l in range(ml.num_levels)])
    depth = [len(s) for s in sizes]
    if fuse == 0 or relax == rb.SOR:
        return depth
    cap = 1024
    while cap >= 64:
        cuts = []
        for s in sizes:
            c = len(s)
            for l in range(len(s) - 2, 0, -1):
                if s[l] > cap:
                    break
                c = l + 1
            cuts.append(c)
        if sum(s[c - 1] * (s[c - 1] + 1 & ~1) * 8 for s, c in zip(sizes, cuts)) <= 32 << 20:
            assert cuts != depth
            return cuts
        cap //= 2
    return depth


@pytest.mark.parametrize("prec", [rb.FP64, rb.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("sides", sorted(SETS))
@pytest.mark.parametrize("relax,compat", [(rb.L1Jacobi, 0), (rb.Jacobi, 1), (rb.SOR, 0)],
                         ids=["l1_jacobi", "jacobi_noop", "sor"])
def test_batch_cycle_with_and_without_the_cut(sides, prec, relax, compat):
    mats = [rb.par_stencil_grid(rb.diffusion_stencil_2d(0.05, 0.3 + 0.01 * i), [m, m])
            for i, m in enumerate(SETS[sides])]
    got, levels = [], []
    for fuse in (0, 1):
        B = rb.Batch(mats, make(prec, fuse, relax, compat))
        assert list(B.cuts) == expected_cuts(mats, prec, fuse, relax, compat)
        b = rb.ParVector(B.total_rows, values=np.random.default_rng(3).uniform(-1, 1, B.total_rows))
        x = rb.ParVector(B.total_rows)
        B.cycle(x, b)
        got.append(x.numpy())
        levels.append(list(B.levels))
    assert levels[0] == levels[1]
    tol = 1e-11 if prec == rb.FP64 else 1e-4
    for s, m in enumerate(SETS[sides]):
        lo, hi = B.offsets[s], B.offsets[s + 1]
        ref = got[0][lo:hi]
        assert np.linalg.norm(got[1][lo:hi] - ref) <= tol * np.linalg.norm(ref), (s, m)
    if relax == rb.SOR:
        return   # the batch's rows are coloured as one matrix, not system by system
    ml = make(prec, 1, relax, compat)
    ml.setup(mats[-1])
    lo, hi = B.offsets[-2], B.offsets[-1]
    y = rb.ParVector(int(hi - lo))
    ml.cycle(y, rb.ParVector(int(hi - lo), values=b.numpy()[lo:hi]))
    assert np.linalg.norm(got[1][lo:hi] - y.numpy()) <= tol * np.linalg.norm(y.numpy())
    assert ml.num_levels == levels[1][-1]
