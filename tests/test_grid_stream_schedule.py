"""The box-grid kernel's schedule (raptor_b200/csrc/grid.cuh, k_grid_rows)
restated on the CPU over box sizes that are not multiples of its tiles or of
its planes a block, for every stencil shape and one or two rows in x a
thread: the per-thread plane loads two steps ahead, the two plane buffers,
the three running sums (outputs z - 1, z, z + 1 of input plane z) and the
row's own value kept for one step.  It checks what the kernel relies on: every
global load lies inside x, every shared read inside the plane that belongs
to the step (buffers carry the plane they hold) and on an even index where
pairs are read, products enter each sum in diagonal order, every row is
written exactly once, and the result is the zero-padded stencil product."""
import numpy as np
import pytest

from tests.test_grid_schedule import CASES, shape


def run_schedule(s, vx, nx, ny, nz, zc):
    sh, hy = shape(s)
    txt = 32 if hy else 256
    txw, tyh = txt * vx, (8 if hy else 1)
    W, H = txw + 2, tyh + 2 * hy
    P, NT = W * H, txt * tyh
    lpt = (P + NT - 1) // NT
    plane, n = nx * ny, nx * ny * nz
    rng = np.random.default_rng(1)
    x, c = rng.standard_normal(n), rng.standard_normal(len(sh))
    y, own_y, cnt = np.full(n, np.nan), np.full(n, np.nan), np.zeros(n, int)
    ntx, nty = -(-nx // txw), -(-ny // tyh)
    t = np.arange(NT)
    tx, ty = t % txt, t // txt
    for blk in range(ntx * nty * -(-nz // zc)):
        bx, bt = blk % ntx, blk // ntx
        x0, y0, z0 = bx * txw, (bt % nty) * tyh, (bt // nty) * zc
        zend = min(z0 + zc, nz)
        goff = []
        for u in range(lpt):
            e = t + u * NT
            gy, gx = y0 - hy + e // W, x0 - 1 + e % W
            goff.append(np.where((e < P) & (gy >= 0) & (gy < ny) & (gx >= 0) & (gx < nx), gy * nx + gx, -1))
        buf, holds = np.full((2, P), np.nan), [None, None]

        def load(zp):
            v = []
            for u in range(lpt):
                vv, m = np.zeros(NT), (goff[u] >= 0) & (0 <= zp < nz)
                idx = zp * plane + goff[u][m]
                assert np.all((idx >= 0) & (idx < n))
                vv[m] = x[idx]
                v.append(vv)
            return zp, v

        def store(slot, zv):
            for u in range(lpt):
                e = t + u * NT
                m = e < P if u == lpt - 1 else np.ones(NT, bool)
                assert np.all(e[m] < P)
                buf[slot, e[m]] = zv[1][u][m]
            holds[slot] = zv[0]

        left = (ty + hy) * W + tx * vx
        xr = x0 + tx * vx
        inr = [(y0 + ty < ny) & (xr + r < nx) for r in range(vx)]
        store(0, load(z0 - 1))
        v = load(z0)
        sums = [[np.zeros(NT) for _ in range(vx)] for _ in range(3)]
        last = [[[-1] for _ in range(vx)] for _ in range(3)]
        own = [np.zeros(NT) for _ in range(vx)]
        for zp in range(z0 - 1, zend + 1):
            K = (zp - (z0 - 1)) & 1
            assert holds[K] == zp
            w = load(zp + 2) if zp + 1 < zend else None
            mid = None
            for dy in range(-hy, hy + 1):
                row = left + dy * W
                assert np.all((row >= 0) & (row % W + vx + 1 < W) & (row + vx + 1 < P))
                assert vx == 1 or np.all(row % 2 == 0)
                val = [buf[K, row + q] for q in range(vx + 2)]
                if dy == 0:
                    mid = val[1:1 + vx]
                for d, (dz, ddy, dx) in enumerate(sh):
                    if ddy != dy:
                        continue
                    for r in range(vx):
                        assert last[1 - dz][r][-1] < d
                        last[1 - dz][r].append(d)
                        sums[1 - dz][r] = sums[1 - dz][r] + c[d] * val[1 + r + dx]
            if zp > z0:
                for r in range(vx):
                    ii = ((zp - 1) * plane + (y0 + ty) * nx + xr + r)[inr[r]]
                    assert last[0][r][1:] == list(range(len(sh)))
                    y[ii], own_y[ii] = sums[0][r][inr[r]], own[r][inr[r]]
                    cnt[ii] += 1
            sums = [sums[1], sums[2], [np.zeros(NT) for _ in range(vx)]]
            last = [last[1], last[2], [[-1] for _ in range(vx)]]
            own = mid
            if zp < zend:
                assert v[0] == zp + 1
                store(K ^ 1, v)
            v = w
    assert np.all(cnt == 1)
    np.testing.assert_array_equal(own_y, x)
    X = np.pad(x.reshape(nz, ny, nx), 1)
    ref = np.zeros((nz, ny, nx))
    for d, (dz, dy, dx) in enumerate(sh):
        ref += c[d] * X[1 + dz:1 + dz + nz, 1 + dy:1 + dy + ny, 1 + dx:1 + dx + nx]
    np.testing.assert_allclose(y, ref.ravel(), rtol=0, atol=1e-12)


@pytest.mark.parametrize("vx", [1, 2])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%s_%dx%dx%d_zc%d" % c)
def test_grid_stream_schedule(case, vx):
    s, nx, ny, nz, zc = case
    run_schedule(s, vx, nx, ny, nz, zc)
