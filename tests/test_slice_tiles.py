"""The FP64 axis contraction over many lines: full tiles of 128, 64 and 32
lines, column chunks that reuse a buffer and a set of accumulators, the narrow
transposition of long axes, and K chunks with full tiles.

Checked against extended precision at sampled points, among them the last
line.  The tolerance is that of the same product on small grids: four
roundings of what goes through a value and the slices' 2^-55 of the largest.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


# many lines: tiles of 128 on every axis, or of 64 and 32 on the short ones;
# then fewer, where a tile's column chunks go to blocks of their own (64, 96
# with two chunks to a block, 160 in K chunks too)
@pytest.mark.parametrize("n,nvec", [((17, 100, 100), 1), ((96, 72, 71), 2), ((80, 80, 80), 3), ((97, 50, 200), 1),
                                    ((33, 64, 152), 1), ((33, 64, 153), 1), ((50, 64, 76), 1), ((50, 48, 102), 1),
                                    ((64, 64, 64), 1), ((96, 60, 80), 1), ((160, 48, 50), 1)])
def test_hx_fp64_over_many_lines(pg, n, nvec):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n[0] * 1000 + n[2])
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    nx, ny, nz = n
    x = rng.standard_normal((nvec, nz, ny, nx))
    v = rng.standard_normal((nz, ny, nx))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=nvec)
    g.check()
    got = y.cpu().numpy().reshape(x.shape)
    T = [g.kinetic(a) for a in range(3)]
    r, k, j, i = (rng.integers(0, m, size=2000) for m in (nvec, nz, ny, nx))
    last = np.arange(nx)
    r, k, j, i = (np.concatenate(p) for p in ((r, np.full(nx, nvec - 1)), (k, np.full(nx, nz - 1)),
                                              (j, np.full(nx, ny - 1)), (i, last)))
    ref, mag = np.zeros(len(r), LD), np.zeros(len(r), LD)
    lines = ((T[0][i], x[r, k, j, :]), (T[1][j], x[r, k, :, i]), (T[2][k], x[r, :, j, i]))
    for t, line in lines + ((v[k, j, i][:, None], x[r, k, j, i][:, None]),):
        p = t.astype(LD) * line.astype(LD)
        ref += p.sum(axis=1)
        mag += abs(p).sum(axis=1)
    big = max(abs(t).sum(axis=1).max() for t in T) * np.max([abs(line).max(axis=1) for _, line in lines], axis=0)
    tol = 4.0 * 2.0 ** -53 * mag + 2.0 ** -55 * big
    bad = abs(got[r, k, j, i].astype(LD) - ref)
    assert np.all(bad <= tol), float((bad / tol).max())
