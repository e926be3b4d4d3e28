"""V(r) of the self-consistent polarisation: the row dots E . (E A) from exact slices against extended precision.

A component of E is off by a dozen roundings (distance, its cube, the
products), the matrix product by one, the row dot by one per term of its
column chunk, and the sum into V by four: 40 x 2^-53 of sum |E| |A| |E|, plus
what the charges and cores carry.  Sizes lie at the edges of the matrix
images: one and two K chunks of 80, column chunks of 64, launches of 160.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def model_of(pg, clusters, nw, seed, change=None):
    w = clusters.water_cluster(nw, 3.4 * nw ** (1 / 3), seed=seed)
    tables = pg.WaterTables(w)
    rng = np.random.default_rng(seed)
    npp = 3 * nw
    a = rng.standard_normal((3 * npp, 3 * npp)) * 10.0 ** rng.uniform(-3, 0, size=(3 * npp, 1))
    a = a + a.T + np.diag(rng.uniform(1, 9, 3 * npp))
    if change:
        change(a)
    ps = (4 * np.arange(nw)[:, None] + [0, 1, 2]).reshape(-1)
    return pg.ScPol(tables=tables, pol_site=ps, inva=a, epc=rng.normal(scale=0.02, size=3 * npp), vpol_ww=-0.03)


def field(grid, m):
    pos = m.base.sites.reshape(-1, 3)[m.pol_site].astype(LD)
    ax = [a.astype(LD) for a in grid.points()]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    d = np.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)[:, None, :] - pos[None]
    r = np.sqrt((d * d).sum(-1))
    r0 = LD(m.model.damp)
    q = np.minimum(r / r0, 1)
    re = np.where(r < r0, r0 * (LD(0.5) + q ** 3 * (1 - LD(0.5) * q)), r)
    return (d / re[:, :, None] ** 3).reshape(len(d), -1) + m.epc.astype(LD)[None]


@pytest.mark.parametrize("nw,n", [(1, (3, 4, 5)), (2, (13, 11, 9)), (7, (5, 5, 5)), (8, (16, 9, 8)), (9, (7, 3, 6)),
                                  (17, (9, 5, 6)), (18, (8, 9, 2))])
def test_scpol_against_extended_precision(pg, torch, clusters, nw, n):
    grid = pg.Grid(n, tuple(6.0 + 1.5 * k for k in n))
    m = model_of(pg, clusters, nw, 5 + nw)
    v0 = torch.zeros(grid.N, dtype=torch.float64, device="cuda")
    v = grid.scpol_add(m, v0.clone()).cpu().numpy()
    E, A = field(grid, m), m.inva.astype(LD)
    ref = -LD(0.5) * (E * (E @ A)).sum(1) - LD(m.vpol_ww)
    tol = 40 * 2.0 ** -53 * (0.5 * (abs(E) * (abs(E) @ abs(A))).sum(1) + abs(LD(m.vpol_ww)))
    assert np.all(abs(v - ref) <= tol), float((abs(v - ref) / tol).max())
    assert torch.equal(grid.scpol_add(m, v0.clone()).cpu(), torch.as_tensor(v))


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e250, 0.0])
def test_matrix_outside_the_slices_range(pg, torch, clusters, value):
    """Infinite, NaN, huge and zero matrices: what FP64 multiply-adds give."""
    def change(a):
        if value == 0.0:
            a[:] = 0.0
        else:
            a[2, 3] = a[3, 2] = value
    grid = pg.Grid((5, 6, 7), 12.0)
    m = model_of(pg, clusters, 2, 3, change)
    v = grid.scpol_add(m, torch.zeros(grid.N, dtype=torch.float64, device="cuda")).cpu().numpy()
    E = field(grid, m).astype(np.float64)
    with np.errstate(invalid="ignore", over="ignore"):
        ref = -0.5 * (E * (E @ m.inva)).sum(1) - m.vpol_ww
    assert np.array_equal(np.isfinite(v), np.isfinite(ref)) and np.array_equal(np.isnan(v), np.isnan(ref))
    f = np.isfinite(ref)
    assert not f.any() or np.all(np.abs(v[f] - ref[f]) <= 1e-12 * np.abs(ref[f]).max())
