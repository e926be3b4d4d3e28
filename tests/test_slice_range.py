"""The FP64 products from slices at the ends of FP64's range, and with matrices of very different columns.

The slices of a line and of the matrix each have a scale of their own; the
result's exponent is the sum of both, and it has to stay that of a normal
number.  Lines and matrices for which it may not, and columns that one scale
for the whole matrix would cut, go through FP64 multiply-adds.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


# T about 1e195, 1e-119, 1e280 (no slices), 1e-290 (no slices)
@pytest.mark.parametrize("L,size,expect", [(1e-95, 1e250, "overflow"), (1e60, 1e-210, "underflow"),
                                           (1e-138, 1e60, "overflow"), (1e146, 1e-60, "underflow"),
                                           (1e-95, 1e-200, "normal"), (1e60, 1e120, "normal"),
                                           (1e-138, 1e-60, "normal"), (1e146, 1e60, "normal")])
def test_hx_fp64_at_the_ends_of_the_range(pg, torch, L, size, expect):
    n = (8, 70, 9)
    rng = np.random.default_rng(3)
    g = pg.Grid(n, L)
    x = rng.uniform(1.0, 2.0, size=(n[2], n[1], n[0])) * size
    v = torch.zeros(g.N, dtype=torch.float64, device="cuda")
    y = g.hx(v, torch.as_tensor(x.reshape(-1), device="cuda"), nvec=1)
    g.check()
    got = y.cpu().numpy().reshape(x.shape)
    T = [g.kinetic(a) for a in range(3)]
    if expect == "overflow":  # products alone pass the largest FP64 number
        assert not np.isfinite(got).any()
        return
    if expect == "underflow":  # 87 products of at most 2^-1022, rounded or flushed
        assert np.all(np.abs(got) <= 87 * 2.0 ** -1022)
        return
    one = x / size
    ref = np.einsum("zyb,ab->zya", one, T[0]) + np.einsum("zbx,ab->zax", one, T[1]) + np.einsum("byx,ab->ayx", one, T[2])
    mag = sum(np.abs(t).sum(axis=1).max() for t in T) * 2.0
    # 87 + 87 multiply-adds of either side, and the scale
    assert np.all(np.abs(got / size - ref) <= 200 * 2.0 ** -53 * mag)


def far_model(pg, clusters, npp, inva, epc):
    """Sites so far away that the field at them is epc alone."""
    tables = pg.WaterTables(clusters.water_cluster(npp // 3 + 1, 20.0, seed=3))
    tables.sites[:] = 1e100
    return pg.ScPol(tables=tables, pol_site=np.arange(npp, dtype=np.int32), inva=inva, epc=epc, vpol_ww=0.0)


@pytest.mark.parametrize("a,e", [(1e190, 1e260), (1e-190, 1e-260), (1e100, 1e30), (1e-280, 1e3)])
def test_row_dots_at_the_ends_of_the_range(pg, torch, clusters, a, e):
    grid = pg.Grid((5, 6, 7), 12.0)
    n = 24
    m = far_model(pg, clusters, n // 3, np.full((n, n), a), np.full(n, e))
    v = grid.scpol_add(m, torch.zeros(grid.N, dtype=torch.float64, device="cuda")).cpu().numpy()
    with np.errstate(over="ignore", under="ignore"):
        ref = -0.5 * np.float64(n * e) * (np.float64(n * e) * np.float64(a))
    if np.isinf(ref):
        assert np.all(v == ref)
    else:
        assert np.all(np.abs(v - ref) <= 60 * 2.0 ** -53 * abs(ref) + n * n * 2.0 ** -1022)


@pytest.mark.parametrize("ratio", [2.0 ** -12, 2.0 ** -30, 2.0 ** -70, 2.0 ** -120])
def test_columns_of_very_different_size(pg, torch, clusters, ratio):
    """Half of the columns a factor smaller, and a field that meets only them: V is theirs alone.

    V = -sum E_k A_kc E_c / 2 with E zero but in the small columns: one
    rounding of each product sum, chains of 24 equal terms: 30 roundings."""
    grid = pg.Grid((5, 6, 7), 12.0)
    n, h = 24, 12
    inva = np.full((n, n), 1.0 / 3.0)
    inva[h:, h:] *= ratio
    inva[:h, h:] *= ratio
    epc = np.zeros(n)
    epc[h:] = 0.7
    v = grid.scpol_add(far_model(pg, clusters, n // 3, inva, epc),
                       torch.zeros(grid.N, dtype=torch.float64, device="cuda")).cpu().numpy()
    ref = -0.5 * (h * 0.7) ** 2 / 3.0 * ratio
    assert np.all(np.abs(v - ref) <= 30 * 2.0 ** -53 * abs(ref)), float(np.abs(v / ref - 1).max() * 2 ** 53)
