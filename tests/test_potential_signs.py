"""V(r) with Slater exponents whose product with R has no size: c exp(-z R) is c for z = +0 and for z = -0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zeros", [(0.0, 0.0), (-0.0, 0.0), (0.0, -0.0), (-0.0, -0.0)])
def test_slater_terms_with_zero_exponents(pg, clusters, zeros):
    torch = pytest.importorskip("torch")
    grid = pg.Grid((7, 6, 5), 9.0)
    t = pg.WaterTables(clusters.water_cluster(1, 3.0, seed=1))
    core = t.sto.reshape(-1, 2)
    core[:, 0] = 60.0 / 1e-3  # beyond the cut everywhere but on a site
    core[:2] = [[zeros[0], 0.75], [zeros[1], -0.5]]  # the two terms of the first site
    _, parts = grid.potential(t, parts=True)
    rep = parts.view(4, -1)[2]
    assert torch.equal(rep, torch.full_like(rep, 0.25)), (rep.min(), rep.max())
