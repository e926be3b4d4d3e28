"""Mixed H*X by axis with one to two tiles per SM (two blocks per SM, the axis matrix resident, the input in K
chunks) against single vectors (one tile per block, one K chunk): the order of the sums is the same, so the results
are bit for bit.  Axes at the edges of the chunks (40 and 41, 48 and 49, 72, 80, 81, 96 and 97 points)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nvec", [((40, 41, 48), 16), ((49, 72, 64), 7), ((72, 80, 81), 4), ((96, 90, 97), 3),
                                    ((17, 96, 33), 18), ((24, 26, 25), 56)])
def test_block_equals_single_vectors(pg, n, nvec):
    import torch
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    g.set_hx_kernel(1)
    assert any(152 < -(-(g.N // m * nvec) // 128) <= 304 for m in n)  # tiles of some axis
    gen = torch.Generator(device="cuda").manual_seed(n[0])
    x = torch.randn(nvec, g.N, dtype=torch.float64, device="cuda", generator=gen)
    x[0, :7] *= 1e-36  # products down to subnormal FP32
    v = torch.randn(g.N, dtype=torch.float64, device="cuda", generator=gen)
    y = g.hx(v, x.reshape(-1), nvec=nvec, precision=pg.PG_MIXED).view(nvec, -1)
    for j in (0, nvec // 2, nvec - 1):
        assert torch.equal(y[j], g.hx(v, x[j].contiguous(), nvec=1, precision=pg.PG_MIXED))
    sigma = [-0.2 + 0.01 * j for j in range(nvec)]
    r = x.clone()
    g.precondition(r.view(-1), sigma, precision=pg.PG_MIXED)
    one = x[nvec - 1].clone()
    g.precondition(one, sigma[-1:], precision=pg.PG_MIXED)
    assert torch.equal(r[nvec - 1], one)
