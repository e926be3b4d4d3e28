"""The FP16 kinetic preconditioner with several planes to a work item (n <= 64, more planes than SMs) against one
plane to an item (a single vector): every plane keeps its own scale and the order of its sums, so the results are bit
for bit.  Sizes at the edges: a last item of 1 to 4 planes, padded rows, both eigenbases, and planes of very
different size, zeros and subnormals among them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nvec,dvrtype", [(64, 5, 2), (62, 3, 2), (50, 4, 2), (34, 6, 2), (34, 40, 2), (32, 9, 2),
                                            (30, 12, 2), (18, 32, 2), (14, 17, 2), (32, 12, 3), (64, 4, 3)])
def test_block_equals_single_vectors(pg, n, nvec, dvrtype):
    import torch
    g = pg.Grid(n, 0.6 * (n + 1), dvrtype=dvrtype)
    assert "k_kin_f16" in g.precond_plan() and nvec * n > 152
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(nvec, n, n * n, dtype=torch.float64, device="cuda", generator=gen)
    x *= 10.0 ** torch.linspace(-12, 12, n, dtype=torch.float64, device="cuda")[None, :, None]
    x[0, :3] = 0.0
    x[-1, 1] *= 1e-300
    x[-1, 2, :5] = 1e-310
    x = x.reshape(nvec, -1)
    sigma = [-0.2 + 0.01 * j for j in range(nvec)]
    y = x.clone()
    g.precondition(y.view(-1), sigma, precision=pg.PG_MIXED)
    for j in (0, nvec // 2, nvec - 1):
        one = x[j].clone()
        g.precondition(one, sigma[j:j + 1], precision=pg.PG_MIXED)
        assert torch.equal(y[j], one)
