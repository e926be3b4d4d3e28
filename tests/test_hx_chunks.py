"""Mixed H*X on axes of more than 112 points (several K chunks): a block of many tiles runs two CTAs per SM, a
single vector one; the order of the sums is the same, so the results are bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nvec", [((130, 40, 39), 14), ((33, 128, 40), 16), ((20, 36, 161), 28), ((256, 16, 9), 140)])
def test_block_equals_single_vectors(pg, n, nvec):
    import torch
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    assert g.N // max(n) * nvec > 152 * 128  # more tiles than SMs along the long axis
    gen = torch.Generator(device="cuda").manual_seed(n[0])
    x = torch.randn(nvec, g.N, dtype=torch.float64, device="cuda", generator=gen)
    x[0, :7] *= 1e-36  # products down to subnormal FP32
    v = torch.randn(g.N, dtype=torch.float64, device="cuda", generator=gen)
    y = g.hx(v, x.reshape(-1), nvec=nvec, precision=pg.PG_MIXED).view(nvec, -1)
    for j in (0, nvec // 2, nvec - 1):
        assert torch.equal(y[j], g.hx(v, x[j].contiguous(), nvec=1, precision=pg.PG_MIXED))
    ref = g.hx(v, x.reshape(-1), nvec=nvec, precision=pg.PG_FP64).view(nvec, -1)
    # the mixed form's bound (TF32 split, FP32 accumulation)
    assert float((y - ref).abs().max()) <= 2e-5 * float(ref.abs().max())
