"""The FP64 block Gram product at the edges of its tiles, against extended precision.

A value is a sum of chains of 8 multiply-adds, 2 additions, one per tile of 32
points of a block and one per 32 blocks and 5 more: at most 8 + 2 + 4 + 10 + 5
roundings in a row at these sizes, so the error is at most 32 x 2^-53 of the
sum of the terms' magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


# 4, 2 and 1 tiles of 32 points at a time (by rows and outputs); points at the
# edges of a tile, of the tiles held at a time and of a block's share
@pytest.mark.parametrize("rows", [(1, 1), (20, 1), (40, 4), (51, 2), (56, 8), (96, 4), (120, 16), (128, 16)])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 9472, 9473, 37889])
def test_block_gram_fp64_tiles(pg, rows, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + rows[0])
    P = rng.standard_normal((rows[0], n)) * 10.0 ** rng.integers(-3, 3, size=(rows[0], 1))
    Q = rng.standard_normal((rows[1], n))
    got = pg.block_gram(torch.as_tensor(P, device="cuda"), torch.as_tensor(Q, device="cuda"), precision=0)
    got = got.cpu().numpy().reshape(rows)
    for q in range(rows[1]):
        terms = P.astype(LD) * Q[q].astype(LD)
        assert np.all(abs(got[:, q] - terms.sum(axis=1)) <= 32 * 2.0 ** -53 * abs(terms).sum(axis=1))
