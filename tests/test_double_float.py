"""The mixed block products at the edges of their double-float arithmetic and of their tiles.

A row s and a row e combined with coefficients 1 give the pair (s + e rounded
to FP32, its error), which is exact, so the FP64 result must be s + e rounded
once: what numpy's FP64 addition gives.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def edge_pairs():
    s, e = [], []
    f = np.float32
    for k in (-100, -76, -75, -74, -40, -1, 0, 1, 60, 126):
        for m in (1.0, 1.0 + 2.0 ** -23, 1.5, 2.0 - 2.0 ** -23):
            for j in (24, 25, 29, 30, 51, 52, 53, 54, 55, 60):
                for r in (1.0, 1.5, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23):
                    for sg in (1.0, -1.0):
                        s.append(f(m * 2.0 ** k)), e.append(f(sg * r * 2.0 ** max(k - j, -125)))
                        s.append(-s[-1]), e.append(e[-1])
            s.append(f(m * 2.0 ** k)), e.append(f(-m * 2.0 ** k))            # cancels to zero
            s.append(f(m * 2.0 ** k)), e.append(f(-m * (1 - 2.0 ** -20) * 2.0 ** k))  # to few bits
    s += [f(0), f(0), f(3e38), f(2.0 ** -126), f(np.inf), f(-np.inf), f(np.nan), f(1)]
    e += [f(0), f(1e-30), f(1e30), f(-2.0 ** -126), f(1), f(2), f(1), f(np.nan)]
    return np.array(s, np.float64), np.array(e, np.float64)


@pytest.mark.parametrize("nr", [1, 2, 3, 4, 7, 8, 12, 16])
def test_combine_mixed_rounds_the_pair_once(pg, nr):
    torch = pytest.importorskip("torch")
    s, e = edge_pairs()
    P = torch.as_tensor(np.stack([s, e]), device="cuda")
    C = torch.ones(2, nr, dtype=torch.float64, device="cuda")
    got = pg.block_combine(P, C, precision=1).cpu().numpy().reshape(nr, -1)
    with np.errstate(invalid="ignore"):
        want = s + e
    for r in range(nr):
        same = (got[r] == want) | (~np.isfinite(want) & ~np.isfinite(got[r]))
        assert same.all(), (s[~same][:4], e[~same][:4], got[r][~same][:4])


# rows of odd length (no pairs of points) and even; products of 1 to 16 output
# blocks' shapes; against extended precision: the sum's own error is below
# 2^-47 for each of at most 150 points a thread adds up
@pytest.mark.parametrize("rows", [(1, 1), (8, 1), (20, 1), (16, 4), (56, 8), (57, 9), (96, 4), (120, 16)])
@pytest.mark.parametrize("n", [1, 2, 37, 1000, 9473, 20000])
def test_block_products_mixed_tiles(pg, rows, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + rows[0])
    P, Q = (rng.standard_normal((k, n)) for k in rows)
    Pd, Qd = torch.as_tensor(P, device="cuda"), torch.as_tensor(Q, device="cuda")
    got = pg.block_gram(Pd, Qd, precision=1)
    # rows already split are copied, not converted: the same values
    twin = pg.block_gram_twin(pg.split_twin(Pd), pg.split_twin(Qd))
    assert torch.equal(got, twin)
    got = got.cpu().numpy().reshape(rows)
    for q in range(rows[1]):
        terms = P.astype(LD) * Q[q].astype(LD)
        assert np.all(abs(got[:, q] - terms.sum(axis=1)) <= 150 * 2.0 ** -47 * abs(terms).sum(axis=1))
    C = rng.standard_normal(rows)
    Cd = torch.as_tensor(C, device="cuda")
    y = pg.block_combine(Pd, Cd, precision=1)
    assert torch.equal(y, pg.block_combine_twin(pg.split_twin(Pd), Cd))
    ref = np.stack([(C[:, r][:, None].astype(LD) * P.astype(LD)).sum(axis=0) for r in range(rows[1])])
    mag = np.stack([abs(C[:, r][:, None] * P).sum(axis=0) for r in range(rows[1])])
    assert np.all(abs(y.cpu().numpy().reshape(ref.shape) - ref) <= 150 * 2.0 ** -47 * mag)


@pytest.mark.parametrize("nr", range(1, 17))
@pytest.mark.parametrize("precision", [0, 1])
def test_combine_columns_do_not_depend_on_their_number(pg, nr, precision):
    """A column of a block combine has the bits of the same column on its own (each count of columns has a kernel)."""
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda").manual_seed(nr)
    P = torch.randn(19, 5003, dtype=torch.float64, device="cuda", generator=gen)
    C = torch.randn(19, nr, dtype=torch.float64, device="cuda", generator=gen)
    y = pg.block_combine(P, C, precision=precision).reshape(nr, -1)
    for r in {0, nr // 2, nr - 1}:
        one = pg.block_combine(P, C[:, r:r + 1].contiguous(), precision=precision).reshape(-1)
        assert torch.equal(y[r], one)
