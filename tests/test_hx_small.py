"""FP64 H*X on both sides of the rule that gives small grids to the in-order kernel.

At most 36 points over the three axes and one turn of its blocks (250 units of
terms x vectors of a group x turns); beyond, the slices.  Either way a value is
within 37 + 1 roundings of its terms' magnitude.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2, 2, 2), (12, 12, 12), (12, 12, 13), (4, 30, 2), (30, 4, 3), (2, 32, 2)])
@pytest.mark.parametrize("nvec", [1, 3, 4, 7, 90, 100])
@pytest.mark.parametrize("dvrtype", [2, 3])
def test_hx_fp64_on_small_grids(pg, n, nvec, dvrtype):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(sum(n) + nvec)
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n), dvrtype=dvrtype)
    x = rng.standard_normal((nvec, n[2], n[1], n[0]))
    v = rng.standard_normal((1, n[2], n[1], n[0]))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=nvec)
    LD = np.longdouble

    def apply(t, d, q):
        return (d * q + np.einsum("vzyb,ab->vzya", q, t[0]) + np.einsum("vzbx,ab->vzax", q, t[1])
                + np.einsum("vbyx,ab->vayx", q, t[2]))
    T = [g.kinetic(a) for a in range(3)]
    ref = apply([t.astype(LD) for t in T], v.astype(LD), x.astype(LD))
    mag = apply([abs(t) for t in T], abs(v), abs(x))
    # the periodic T is symmetric up to its own rounding, and x reads it by columns
    tol = 38 * 2.0 ** -53 * mag + (2.0 ** -50 * max(abs(t).max() for t in T) * abs(x).sum(-1, keepdims=True)
                                   if dvrtype == 3 else 0.0)
    assert np.all(abs(y.cpu().numpy().reshape(x.shape) - ref) <= tol)
