"""The in-order FP64 kernels over any number of vectors: each vector has the bits of a call of its own.

Vectors go in groups of four, and the one to three that are left in a group of
their own beside them: 1 to 9 vectors meet every combination.  FP64 solves of
several states are what runs them; a sine-DVR axis above about 750 points
brings pg_hx to them too.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvec", range(1, 10))
@pytest.mark.parametrize("n", [(2, 2, 1000), (800, 3, 2)])
def test_vectors_are_independent(pg, n, nvec):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nvec)
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    x = torch.as_tensor(rng.standard_normal((nvec, g.N)), device="cuda")
    v = torch.as_tensor(rng.standard_normal(g.N), device="cuda")
    y = g.hx(v, x.reshape(-1), nvec=nvec).view(nvec, g.N)
    for q in range(nvec):
        assert torch.equal(y[q], g.hx(v, x[q].contiguous(), nvec=1))
    # a chain of sum(n) + 1 multiply-adds a value
    T = [g.kinetic(a) for a in range(3)]
    X, V = x.cpu().numpy().reshape(nvec, n[2], n[1], n[0]), v.cpu().numpy().reshape(1, n[2], n[1], n[0])

    def apply(t, d, q):
        return (d * q + np.einsum("vzyb,ab->vzya", q, t[0]) + np.einsum("vzbx,ab->vzax", q, t[1])
                + np.einsum("vbyx,ab->vayx", q, t[2]))
    LD = np.longdouble
    ref = apply([t.astype(LD) for t in T], V.astype(LD), X.astype(LD))
    mag = apply([abs(t) for t in T], abs(V), abs(X))
    assert np.all(abs(y.cpu().numpy().reshape(X.shape) - ref) <= (sum(n) + 1) * 2.0 ** -53 * mag)
