"""The FP64 products from slices value by value: each against the magnitudes that went through it.

A chain of n FP64 multiply-adds is off by up to n roundings of sum |a x|, of
the point's own terms.  The slices round once, but take the operands as
integers below the largest value of a line and of the matrix, so a point in
the tail of a wavefunction shows what they drop.  Allowed here: 8 x 2^-53 of
the point's own |v x| + sum_axes sum_b |T| |x| -- six roundings of results
(two for the z product with V X, two each for y and x; twice that above 96
points, where the two launches halve the terms) and, at 160 points, 2.7 for the
operands' rounding to 79 bits below their largest values, at T entries of
2^-25.4 of it -- for any vector, with no term in the line's largest value.
On longer sine-DVR axes, whose T reaches further down, as many roundings as
the chain is allowed.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
U = 2.0 ** -53


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def axes_apply(mats, q):
    return (np.einsum("zyb,ab->zya", q, mats[0]) + np.einsum("zbx,ab->zax", q, mats[1])
            + np.einsum("byx,ab->ayx", q, mats[2]))


def vector(kind, n, rng):
    nx, ny, nz = n
    shape = (nz, ny, nx)
    r2 = sum(d ** 2 for d in np.meshgrid(*(0.6 * (np.arange(m) - 0.45 * m) for m in (nz, ny, nx)), indexing="ij"))
    if kind == "unit":
        x = np.zeros(shape)
        x[nz // 2, ny // 2, nx // 3] = 1.0 + 2.0 ** -52
        return x
    if kind == "corner":  # one value at an end of the box
        x = np.zeros(shape)
        x[0, 0, 0] = rng.standard_normal()
        return x
    if kind == "exponential":
        return np.exp(-np.sqrt(r2))
    if kind == "steep":
        return np.exp(-6.0 * np.sqrt(r2))
    return np.exp(-r2 / 60.0) * rng.uniform(0.5, 1.5, size=shape)


@pytest.mark.parametrize("kind", ["unit", "corner", "exponential", "steep", "gaussian"])
@pytest.mark.parametrize("n", [(32, 31, 33), (64, 9, 8), (7, 65, 6), (96, 5, 4), (5, 4, 97), (160, 4, 3), (3, 161, 4),
                               (3, 2, 400), (2, 700, 3), (1000, 2, 2)])
@pytest.mark.parametrize("dvrtype", [2, 3])
def test_hx_fp64_value_by_value(pg, torch, n, kind, dvrtype):
    rng = np.random.default_rng(n[0] + n[2])
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n), dvrtype=dvrtype)
    x = vector(kind, n, rng)
    v = rng.standard_normal((n[2], n[1], n[0]))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=1)
    g.check()
    got = y.cpu().numpy().reshape(x.shape).astype(LD)
    T = [g.kinetic(a).astype(LD) for a in range(3)]
    ref = v.astype(LD) * x + axes_apply(T, x.astype(LD))
    mag = abs(v.astype(LD) * x) + axes_apply([abs(t) for t in T], abs(x).astype(LD))
    # above 160 points of a sine DVR the smallest entries of T lose bits: within the chain's n roundings
    tol = (8 if dvrtype == 3 or max(n) <= 160 else sum(n)) * U * mag
    assert np.all(abs(got - ref) <= tol), float((abs(got - ref) / np.maximum(U * mag, 1e-4000)).max())


@pytest.mark.parametrize("n", [48, 96, 159, 162])
@pytest.mark.parametrize("bits,last", [(8, 10), (8, 4), (9, 7), (9, 6), (9, 4)])
def test_coherent_digits(pg, torch, clusters, n, bits, last):
    """Every digit product of one sign and as large as it can be, over all n values: the accumulators' worst case.

    Polarisable sites so far away that the field at them is epc alone: E = c in every component, A = a in every
    entry, V = -n^2 c^2 a / 2, c and a with `last` leading digits of `bits` bits at their maximum.  One rounding per
    launch of 96 values, and the sum of n equal terms in chains of at most 48: 60 roundings."""
    def value(scale):
        f = sum(((1 << (bits - 1)) - 1) << (bits * (last - 1 - i)) for i in range(last))
        while f >> 53:  # the leading 53 bits
            f >>= 1
        return scale * float(f) / 2.0 ** f.bit_length()
    c, a = value(1.0), value(4.0)
    w = clusters.water_cluster(n // 9 + 1, 30.0, seed=3)
    tables = pg.WaterTables(w)
    npp = n // 3
    tables.sites[:] = 1e100
    m = pg.ScPol(tables=tables, pol_site=np.arange(npp, dtype=np.int32), inva=np.full((n, n), a),
                 epc=np.full(n, c), vpol_ww=0.0)
    grid = pg.Grid((5, 6, 7), 12.0)
    v = grid.scpol_add(m, torch.zeros(grid.N, dtype=torch.float64, device="cuda")).cpu().numpy()
    ref = -LD(0.5) * n * n * LD(c) * LD(c) * LD(a)
    err = float((abs(v - ref) / abs(ref)).max() / U)
    assert err <= 60, err
