"""The FP64 axis contraction from exact slices (k_slice_axis) against extended precision.

H*X is three contractions, each rounded once where it joins the sum, so a
value may be off by four roundings of the magnitude that went through it:
4 x 2^-53 (|v x| + sum_axes sum_b |T| |x|), plus the slices' own 2^-55.
Sizes lie at the edges of the kernel: MMA rows and K steps of 16, column
chunks of 64, K chunks of 80, launches of two K chunks, tiles of 128 lines.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def hx_terms(T, v, x):
    """(H x, the magnitudes summed) in extended precision, x[vector, z, y, x]."""
    def apply(mats, d, q):
        out = d * q
        for r in range(len(q)):
            out[r] += np.einsum("zyb,ab->zya", q[r], mats[0]) + np.einsum("zbx,ab->zax", q[r], mats[1]) \
                + np.einsum("byx,ab->ayx", q[r], mats[2])
        return out
    t = [m.astype(LD) for m in T]
    return apply(t, v.astype(LD), x.astype(LD)), apply([abs(m) for m in t], abs(v).astype(LD), abs(x).astype(LD))


@pytest.mark.parametrize("n,nvec", [
    ((2, 3, 5), 1), ((16, 8, 8), 2), ((15, 17, 16), 1), ((31, 33, 32), 3), ((63, 5, 64), 1), ((65, 6, 7), 2),
    ((79, 4, 80), 1), ((81, 5, 9), 1), ((96, 8, 4), 1), ((4, 129, 3), 1), ((5, 6, 160), 1), ((3, 161, 4), 2),
    ((330, 3, 4), 1)])
@pytest.mark.parametrize("kind", ["random", "smooth", "graded"])
def test_hx_fp64_against_extended_precision(pg, torch, n, nvec, kind):
    rng = np.random.default_rng(n[0] * 1000 + n[2])
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    x = rng.standard_normal((nvec, n[2], n[1], n[0]))
    if kind == "smooth":
        ax = g.points()
        r2 = ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2
        x = np.stack([np.exp(-r2 / (9 + 4 * j)) for j in range(nvec)])
    elif kind == "graded":  # lines of very different size, and exact zeros
        x *= 10.0 ** rng.integers(-120, 120, size=(nvec, n[2], n[1], 1))
        x[:, 0, :, :] = 0.0
    v = rng.standard_normal((1, n[2], n[1], n[0]))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=nvec)
    g.check()
    ref, mag = hx_terms([g.kinetic(a) for a in range(3)], v, x)
    got = y.cpu().numpy().reshape(ref.shape).astype(LD)
    # the slices of a line: quantised to 2^-62 of its largest value, and the
    # digit products left out (six of 2^-63 scale for each of up to 160
    # values: 2^-58 standard deviation, 2^-55 at six of them)
    big = np.maximum.reduce([abs(x).max(axis=a, keepdims=True) * np.ones_like(x) for a in (1, 2, 3)])
    tol = 4.0 * 2.0 ** -53 * mag + 2.0 ** -55 * max(abs(g.kinetic(a)).sum(axis=1).max() for a in range(3)) * big
    assert np.all(abs(got - ref) <= tol), float((abs(got - ref) / np.maximum(tol, 1e-300)).max())


@pytest.mark.parametrize("what", ["inf", "nan", "tiny", "huge"])
def test_lines_outside_the_slices_range(pg, torch, what):
    """Infinities, NaN, subnormal and huge values go through FP64 multiply-adds, line by line."""
    n = (24, 20, 28)
    rng = np.random.default_rng(5)
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    x = rng.standard_normal((1, n[2], n[1], n[0]))
    if what == "inf":
        x[0, 3, 4, 5] = np.inf
    elif what == "nan":
        x[0, 7, 1, 2] = np.nan
    else:
        x *= 1e-309 if what == "tiny" else 1e300
    v = rng.standard_normal((1, n[2], n[1], n[0]))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=1)
    g.check()
    got = y.cpu().numpy().reshape(x.shape)
    T = [g.kinetic(a) for a in range(3)]
    with np.errstate(invalid="ignore", over="ignore"):
        ref = v * x + np.einsum("vzyb,ab->vzya", x, T[0]) + np.einsum("vzbx,ab->vzax", x, T[1]) \
            + np.einsum("vbyx,ab->vayx", x, T[2])
    fine = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fine) and np.array_equal(np.isnan(got), np.isnan(ref))
    # 72 terms a point, each a rounding of what went through it
    size = max(np.abs(m).sum(axis=1).max() for m in T) * 3 * np.abs(x[np.isfinite(x)]).max()
    assert np.all(np.abs(got[fine] - ref[fine]) <= 76 * 2.0 ** -53 * size + 76 * 5e-324)
