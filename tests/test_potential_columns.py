"""V(r) by columns of one, two and four points per thread, against extended precision.

A part may be off by (ns + 20) 2^-53 of the sum of its terms' magnitudes: ns
additions, and a dozen roundings inside a term (the steepest one, R^-4, takes
the distance's own rounding four times).  A Slater term beyond z R = 50 is
left out.
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


def reff(r, r0):
    if not r0 > 0:
        return r
    q = np.minimum(r / LD(r0), 1)
    return np.where(r < r0, LD(r0) * (LD(0.5) + q ** 3 * (1 - LD(0.5) * q)), r)


def parts_of(grid, t):
    """(parts, magnitudes) in extended precision from the tables of t."""
    T = t.table
    ax = [a.astype(LD) for a in grid.points()]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    P, M = [[np.zeros(grid.N, dtype=LD) for _ in range(4)] for _ in range(2)]
    sites = t.sites.reshape(-1, 3)

    def distance(s):
        d = [(a - LD(c)).reshape(-1) for a, c in zip((x, y, z), sites[s])]
        return d, np.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)

    for e, s in enumerate(t.charge_site):
        v = -LD(t.charges[e]) / reff(distance(s)[1], T.charge_damp)
        P[0], M[0] = P[0] + v, M[0] + abs(v)
    for e, s in enumerate(t.dipole_site):
        d, r = distance(s)
        w = [a * LD(m) / reff(r, T.dipole_damp) ** 3 for a, m in zip(d, t.dipoles.reshape(-1, 3)[e])]
        P[1], M[1] = P[1] - sum(w), M[1] + sum(abs(q) for q in w)
    for e, s in enumerate(t.sto_site):
        r = distance(s)[1]
        zeta, c = LD(t.sto[2 * e]), LD(t.sto[2 * e + 1])
        v = np.where(zeta * r < 50, c * np.exp(-zeta * r), 0)
        P[2], M[2] = P[2] + v, M[2] + abs(v) * (1 + abs(zeta * r) / 4) + abs(c) * LD(2e-22) * 2 ** 40
    for e, s in enumerate(t.pol_site):
        r = distance(s)[1]
        v = -LD(0.5) * LD(t.pol_alpha[e]) * r ** 2 / reff(r, T.pol_damp) ** 6
        P[3], M[3] = P[3] + v, M[3] + abs(v)
    return P, M


@pytest.mark.parametrize("n,L,nw,what", [(*s, w) for s in (
    ((2, 3, 5), 12.0, 1), ((9, 8, 7), 30.0, 16), ((13, 5, 7), 30.0, 17), ((65, 3, 9), (90.0, 20.0, 25.0), 6))
    for w in ("default", "on a site", "odd parameters", "no damping")] + [
        ((48, 42, 41), 36.0, 2, "default"), ((60, 59, 58), 40.0, 1, "default")])
def test_parts_against_extended_precision(pg, torch, clusters, n, L, nw, what):
    grid = pg.Grid(n, L)
    t = pg.WaterTables(clusters.water_cluster(nw, 3.4 * nw ** (1 / 3), seed=3 + nw))
    if what == "on a site":  # a charge, a dipole and a core at the box centre, a grid point of odd boxes
        t.sites.reshape(-1, 3)[0] = 0.0
        t.sites.reshape(-1, 3)[3] = [0.0, 0.0, 1.0]
    elif what == "odd parameters":  # steep, negative and zero exponents, signs, zero values
        t.sto.reshape(-1, 2)[:3] = [[40.0, 1e3], [-0.05, 1e-3], [0.0, -0.7]]
        t.pol_alpha[0] = -3.0
        t.charges[:2] = [0.0, 1e-9]
        t.dipoles[:9] = 0.0
    elif what == "no damping":
        t.table.charge_damp = t.table.dipole_damp = t.table.pol_damp = 0.0
    v, parts = grid.potential(t, parts=True)
    assert torch.equal(v, grid.potential(t))
    P, M = parts_of(grid, t)
    ns = len(t.sites) // 3
    tol = [(ns + 20) * 2.0 ** -53 * m for m in M]
    for k in range(4):
        off = abs(parts[k].cpu().numpy() - P[k])
        assert np.all(off <= tol[k]), (k, float((off / np.maximum(tol[k], 1e-300)).max()))
    assert np.all(abs(v.cpu().numpy() - sum(P)) <= sum(tol) + 4 * 2.0 ** -53 * sum(abs(p) for p in P))
