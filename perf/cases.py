"""The measured workload: the calls a user of this package makes, over the sizes they are made at.

A single point of an excess electron on a water cluster is V(r) on the grid (the one-site or the
self-consistent polarisation model), then a Davidson solve; the solve is H*X products, kinetic
preconditioning of residuals and skinny block products (Gram and combine), each of which is a public
entry point of its own that the reference's classes and other solvers call.  Sizes are those of the
configurations (32^3 with 6 waters, 64^3 with 24, 96^3 with 32, 160^3 with 16 states; serving grids of
48 to 96 points per axis and 1 to 4 states) and ragged boxes in between.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package folder has a dash in its name: imported as pisces_gb300 by its place."""
    if "pisces_gb300" not in sys.modules:
        folder = os.path.join(ROOT, "pisces-1_gb300")
        spec = importlib.util.spec_from_file_location("pisces_gb300", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pisces_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["pisces_gb300"]


# ------------------------------------------------------------------ the cases

def listed():
    def grid(nx, ny=None, nz=None):
        return {"nx": nx, "ny": ny or nx, "nz": nz or nx}

    return [
        # the drop-in matrix-vector product, one vector at a time on the smallest configured grid: latency
        {"name": "hx fp64 32^3 x1", "op": "hx", **grid(32), "nvec": 1, "prec": "fp64"},
        # the drop-in form on a box with three different, ragged axes and a block of vectors
        {"name": "hx fp64 83x90x71 x6", "op": "hx", **grid(83, 90, 71), "nvec": 6, "prec": "fp64"},
        # the mixed form on the 64^3, four-state configuration: one product per Davidson iteration
        {"name": "hx mixed 64^3 x4", "op": "hx", **grid(64), "nvec": 4, "prec": "mixed"},
        # the largest configuration's block product
        {"name": "hx mixed 160^3 x16", "op": "hx", **grid(160), "nvec": 16, "prec": "mixed"},
        # the kinetic preconditioner of the mixed solve (corrflag 3), one call per iteration
        {"name": "precond mixed 64^3 x4", "op": "precond", **grid(64), "nvec": 4, "prec": "mixed"},
        # the same of the FP64 solve on an 80^3 serving grid
        {"name": "precond fp64 80^3 x3", "op": "precond", **grid(80), "nvec": 3, "prec": "fp64"},
        # subspace products of the FP64 solve: 40 basis vectors against a block of 4 on 64^3
        {"name": "block fp64 64^3 40x4", "op": "block", "npoints": 64 ** 3, "na": 40, "nb": 4, "prec": "fp64"},
        # and of the mixed solve at the 96^3, eight-state configuration
        {"name": "block mixed 96^3 56x8", "op": "block", "npoints": 96 ** 3, "na": 56, "nb": 8, "prec": "mixed"},
        # V(r) with its energy parts, the 24-water configuration
        {"name": "potential 64^3 w24", "op": "potential", **grid(64), "nw": 24},
        # V(r) of the self-consistent polarisation model on a small serving grid
        {"name": "scpol 48^3 w8", "op": "scpol", **grid(48), "nw": 8},
        # a whole single point with the defaults: FP64, diagonal correction, one state
        {"name": "point fp64 32^3 w6", "op": "point", **grid(32), "nw": 6, "nroots": 1, "maxsub": 20, "ptol": 5,
         "corrflag": 1, "prec": "fp64"},
        # a whole single point in the mixed form, four states (the benchmark's configuration)
        {"name": "point mixed 64^3 w24 x4", "op": "point", **grid(64), "nw": 24, "nroots": 4, "maxsub": 60, "ptol": 6,
         "corrflag": 3, "prec": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["hx", "hx", "hx", "precond", "precond", "block", "block", "potential", "scpol", "point"])
    prec = rng.choice(["fp64", "mixed"])
    cubic = rng.random() < 0.5
    axes = [_log_int(rng, 24, 104) for _ in range(3)]
    n = [axes[0]] * 3 if cubic else axes
    size = {"nx": n[0], "ny": n[1], "nz": n[2]}
    if op in ("hx", "precond"):
        return {"op": op, **size, "nvec": rng.randint(1, 10), "prec": prec}
    if op == "block":
        nb = rng.randint(1, 12)
        na = rng.randint(nb, 64)
        return {"op": op, "npoints": _log_int(rng, 15000, 900000), "na": na, "nb": nb, "prec": prec}
    if op == "potential":
        return {"op": op, **size, "nw": _log_int(rng, 2, 48)}
    if op == "scpol":
        m = [min(v, 64) for v in n]
        return {"op": op, "nx": m[0], "ny": m[1], "nz": m[2], "nw": _log_int(rng, 2, 16)}
    # serving-like single points: cubes of 32 to 64 points, one to three states
    m = rng.choice([32, 40, 45, 48, 56, 60, 64])
    nroots = rng.randint(1, 3)
    return {"op": "point", "nx": m, "ny": m, "nz": m, "nw": rng.randint(8, 24), "nroots": nroots,
            "maxsub": 24 + 8 * nroots, "ptol": 6, "corrflag": 3, "prec": prec}


# ------------------------------------------------------------------ inputs

SPACING = 40.0 / 65.0  # bohr between grid points, the 64^3 configuration's


def _n(case):
    return (case["nx"], case["ny"], case["nz"])


def _box(case):
    """Box lengths in bohr: the configurations' spacing, and for clusters room around them."""
    return tuple(SPACING * (m + 1) if "nw" not in case else max(SPACING * (m + 1), _radius(case["nw"]) * 2 + 8.0)
                 for m in _n(case))


def _radius(nw):
    """Radius (bohr) of the sphere that holds nw oxygens, near the configurations' density."""
    return 3.15 * nw ** (1.0 / 3.0) / 0.52917720859


def _water_lists(nw, seed):
    """Sites (O, H, H, M of each water, bohr), charges and induced dipoles of a seeded rigid-water cluster."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 11]))
    a2b = 1.0 / 0.52917720859
    half = np.deg2rad(104.52) / 2.0
    hy, hz = 0.9572 * np.sin(half) * a2b, 0.9572 * np.cos(half) * a2b
    body = np.array([[0, 0, 0], [0, hy, hz], [0, -hy, hz], [0, 0, 0.25 * a2b]])
    oxy, radius = [], _radius(nw)
    while len(oxy) < nw:
        p = rng.uniform(-radius, radius, size=3)
        if p @ p <= radius * radius and all(np.linalg.norm(p - o) >= 2.6 * a2b for o in oxy):
            oxy.append(p)
    sites = np.empty((nw, 4, 3))
    for i, o in enumerate(oxy):
        w, x, y, z = (lambda q: q / np.linalg.norm(q))(rng.normal(size=4))
        R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                      [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                      [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])
        sites[i] = body @ R.T + o
    qh = 0.5742185854046506
    charges = np.tile([qh, qh, -2 * qh], nw)
    first = 4 * np.arange(nw)[:, None]
    charge_site = (first + [1, 2, 3]).reshape(-1).astype(np.int32)
    dipole_site = (first + [0, 1, 2]).reshape(-1).astype(np.int32)
    # induced dipoles of a cluster: about 0.2 a.u. on O, a fifth of it on each H
    dipoles = rng.normal(size=(nw, 3, 3)) * np.array([0.12, 0.025, 0.025])[None, :, None]
    return sites.reshape(-1), charges, charge_site, dipoles.reshape(-1), dipole_site


def _scpol_lists(sites, nw, seed):
    """Polarisable atoms O, H, H of every water: sites, A = (1/alpha - T)^-1 with Thole damping, the water field."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 12]))
    pol_site = (4 * np.arange(nw)[:, None] + [0, 1, 2]).reshape(-1).astype(np.int32)
    pos = sites.reshape(-1, 3)[pol_site]
    b3 = (1.0 / 0.52917720859) ** 3
    alpha = np.tile([1.22 * b3, 0.28 * b3, 0.28 * b3], nw)
    m = len(alpha)
    a = np.zeros((m, 3, m, 3))
    d = pos[:, None, :] - pos[None, :, :]
    r = np.sqrt((d * d).sum(-1)) + np.eye(m)
    x = 0.3 * r ** 3 / np.sqrt(alpha[:, None] * alpha[None, :])
    ex = np.exp(-x)
    c1, c2 = (1 - (1 + x) * ex) * 3.0 / r ** 5, (1 - ex) / r ** 3
    off = 1.0 - np.eye(m)
    for p in range(3):
        for q in range(3):
            a[:, p, :, q] = -off * (c1 * d[:, :, p] * d[:, :, q] - (c2 if p == q else 0.0))
        a[np.arange(m), p, np.arange(m), p] = 1.0 / alpha
    inva = np.linalg.inv(a.reshape(3 * m, 3 * m))
    epc = rng.normal(scale=0.02, size=3 * m)
    return pol_site, 0.5 * (inva + inva.T), epc, -0.01 * nw


def _fields(npoints, count, seed, salt):
    """Wavefunction-like rows on the GPU: a smooth envelope times a wave, and a little noise; of unit norm."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * salt + int(seed))
    t = torch.linspace(-1.0, 1.0, npoints, dtype=torch.float64, device="cuda")
    u = torch.rand(count, 4, dtype=torch.float64, device="cuda", generator=gen)
    out = torch.randn(count, npoints, dtype=torch.float64, device="cuda", generator=gen)
    out *= 0.02
    for j in range(count):
        width, centre, wave, phase = (float(v) for v in u[j])
        env = torch.exp(-((t - (0.6 * centre - 0.3)) / (0.2 + 0.5 * width)) ** 2)
        out[j] += 1.0
        out[j] *= env * torch.cos(3.0 + 2000.0 * wave * t + 6.0 * phase)
        out[j] /= torch.linalg.vector_norm(out[j])
    return out


def _model_potential(case, seed):
    """A smooth attractive V with the depth and range of a cluster's, for products without a V(r) call."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 13]))
    axes = [torch.as_tensor(_points(m, L), device="cuda") for m, L in zip(_n(case), _box(case))]
    z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    v = torch.zeros_like(x)
    for q in (-0.4, 0.3, -0.3, 0.4):
        c = rng.uniform(-5.0, 5.0, size=3)
        v += q / torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 + 2.0)
    return v.reshape(-1)


def prepare(case, seed):
    pg = _package()
    op = case["op"]
    s = {"case": dict(case), "prec": pg.PG_MIXED if case.get("prec") == "mixed" else pg.PG_FP64}
    if op == "block":
        s["P"], s["Q"] = _blocks(case, seed)
        s["C"] = _coefficients(case, seed)
        return s
    s["grid"] = pg.Grid(_n(case), _box(case))
    if op in ("hx", "precond"):
        s["X"] = _fields(s["grid"].N, case["nvec"], seed, 3).reshape(-1)
        if op == "hx":
            s["v"] = _model_potential(case, seed)
        else:
            s["R"] = torch.empty_like(s["X"])
            s["sigma"] = _shifts(case, seed)
        return s
    lists = _water_lists(case["nw"], seed)
    s["tables"] = pg.WaterTables.from_lists(*lists)
    if op == "scpol":
        pol_site, inva, epc, vww = _scpol_lists(lists[0], case["nw"], seed)
        s["model"] = pg.ScPol(tables=s["tables"], pol_site=pol_site, inva=inva, epc=epc, vpol_ww=vww)
    return s


def _blocks(case, seed):
    """A basis and a block that overlaps it, as H times basis vectors and new corrections do."""
    P = _fields(case["npoints"], case["na"], seed, 1)
    return P, 0.6 * _fields(case["npoints"], case["nb"], seed, 2) + 0.8 * P[:case["nb"]]


def _coefficients(case, seed):
    """Ritz coefficients: na x nb with orthonormal columns."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 14]))
    q, _ = np.linalg.qr(rng.normal(size=(case["na"], case["nb"])))
    return torch.as_tensor(np.ascontiguousarray(q), device="cuda")


def _shifts(case, seed):
    """Ritz values of bound and nearly bound states, the preconditioner's shifts (hartree)."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 15]))
    return -rng.uniform(0.005, 0.2, size=case["nvec"])


# ------------------------------------------------------------------ one pass

def run(s):
    pg, case = _package(), s["case"]
    op = case["op"]
    if op == "hx":
        return s["grid"].hx(s["v"], s["X"], nvec=case["nvec"], precision=s["prec"])
    if op == "precond":
        # in place: the block of residuals becomes the block of corrections
        s["R"].copy_(s["X"])
        return s["grid"].precondition(s["R"], s["sigma"], precision=s["prec"])
    if op == "block":
        return {"gram": pg.block_gram(s["P"], s["Q"], precision=s["prec"]),
                "combine": pg.block_combine(s["P"], s["C"], precision=s["prec"])}
    if op == "potential":
        v, parts = s["grid"].potential(s["tables"], parts=True)
        return {"v": v, "parts": parts}
    if op == "scpol":
        return s["grid"].potential_scpol(s["model"])
    v = s["grid"].potential(s["tables"])
    evals, evecs, _ = s["grid"].solve(v, nroots=case["nroots"], maxsub=case["maxsub"], ptol=case["ptol"],
                                      corrflag=case["corrflag"], precision=s["prec"])
    return {"v": v, "evals": evals, "evecs": evecs}


def work(case):
    op = case["op"]
    if op == "block":
        n, na, nb = case["npoints"], case["na"], case["nb"]
        return {"bytes": 8.0 * n * (na + nb) * 2, "flops": 4.0 * n * na * nb}
    n = _n(case)
    N, axes = float(np.prod(n)), sum(n)
    if op == "hx":
        return {"bytes": 8.0 * N * (2 * case["nvec"] + 1), "flops": 2.0 * N * (axes + 1) * case["nvec"]}
    if op == "precond":
        return {"bytes": 16.0 * N * case["nvec"], "flops": 4.0 * N * axes * case["nvec"]}
    pairs = N * case["nw"] * 4 * 30.0  # per site and point: the distance, its inverse powers, an exponential
    if op == "potential":
        return {"bytes": 8.0 * N * 5, "flops": pairs}
    if op == "scpol":
        return {"bytes": 8.0 * N, "flops": pairs + 2.0 * N * (9 * case["nw"]) ** 2}
    # a point: V and the states written; V(r), then some thirty products and block work on 25 basis vectors
    k = case["nroots"]
    return {"bytes": 8.0 * N * (1 + k), "flops": pairs + 30 * 2.0 * N * k * (axes + 4 * 25)}


# ------------------------------------------------------------------ the same in 64 bits

PI15 = 3.14159265358979  # the model's pi


def _points(n, L):
    dx = L / (n + 1)
    return -0.5 * L + dx * np.arange(1, n + 1)


def _kinetic(n, L):
    """Sine-DVR kinetic matrix of a particle of mass 1 in a box of length L (n interior points)."""
    dx, f3 = L / (n + 1), float((n + 1) ** 2)
    f1, a = 0.5 * PI15 * PI15 / (dx * dx), np.arange(1, n + 1) * (PI15 / (n + 1))
    with np.errstate(divide="ignore", invalid="ignore"):
        t = f1 * 2.0 / f3 * np.outer(np.sin(a), np.sin(a)) / (np.cos(a)[:, None] - np.cos(a)[None, :]) ** 2
    t *= np.where((np.arange(n)[:, None] - np.arange(n)[None, :]) % 2 == 0, 1.0, -1.0)
    t[np.arange(n), np.arange(n)] = f1 * (1.0 / 3.0 + 1.0 / (6.0 * f3) - 0.5 / (f3 * np.sin(a) ** 2))
    return torch.as_tensor(t, device="cuda")


def _three_axes(mats, X):
    """mats = (Ax, Ay, Az) applied along each axis of X[vector, z, y, x]: the three separate results."""
    return (torch.matmul(X, mats[0].T), torch.matmul(mats[1], X),
            torch.einsum("ab,vbyx->vayx", mats[2], X))


def _apply_h(T, v, X):
    return v * X + sum(_three_axes(T, X))


def _apply_green(Q, d, sigma, X):
    """(T - sigma_j)^-1 X_j in the eigenbasis Q of each axis."""
    Y = torch.matmul(X, Q[0])
    Y = torch.matmul(Q[1].T, Y)
    Y = torch.einsum("ab,vbyx->vayx", Q[2].T, Y)
    Y = Y / (d[0][None, None, None, :] + d[1][None, None, :, None] + d[2][None, :, None, None]
             - sigma[:, None, None, None])
    Y = torch.matmul(Y, Q[0].T)
    Y = torch.matmul(Q[1], Y)
    return torch.einsum("ab,vbyx->vayx", Q[2], Y)


def _reff(r, r0):
    q = torch.clamp(r / r0, max=1.0)
    return torch.where(r < r0, r0 * (0.5 + q ** 3 * (1.0 - 0.5 * q)), r)


def _grid_points(case):
    ax = [torch.as_tensor(_points(m, L), device="cuda") for m, L in zip(_n(case), _box(case))]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return x.reshape(-1), y.reshape(-1), z.reshape(-1)


def _exact_parts(case, lists, dipoles=True, one_site_pol=True):
    """Charges, induced dipoles, Slater cores and one-site polarisation of V(r), in the model's damping."""
    sites, charges, charge_site, dip, dipole_site = lists
    xyz = _grid_points(case)
    parts = [torch.zeros_like(xyz[0]) for _ in range(4)]
    q = dict(zip(charge_site.tolist(), charges.tolist()))
    mu = dict(zip(dipole_site.tolist(), dip.reshape(-1, 3).tolist())) if dipoles else {}
    sig = 1.0 / 4.4837
    sto = {0: [(9.98526, 192.608 * sig), (1.67075, 13.8937 * sig)], 1: [(1.64121, 1.7643 * sig)],
           2: [(1.64121, 1.7643 * sig)]}
    for s, p in enumerate(sites.reshape(-1, 3).tolist()):
        d = [a - b for a, b in zip(xyz, p)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        r = torch.sqrt(r2)
        if s in q:
            parts[0] -= q[s] / _reff(r, 1.7724)
        if s in mu:
            parts[1] -= (d[0] * mu[s][0] + d[1] * mu[s][1] + d[2] * mu[s][2]) / _reff(r, 1.7724) ** 3
        for zeta, coef in sto.get(s % 4, []):
            parts[2] += coef * torch.exp(-zeta * r)
        if one_site_pol and s % 4 == 3:
            parts[3] -= 0.5 * 9.745 * r2 / _reff(r, 2.536) ** 6
    return parts


def _exact_scpol(case, seed, lists):
    pol_site, inva, epc, vww = _scpol_lists(lists[0], case["nw"], seed)
    v = sum(_exact_parts(case, lists, dipoles=False, one_site_pol=False))
    pos = torch.as_tensor(lists[0].reshape(-1, 3)[pol_site], device="cuda")
    A, e0 = torch.as_tensor(inva, device="cuda"), torch.as_tensor(epc, device="cuda").view(1, -1)
    pts = torch.stack(_grid_points(case), 1)
    for c0 in range(0, len(pts), 65536):
        d = pts[c0:c0 + 65536, None, :] - pos[None, :, :]
        r = torch.sqrt((d * d).sum(-1))
        E = (d / _reff(r, 2.536)[:, :, None] ** 3).reshape(len(d), -1) + e0
        v[c0:c0 + 65536] += -0.5 * (E * (E @ A)).sum(1) - vww
    return v


def _lowest(case, v, count):
    """The lowest eigenvalues of T + v by preconditioned block Rayleigh-Ritz on a growing basis, in 64 bits."""
    n, L = _n(case), _box(case)
    T = [_kinetic(m, l) for m, l in zip(n, L)]
    eig = [torch.linalg.eigh(t) for t in T]
    Q, d = [e[1] for e in eig], [e[0] for e in eig]
    v = v.view(1, n[2], n[1], n[0])
    keep = count + 3
    gen = torch.Generator(device="cuda").manual_seed(5)
    X = torch.randn(keep, n[2], n[1], n[0], dtype=torch.float64, device="cuda", generator=gen)
    B = torch.linalg.qr(_apply_green(Q, d, torch.full((keep,), -0.1, dtype=torch.float64, device="cuda"),
                                     X).reshape(keep, -1).T)[0].T
    HB = _apply_h(T, v, B.reshape(-1, n[2], n[1], n[0])).reshape(len(B), -1)
    for _ in range(300):
        w, V = torch.linalg.eigh(0.5 * (B @ HB.T + HB @ B.T))
        w, V = w[:keep], V[:, :keep]
        U, HU = V.T @ B, V.T @ HB
        R = HU - w[:, None] * U
        if float(torch.linalg.vector_norm(R[:count], dim=1).max()) < 1e-9:
            break
        if len(B) > 12 * keep:
            B, HB = U, HU
        C = _apply_green(Q, d, torch.clamp(w, max=-0.01), R.reshape(-1, n[2], n[1], n[0])).reshape(keep, -1)
        for _ in range(2):
            C = C - (C @ B.T) @ B
            C = torch.linalg.qr(C.T)[0].T
        B = torch.cat([B, C])
        HB = torch.cat([HB, _apply_h(T, v, C.reshape(-1, n[2], n[1], n[0])).reshape(keep, -1)])
    return w[:count].cpu().numpy()


def exact(case, seed):
    op = case["op"]
    if op == "block":
        P, Q = _blocks(case, seed)
        return {"gram": torch.stack([(P * q).sum(1) for q in Q], 1), "combine": _coefficients(case, seed).T @ P}
    n, L = _n(case), _box(case)
    shape = (-1, n[2], n[1], n[0])
    if op == "hx":
        X = _fields(int(np.prod(n)), case["nvec"], seed, 3).view(shape)
        T = [_kinetic(m, l) for m, l in zip(n, L)]
        return _apply_h(T, _model_potential(case, seed).view(1, *shape[1:]), X).reshape(-1)
    if op == "precond":
        X = _fields(int(np.prod(n)), case["nvec"], seed, 3).view(shape)
        eig = [torch.linalg.eigh(_kinetic(m, l)) for m, l in zip(n, L)]
        sigma = torch.as_tensor(_shifts(case, seed), device="cuda")
        return _apply_green([e[1] for e in eig], [e[0] for e in eig], sigma, X).reshape(-1)
    lists = _water_lists(case["nw"], seed)
    if op == "potential":
        parts = _exact_parts(case, lists)
        return {"v": sum(parts), "parts": torch.stack(parts)}
    if op == "scpol":
        return _exact_scpol(case, seed, lists)
    v = sum(_exact_parts(case, lists))
    # the sign of an eigenvector is the iteration's own
    return {"v": v, "evals": _lowest(case, v, case["nroots"]), "evecs": None}
