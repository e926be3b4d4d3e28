"""The FP64 slices where the waits inside the kernel run out: the same products, by multiply-adds.

pg_slice.cu is compiled with waits of no or few polls, so that none, or some
of the warps, see the copies and the products in time, and linked with the
library's other objects.  What the kernel has in flight then is waited for
with the usual limit before a block ends.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import json, sys
import numpy as np, torch
sys.path[:0] = [%(root)r, %(root)r + "/tests"]
import __graft_entry__ as entry
pg = entry.load_package()
pg.LIB_PATH = sys.argv[1]
entry.load_package().lib()
import importlib
clusters = importlib.import_module("pisces_gb300.clusters")
LD = np.longdouble
out = {}
def apply(t, d, q):
    return (d * q + np.einsum("vzyb,ab->vzya", q, t[0]) + np.einsum("vzbx,ab->vzax", q, t[1])
            + np.einsum("vbyx,ab->vayx", q, t[2]))
for n, nvec in (((64, 40, 24), 2), ((33, 64, 50), 1), ((96, 20, 18), 2), ((20, 160, 6), 1), ((6, 5, 97), 3)):
    rng = np.random.default_rng(n[0])
    g = pg.Grid(n, tuple(0.6 * (m + 1) for m in n))
    x = rng.standard_normal((nvec, n[2], n[1], n[0]))
    v = rng.standard_normal((1, n[2], n[1], n[0]))
    y = g.hx(torch.as_tensor(v.reshape(-1), device="cuda"), torch.as_tensor(x.reshape(-1), device="cuda"), nvec=nvec)
    torch.cuda.synchronize()
    T = [g.kinetic(a).astype(LD) for a in range(3)]
    ref = apply(T, v.astype(LD), x.astype(LD))
    mag = apply([abs(t) for t in T], abs(v).astype(LD), abs(x).astype(LD))
    err = abs(y.cpu().numpy().reshape(x.shape) - ref) / (2.0 ** -53 * mag)
    out["hx %%s" %% (n,)] = [float(err.max()), sum(n) + 6]
    R = torch.as_tensor(x.reshape(-1), device="cuda")
    g.precondition(R, [-0.3] * nvec, precision=pg.PG_FP64)
    w = T[0], T[1], T[2]
    back = apply(T, np.full_like(v, 0.3).astype(LD), R.cpu().numpy().reshape(x.shape).astype(LD))
    out["precondition %%s" %% (n,)] = [float(abs(back - x).max() / abs(x).max() / 2.0 ** -53), 2.0 ** 20]
    g.check()
m = pg.ScPol(clusters.water_cluster(8, 12.0, seed=2))
g = pg.Grid((12, 11, 10), 20.0)
v = g.scpol_add(m, torch.zeros(g.N, dtype=torch.float64, device="cuda")).cpu().numpy()
np.save(sys.argv[2], v)
g.check()
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def run(pg, tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "pisces-1_gb300"))
    import build as B
    sys.path.pop(0)
    folder = tmp_path_factory.mktemp("waits")

    def go(polls, issue):
        obj, lib = str(folder / f"slice_{polls}_{issue}.o"), str(folder / f"lib_{polls}_{issue}.so")
        flags = [] if polls is None else [f"-DPG_SLICE_POLLS={polls}l", f"-DPG_SLICE_POLLS_ISSUE={issue}l"]
        subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, *flags, "-c", os.path.join(B.CSRC, "pg_slice.cu"), "-o", obj],
                       check=True)
        objs = [os.path.join(B.BUILD, f + ".o") for f in B.sources() if f != "pg_slice.cu"]
        subprocess.run([B._nvcc(), *B.ARCH, "-shared", "-cudart", "static", "-o", lib, obj, *objs, "-lpthread", "-lcuda"],
                       check=True)
        npy = str(folder / f"v_{polls}_{issue}.npy")
        r = subprocess.run([sys.executable, "-c", PROGRAM % {"root": ROOT}, lib, npy], capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1]), np.load(npy)
    return go


@pytest.fixture(scope="module")
def plain(run):
    return run(None, None)


# nothing lands in time; products run unread; some of both
@pytest.mark.parametrize("polls,issue", [(0, 0), (0, 16384), (6, 16384), (25, 16384), (25, 40)])
def test_products_without_the_waits(run, plain, polls, issue):
    out, v = run(polls, issue)
    for name, (err, most) in out.items():
        assert err <= most, (name, err, most, plain[0][name])
    # row dots: 72 terms each way
    assert np.all(np.abs(v - plain[1]) <= 200 * 2.0 ** -53 * np.abs(plain[1]).max() * 72)
