"""The in-order FP64 products of the solver of several roots, over every number of vectors left after groups of four:
a solve's states against the dense spectrum of the same operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nroots", [2, 3, 4, 5, 6, 7])
def test_fp64_states_of_several_roots(pg, nroots):
    torch = pytest.importorskip("torch")
    n = (9, 10, 11)
    g = pg.Grid(n, (8.0, 8.5, 9.0))
    rng = np.random.default_rng(nroots)
    v = torch.as_tensor(rng.standard_normal(g.N) * 0.3, device="cuda")
    evals, evecs, stats = g.solve(v, nroots=nroots, maxsub=8 * nroots, ptol=8, corrflag=3, precision=pg.PG_FP64)
    tx, ty, tz = (g.kinetic(a) for a in range(3))
    ex, ey, ez = (np.eye(m) for m in n)
    H = np.kron(ez, np.kron(ey, tx)) + np.kron(ez, np.kron(ty, ex)) + np.kron(tz, np.kron(ey, ex))
    H[np.diag_indices(g.N)] += v.cpu().numpy()
    w = np.linalg.eigvalsh(H)[:nroots]
    assert np.max(abs(np.asarray(evals) - w)) <= 1e-10 * max(1.0, abs(w).max())
    u = evecs.cpu().numpy().reshape(nroots, -1)
    assert np.max(abs(u @ u.T - np.eye(nroots))) <= 1e-10
    # the residual asked for, with the norm's rounding
    assert np.max(np.linalg.norm(u @ H - np.asarray(evals)[:, None] * u, axis=1)) <= 2e-8
