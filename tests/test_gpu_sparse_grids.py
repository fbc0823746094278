"""Open systems whose grid has more tiles than the sort's kernels have blocks:
particles in a few corners of 10^8 cells, alone and as one of two systems.
Lists against brute force, slots against the stable (cell, old slot) order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def corners(sep, seed):
    g = np.random.default_rng(seed)
    c = np.array([[0, 0, 0], [sep, 0, 0], [0, sep, sep], [sep, sep, sep], [0.4 * sep, 0.7 * sep, 0.5 * sep]])
    x = np.concatenate([g.uniform(-9.0, 9.0, (397, 3)) + c[k % 5] for k in range(5)] + [[[0.2 * sep] * 3]])
    return x[g.permutation(len(x))]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("seps", [(950.0,), (700.0, 950.0), (950.0, 30.0)])
def test_sorted_and_listed(precision, seps):
    from openrbc_gb300 import RTParameter, Simulation
    xs = [corners(s, k) for k, s in enumerate(seps)]
    n = len(xs[0])
    x = np.concatenate(xs)
    nrm = np.tile([0.0, 0.0, 1.0], (len(x), 1))
    z = np.zeros_like(x)
    desc = {"lo": (-1e6,) * 3, "hi": (1e6,) * 3}
    off = np.arange(len(xs) + 1) * n
    with Simulation(RTParameter(init="lipid", kBT=0.0, precision=precision), skin=0.4, max_neighbors=96) as s:
        s.upload_batch([desc] * len(xs), x, nrm, z, z, np.zeros(len(x), np.int32),
                       np.arange(1, len(x) + 1, dtype=np.int32), off)
        for _ in range(2):  # the counts are zero again after a build
            s.rebuild()
        counts, lst = s.neighbors()
        slot0 = 0
        cells = 0
        for k in range(len(xs)):
            c = s.cells(k)
            cells += np.prod((c["nc"] + 3) // 4 * 4, dtype=np.int64)
            q = np.stack([c["cell"] & 2047, (c["cell"] >> 11) & 2047, (c["cell"] >> 22) & 1023], 1).astype(np.int64)
            q, slot = q[off[k]:off[k + 1]], c["slot"][off[k]:off[k + 1]]
            nt = ((c["nc"] + 3) // 4).astype(np.int64)
            spread = lambda v: (v & 1) | ((v & 2) << 2)
            tile = (q[:, 0] >> 2) + nt[0] * ((q[:, 1] >> 2) + nt[1] * (q[:, 2] >> 2))
            code = (tile << 6) | spread(q[:, 0] & 3) | (spread(q[:, 1] & 3) << 1) | (spread(q[:, 2] & 3) << 2)
            assert np.array_equal(np.sort(slot), slot0 + np.arange(n))  # one slot each, no gaps
            assert (np.diff(code[np.argsort(slot)]) >= 0).all()         # by cell
            slot0 += (n + 255) // 256 * 256
        assert cells > 100_000_000  # more than the kernels' blocks cover at once
    lim = float(np.float32(3.0 * 3.0))
    tol = 1e-11 if precision == "fp64" else 2e-6
    rows = np.repeat(np.arange(len(x)), counts)
    for k in range(len(xs)):
        r2 = ((xs[k][:, None, :] - xs[k][None, :, :]) ** 2).sum(2)
        near = (r2 < lim) & ~np.eye(n, dtype=bool)
        got = np.zeros((n, n), bool)
        m = (rows >= off[k]) & (rows < off[k + 1])
        assert (lst[m] >= off[k]).all() and (lst[m] < off[k + 1]).all()
        got[rows[m] - off[k], lst[m] - off[k]] = True
        assert m.sum() == got.sum()
        assert (np.abs(r2[got != near] - lim) < tol * lim).all()
