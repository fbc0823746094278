"""Rules that follow the number of particles -- rows per batch of the force
loop, warps per 32 slots of the list build -- must not show in the results: a
system advanced alone (four rows, four warps) and as one of a batch that fills
the GPU (two rows, one warp) agrees bit for bit when lists are rebuilt every
step, with plain and compensated sums, in both precisions.  The sort's places
follow the stable (cell, old slot) order in a crowded cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vesicle(n, seed):
    from openrbc_gb300 import workloads
    w = workloads.vesicles(nves=1, nmin=n, nmax=n, median=n, total=n, kT=1.0, seed=seed)
    g = np.random.default_rng(seed)
    w["n"] = w["n"] + 0.1 * g.standard_normal(w["n"].shape)
    w["n"] /= np.linalg.norm(w["n"], axis=1, keepdims=True)
    return w


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("form", [0, 64])
def test_alone_and_in_a_full_batch(precision, form):
    from openrbc_gb300 import RTParameter, Simulation
    w = vesicle(3001, 3)
    n = len(w["x"])
    copies = 40  # 40 x 3,072 slots: past 97 thousand and past 4,256 warps / 2
    out = []
    for k in (1, copies):
        p = RTParameter(init="lipid", kBT=1.0, precision=precision, integrator="nose-hoover")
        rep = {q: np.concatenate([w[q]] * k) for q in ("x", "n", "v", "o", "type")}
        tag = np.arange(1, k * n + 1, dtype=np.int32)
        with Simulation(p, rebuild_every=1, kernel_variant=form) as s:
            s.upload_batch(w["systems"] * k, rep["x"], rep["n"], rep["v"], rep["o"], rep["type"], tag,
                           np.arange(k + 1) * n)
            s.step(3)
            out.append([a.reshape(k, n, 3) for a in s.download()])
            if k == 1:
                single = s.neighbors()
            else:
                counts, lst = s.neighbors()
                assert np.array_equal(counts[-n:], single[0])
                assert np.array_equal(lst[-len(single[1]):] - (k - 1) * n, single[1])
    for a, b in zip(*out):
        assert np.array_equal(np.broadcast_to(a, b.shape), b)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_crowded_cells_keep_the_stable_order(precision):
    from openrbc_gb300 import RTParameter, Simulation
    g = np.random.default_rng(1)
    n = 1500
    # a few cells of a hundred and more particles, a stray one far away, 36 ghosts
    x = np.concatenate([g.uniform(-4.0, 4.0, (n - 1, 3)), [[60.0, 0.0, 0.0]]])
    nrm = np.tile([0.0, 0.0, 1.0], (n, 1))
    z = np.zeros((n, 3))
    with Simulation(RTParameter(init="lipid", precision=precision), skin=0.4, max_neighbors=512) as s:
        s.upload(x, nrm, z, z, np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32))
        c = s.cells()
        nt = (c["nc"] + 3) // 4
        q = np.stack([c["cell"] & 2047, (c["cell"] >> 11) & 2047, (c["cell"] >> 22) & 1023], 1).astype(np.int64)
        spread = lambda v: (v & 1) | ((v & 2) << 2)
        tile = (q[:, 0] >> 2) + nt[0] * ((q[:, 1] >> 2) + nt[1] * (q[:, 2] >> 2))
        code = (tile << 6) | spread(q[:, 0] & 3) | (spread(q[:, 1] & 3) << 1) | (spread(q[:, 2] & 3) << 2)
        assert np.bincount(np.unique(code, return_inverse=True)[1]).max() > 64
        order = np.lexsort((np.arange(n), code))
        assert np.array_equal(c["slot"][order], np.arange(n))
        counts, lst = s.neighbors()
    d = x[:, None, :] - x[None, :, :]
    r2 = (d * d).sum(2)
    lim = float(np.float32(3.0 * 3.0))
    near = (r2 < lim) & ~np.eye(n, dtype=bool)
    tol = 1e-12 if precision == "fp64" else 2e-6
    got = np.zeros((n, n), bool)
    got[np.repeat(np.arange(n), counts), lst] = True
    assert counts.sum() == got.sum()
    assert (np.abs(r2[got != near] - lim) < tol * lim).all()
