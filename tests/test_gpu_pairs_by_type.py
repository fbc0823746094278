"""Which pairs are listed and which interact, with particles of all six types:
neighbour lists against brute force with each type pair's own range, forces
against the oracle, and FP64 decisions for pairs that sit closer to a cutoff
than single precision can tell."""
import numpy as np
import pytest

from conftest import load_golden, rel_l2
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BOX = ((-1000.0, 1000.0),) * 3
# interaction ranges by type pair (src/forcefield_canonical.h): lipid 0, proteins 1..5
S, W = 1.1225, 3.4 * 1.1225
RANGE = np.array([[2.6, 2.6, 2.6, 2.6, S, S],
                  [2.6, 2.6, 2.6, 2.6, W, W],
                  [2.6, 2.6, 2.6, 2.6, W, S],
                  [2.6, 2.6, 2.6, 2.6, 0, 0],
                  [S, W, W, 0, 0, 0],
                  [S, W, S, 0, 0, 0]])


def cell(order_seed=None):
    """The reference's 3,544-particle cell with every other particle of type 2 made one of type 1."""
    g = dict(load_golden("cell_ico12.npz"))
    g["type"] = g["type"].copy()
    g["type"][np.flatnonzero(g["type"] == 2)[::2]] = 1
    assert set(g["type"].tolist()) == set(range(6))
    if order_seed is not None:
        p = np.random.default_rng(order_seed).permutation(len(g["x"]))
        for k in ("x", "nrm", "v", "o", "type", "tag"):
            g[k] = g[k][p]
    return g


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("subset", ["all", "proteins", "no_lipid_partners"])
@pytest.mark.parametrize("skin", [0.4, 1.3])
def test_lists_against_brute_force(precision, subset, skin):
    from openrbc_gb300 import RTParameter, Simulation
    g = cell(7)
    keep = {"all": g["type"] >= 0, "proteins": g["type"] > 0, "no_lipid_partners": g["type"] >= 4}[subset]
    x, ty = g["x"][keep], g["type"][keep]
    n = len(x)
    with Simulation(RTParameter(init="lipid", precision=precision), box=BOX, skin=skin, max_neighbors=128) as s:
        s.upload(x, g["nrm"][keep], g["v"][keep], g["o"][keep], ty, np.arange(1, n + 1, dtype=np.int32))
        counts, lst = s.neighbors()
    got = np.zeros((n, n), bool)
    got[np.repeat(np.arange(n), counts), lst] = True
    assert counts.sum() == got.sum()  # no pair twice
    r2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(2)
    rng = RANGE[ty[:, None], ty[None, :]]
    lim = np.where(rng > 0, (rng + skin) ** 2, 0.0)
    want = (r2 < lim) & ~np.eye(n, dtype=bool)
    # cutoffs are kept in single precision (2^-24); single-precision positions in a cell of 5 add 2e-6
    tol = 1.2e-7 if precision == "fp64" else 2e-6
    off = got != want
    assert (np.abs(r2 - lim)[off] <= tol * lim[off]).all()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", [0, 64])
def test_forces_by_type_against_the_oracle(precision, form):
    from openrbc_gb300 import RTParameter, Simulation
    g = cell()
    st = orc.State(x=g["x"], nrm=g["nrm"], v=g["v"], o=g["o"], type=g["type"], tag=g["tag"], bonds=g["bonds"])
    f_ref, t_ref, _, _ = orc.forces(st)
    with Simulation(RTParameter(init="lipid", kBT=0.22, precision=precision), box=BOX, kernel_variant=form) as s:
        s.upload(g["x"], g["nrm"], g["v"], g["o"], g["type"], g["tag"], g["bonds"])
        f, t, _ = s.forces()
    tol = 1e-12 if precision == "fp64" else 1e-5
    for k in range(6):
        m = g["type"] == k
        assert rel_l2(f[m], f_ref[m]) < tol
        if k < 4:
            assert rel_l2(t[m], t_ref[m]) < tol
        else:
            assert np.array_equal(t[m], t_ref[m])  # none


@pytest.mark.parametrize("types", [(0, 0), (0, 3), (1, 2), (0, 4), (2, 5), (1, 4)])
def test_fp64_decisions_at_the_cutoffs(types):
    """Isolated pairs at the list cutoff and at the interaction range, apart by
    1e-7 of it and less: listed below the (single-precision) list cutoff and
    not above, and in range below the FP64 range and not above.  The force
    is of the size of the step that the purely repulsive pairs have there."""
    from openrbc_gb300 import RTParameter, Simulation
    skin = 0.4
    rng = np.random.default_rng(3)
    R = RANGE[types]
    r_list = np.sqrt(np.float64(np.float32((R + skin) ** 2)))
    delta = np.concatenate([s * np.array([1e-7, 3e-8, 1e-8, 1e-9, 1e-10]) for s in (1.0, -1.0)])
    r = np.concatenate([r_list * (1 + delta), R * (1 + delta)])
    r = np.tile(r, 12)
    m = len(r)
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    side = int(np.ceil(m ** (1 / 3)))
    grid = np.stack(np.unravel_index(np.arange(m), (side,) * 3), 1) * 12.0 - 6.0 * side
    a = grid + rng.uniform(-1.5, 1.5, (m, 3))
    x = np.stack([a, a + r[:, None] * u], 1).reshape(-1, 3)
    d = x[0::2] - x[1::2]
    d2 = (d * d).sum(1)
    sure = np.abs(d2 / np.float64(np.float32((R + skin) ** 2)) - 1) > 1e-11
    nrm = rng.normal(size=x.shape)
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    ty = np.tile(np.array(types, np.int32), m)
    tag = np.arange(1, 2 * m + 1, dtype=np.int32)
    z = np.zeros_like(x)
    with Simulation(RTParameter(init="lipid", precision="fp64"), box=BOX, skin=skin) as s:
        s.upload(x, nrm, z, z, ty, tag)
        counts, _ = s.neighbors()
        f, t, _ = s.forces()
    listed = d2 < np.float64(np.float32((R + skin) ** 2))
    assert listed.any() and not listed.all()
    assert np.array_equal(counts[0::2][sure] > 0, listed[sure])
    assert np.array_equal(counts[1::2], counts[0::2])
    st = orc.State(x=x, nrm=nrm, v=z, o=z, type=ty, tag=tag)
    f_ref, _, _, _ = orc.forces(st)
    at_range = np.abs(d2 / (R * R) - 1)
    ok = np.repeat(at_range > 1e-11, 2)
    step = np.abs(f_ref).max()
    if 4 in types or 5 in types:
        assert step > 1e-4  # an interaction that is cut off where it has not died out
    assert np.abs(f - f_ref)[ok].max() <= 1e-6 * step


@pytest.mark.parametrize("stray", [1e8, 2e13])
def test_fp64_in_cells_that_single_precision_cannot_resolve(stray):
    """A particle far away makes the cells of its axis large: coordinates in
    them, rounded to single precision, no longer tell which pairs are near."""
    from openrbc_gb300 import RTParameter, Simulation
    g = np.random.default_rng(5)
    n = 400
    k = np.arange(n)
    x = np.stack([1.3 * (k % 20), 1.3 * (k // 20), np.zeros(n)], 1) + g.uniform(-0.1, 0.1, (n, 3))
    far = np.concatenate([x, [[stray, 0.0, 0.0]]])
    nrm = np.tile([0.0, 0.0, 1.0], (n + 1, 1))
    nrm[:, 1] += 0.1 * np.sin(np.arange(n + 1))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    res = []
    for p in (far, x):
        m = len(p)
        z = np.zeros((m, 3))
        with Simulation(RTParameter(init="lipid", precision="fp64"), box=((-1e14, 1e14),) * 3, skin=0.4) as s:
            s.upload(p, nrm[:m], z, z, np.zeros(m, np.int32), np.arange(1, m + 1, dtype=np.int32))
            counts, lst = s.neighbors()
            f, t, _ = s.forces()
            res.append((counts[:n], f[:n], t[:n]))
    # offsets in a cell of 1.5e10 resolve 1e-6; the list cutoff's neighbourhood is left out
    d2 = ((x[:, None, :] - x[None, :, :]) ** 2).sum(2)
    edge = (np.abs(np.sqrt(d2) - 3.0) < 1e-4).any(1)
    assert np.array_equal(res[0][0][~edge], res[1][0][~edge])
    scale = np.abs(res[1][1]).max()
    assert np.abs(res[0][1] - res[1][1]).max() < 1e-4 * scale
    assert np.abs(res[0][2] - res[1][2]).max() < 1e-4 * np.abs(res[1][2]).max()
