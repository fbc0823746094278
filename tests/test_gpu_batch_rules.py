"""Rules that follow the number of particles (rows per batch of the force
loop, warps per 32 slots of the list build) on cells with proteins, bonds and
faces: a cell alone, as one of a batch that half fills the GPU and as one of
a batch that fills it agrees bit for bit when lists are rebuilt every step."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def network_cell():
    g = load_golden("cell_ico12.npz")
    ty = g["type"].copy()
    ty[np.flatnonzero(ty == 2)[::2]] = 1  # all six types
    return {"x": g["x"], "n": g["nrm"], "v": g["v"], "o": g["o"], "type": ty, "tag": g["tag"], "bonds": g["bonds"],
            "bond_r0": np.array([2.25, 1.1225, 2.25, 2.24])[g["bonds"][:, 0]], "faces": None, "constraint": {}}, None


def meshed_cell():
    from openrbc_gb300 import workloads
    return workloads.rbc(n_lipid=3000, freq=3, kT=1.0, seed=5), workloads.RBC_BOND_TABLE


def run(w, table, copies, precision, form, energy):
    from openrbc_gb300 import RTParameter, Simulation
    n = len(w["x"])
    lo = int(w["tag"].min())
    span = int(w["tag"].max()) - lo + 1
    rep = {q: np.concatenate([w[q]] * copies) for q in ("x", "n", "v", "o", "type", "bond_r0")}
    tag = np.concatenate([w["tag"] + k * span for k in range(copies)])
    bonds = np.concatenate([w["bonds"] + np.array([0, k * span, k * span]) for k in range(copies)])
    faces = None if w["faces"] is None else np.concatenate([w["faces"] + k * span for k in range(copies)])
    desc = {"lo": (-1000.0,) * 3, "hi": (1000.0,) * 3, **w["constraint"]}
    kw = {"bond_table": table} if table else {}
    p = RTParameter(init="lipid", kBT=1.0, precision=precision, integrator="nose-hoover")
    with Simulation(p, rebuild_every=1, kernel_variant=form, energy=energy, **kw) as s:
        s.upload_batch([desc] * copies, rep["x"], rep["n"], rep["v"], rep["o"], rep["type"], tag,
                       np.arange(copies + 1) * n, bonds=bonds, bond_r0=rep["bond_r0"], faces=faces)
        s.step(3)
        state = [a.reshape(copies, n, 3) for a in s.download()]
        f, t, e = s.forces()
        counts, lst = s.neighbors()
        th = s.thermo(copies - 1)
    state += [f.reshape(copies, n, 3), t.reshape(copies, n, 3), e.reshape(copies, n)]
    last = lst[len(lst) - counts[-n:].sum():] - (copies - 1) * n
    return state, (counts[-n:], last), [th[k] for k in ("zeta", "ke2", "epot", "area", "volume")]


@pytest.mark.parametrize("cell", [network_cell, meshed_cell])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("form,energy", [(0, False), (0, True), (64, True)])
def test_alone_and_in_batches(cell, precision, form, energy):
    w, table = cell()
    assert (w["type"] != 0).sum() > 50 and len(w["bonds"]) > 100
    one, rows1, th1 = run(w, table, 1, precision, form, energy)
    pad = (len(w["x"]) + 255) // 256 * 256
    for slots in (45_000, 110_000):  # two warps per 32 slots; one, and two rows per batch
        many, rows, th = run(w, table, slots // pad + 1, precision, form, energy)
        for a, b in zip(rows, rows1):
            assert np.array_equal(a, b)
        for a, b in zip(many, one):
            assert np.array_equal(np.broadcast_to(b, a.shape), a)
        assert th == th1
