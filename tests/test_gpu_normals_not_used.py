"""A normal that no pair in range uses must not reach the forces: particles
whose type has no anisotropic pair may carry any normal, and a partner that is
listed (inside the skin) but out of range contributes nothing, whatever its
normal holds."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

BOX = ((-1000.0, 1000.0),) * 3


def forces(g, nrm, precision, form, energy=False):
    from openrbc_gb300 import RTParameter, Simulation
    p = RTParameter(init="lipid", kBT=0.22, precision=precision)
    with Simulation(p, box=BOX, kernel_variant=form, skin=0.5) as s:
        s.upload(g["x"], nrm, g["v"], g["o"], g["type"], g["tag"], g.get("bonds"))
        return s.forces()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", [0, 64])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_normals_of_types_without_anisotropic_pairs(precision, form, value):
    g = load_golden("cell_ico12.npz")
    plain = g["type"] >= 4  # repulsive and bonded interactions only
    assert plain.sum() > 100
    nrm = g["nrm"].copy()
    nrm[plain] = value
    for a, b in zip(forces(g, nrm, precision, form), forces(g, g["nrm"], precision, form)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", [0, 64])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("types", [(0, 0, 0), (0, 0, 3), (3, 0, 0)])
def test_listed_partner_out_of_range(precision, form, value, types):
    # 0 - 1 are in range of each other; 2 is within the skin of 1 alone
    x = np.array([[0.0, 0.0, 0.0], [2.0, 0.0, 0.0], [4.7, 0.0, 0.0]])
    n = np.array([[0.0, 0.6, 0.8], [0.0, 0.0, 1.0], [0.0, 0.0, 1.0]])
    g = {"x": x, "v": np.zeros((3, 3)), "o": np.zeros((3, 3)), "type": np.array(types, np.int32),
         "tag": np.arange(1, 4, dtype=np.int32)}
    bad = n.copy()
    bad[2] = value
    good = forces(g, n, precision, form)
    assert np.abs(good[0][:2]).min(axis=0).max() > 0.0
    for a, b in zip(forces(g, bad, precision, form), good):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", [0, 64])
def test_particle_without_partners(precision, form):
    g = {"x": np.zeros((1, 3)), "v": np.zeros((1, 3)), "o": np.zeros((1, 3)), "type": np.zeros(1, np.int32),
         "tag": np.ones(1, np.int32)}
    for a in forces(g, np.full((1, 3), np.nan), precision, form):
        assert np.array_equal(a, np.zeros_like(a))
