"""Pair histogram where its estimate must give way to the rounded operations:
distances on bin edges and at the cutoff, coordinate differences of exactly
half a box edge, coinciding points, a ragged last tile, pairs beyond the last
bin.  Counts are integers: compared with the oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (1, 0, 1)])
@pytest.mark.parametrize("n,dr,nbins,rcut", [(2, 0.25, 100, 0.0), (257, 0.25, 400, 0.0), (600, 0.5, 40, 0.0),
                                             (600, 0.25, 400, 8.0), (1025, 0.1, 700, 0.0)])
def test_rdf_on_bin_edges_and_ties(precision, periodic, n, dr, nbins, rcut):
    from openrbc_gb300 import RTParameter, Simulation
    g = np.random.default_rng(n)
    box = ((-32.0, 32.0), (-32.0, 32.0), (-16.0, 16.0))
    x = np.stack([0.5 * g.integers(2 * int(b[0]), 2 * int(b[1]), n) for b in box], 1)
    nrm = np.tile([0.0, 0.0, 1.0], (n, 1))
    z = np.zeros((n, 3))
    with Simulation(RTParameter(init="lipid", precision=precision), box=box, periodic=periodic) as s:
        s.upload(x, nrm, z, z, np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32))
        xd = s.download()[0]
        counts, dropped = s.rdf(dr=dr, nbins=nbins, rcut=rcut)
    L = [(b[1] - b[0]) if p else 0.0 for b, p in zip(box, periodic)]
    ref, _, ref_drop = orc.rdf(xd, np.zeros(n, np.int32), dr=dr, nbins=nbins, rcut=rcut, centre=[0.0] * 3, L=L,
                               single=precision == "mixed")
    assert np.array_equal(counts, ref) and dropped == ref_drop
