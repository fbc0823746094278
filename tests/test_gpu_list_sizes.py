"""Neighbour lists on both sides of the sizes where the list build changes the
number of warps that share 32 slots (four, two, one; the lines follow the
resident warps, which differ between the precisions), against a k-d tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,slots", [("fp64", k) for k in (29184, 29440, 58368, 58624)]
                         + [("mixed", k) for k in (34048, 34304, 68096, 68352)])
def test_lists_against_a_tree(precision, slots):
    from scipy.spatial import cKDTree
    from openrbc_gb300 import RTParameter, Simulation, workloads
    n = slots - 3  # a few ghosts
    w = workloads.lattice(n=n, ncol=int(n ** 0.5), kT=0.0, seed=6)
    rng = np.random.default_rng(1)
    x = w["x"][rng.permutation(n)]
    with Simulation(RTParameter(init="lipid", kBT=0.0, precision=precision), skin=0.4) as s:
        s.upload(x, w["n"], w["v"], w["o"], w["type"], w["tag"])
        counts, lst = s.neighbors()
    cut = np.sqrt(np.float64(np.float32(3.0 * 3.0)))
    ref = cKDTree(x).query_pairs(cut, output_type="ndarray")
    key = lambda i, j: i.astype(np.int64) * n + j
    want = np.sort(np.concatenate([key(ref[:, 0], ref[:, 1]), key(ref[:, 1], ref[:, 0])]))
    got = np.sort(key(np.repeat(np.arange(n), counts), lst))
    assert (np.diff(got) > 0).all()  # no pair twice
    off = np.setxor1d(got, want, assume_unique=True)
    d = x[off // n] - x[off % n]
    tol = 1e-11 if precision == "fp64" else 2e-6
    assert (np.abs((d * d).sum(1) / cut ** 2 - 1) < tol).all()
