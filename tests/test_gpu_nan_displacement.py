"""A displacement that is not a number counts as one beyond the skin in every
step form: the list is rebuilt at each step from then on (and the step reports
the state), whichever kernel takes the maximum.  (In FP64 the rebuild finds the
particle outside its grid and the re-grid starts the counter again.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator,energy", [("langevin", False), ("langevin", True), ("nose-hoover", False)])
@pytest.mark.parametrize("n", [300, 9000])  # one group of warp partials, several
def test_rebuild_is_requested(integrator, energy, n):
    from openrbc_gb300 import RTParameter, Simulation, workloads
    from openrbc_gb300._native import OrbcError
    w = workloads.lattice(n=n, ncol=int(n ** 0.5), kT=0.0, seed=2)
    w["v"] = w["v"].copy()
    w["v"][n // 3, 1] = np.nan
    p = RTParameter(init="lipid", kBT=0.0, precision="mixed", integrator=integrator)
    with Simulation(p, energy=energy, skin=1.0) as s:
        s.upload(w["x"], w["n"], w["v"], w["o"], w["type"], w["tag"])
        before = s.thermo()["rebuilds"]
        with pytest.raises(OrbcError):
            s.step(4)
        assert s.thermo()["rebuilds"] - before >= 3
