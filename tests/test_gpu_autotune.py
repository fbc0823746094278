"""The tuner's choice rests on one measurement per skin and cadence: rows that
differ in the kernel form alone, which selects nothing, carry the same time,
and the chosen pair is the fastest of the table."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,skin", [(0, 0.4), (71, 0.6)])
def test_one_time_per_skin_and_cadence(form, skin):
    from openrbc_gb300 import RTParameter, Simulation, workloads
    w = workloads.lattice(n=4096, ncol=64, kT=1.0, seed=3)
    with Simulation(RTParameter(init="lipid", kBT=1.0, precision="mixed"), skin=skin, kernel_variant=form) as s:
        s.upload(w["x"], w["n"], w["v"], w["o"], w["type"], w["tag"])
        rows = s.autotune(trial_steps=5)
    assert len(rows) == 35
    times = {}
    for r in rows:
        times.setdefault((r["skin"], r["rebuild_every"]), set()).add((r["ms_per_step"], r["rebuilds_per_step"]))
        assert (r["variant"] ^ form) & 64 == 0
    assert all(len(t) == 1 for t in times.values())
    assert 8 <= len(times) <= 10
