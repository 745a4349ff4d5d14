"""Linear-spring contacts over the range of impact velocities (the law's powers
of it, below 0.01 m/s their floor) against the oracle, whose powers are libm's."""
import pytest

from oracle.oracle import OracleSystem
from sdem_gb300 import beds, props
from sdem_gb300.capi import DEMSystem
from tests.helpers import assert_step_matches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vmax", [1.0e-4, 0.05, 3.0, 400.0, 1.0e6])
def test_impact_velocities(gpu_lib, vmax):
    case = beds.lattice_cloud_case(1500, seed=91, cf_type=props.CFT_LSD, ntypes=3, vmax=vmax)
    g, o = DEMSystem(case), OracleSystem(case)
    g.step(1)
    o.step(1)
    assert g.counters()["pp"] > 500
    assert g.counters() == o.counters()
    if g.counters()["nlocal"] == 0:   # at 1e6 m/s every sphere leaves the box in the step
        return
    assert_step_matches(g, o, what=f"vmax {vmax}", pre=case.particles, case=case)
