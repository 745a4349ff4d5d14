"""Per-phase timing: a phase without kernels of its own reports no time, the others do."""
import pytest

from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem

pytestmark = pytest.mark.gpu

WITHIN_OTHERS = {"scan_rows", "row_fill", "wall_force", "delete", "step_end"}


# sums and update in one kernel, and in two
@pytest.mark.parametrize("n", [900, 131500])
def test_phases(gpu_lib, n):
    g = DEMSystem(beds.lattice_cloud_case(n, seed=105, nn=1.12e-3))
    g.step(2)
    g.profile_begin(4)
    g.step(3)
    ms, steps = g.profile_end()
    assert steps == 3 and WITHIN_OTHERS < set(ms)
    for name, t in ms.items():
        assert (t == 0.0) == (name in WITHIN_OTHERS), (name, t)
    g.step(2)
