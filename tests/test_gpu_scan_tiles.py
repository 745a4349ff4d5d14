"""The two-launch cell scan over a mostly empty grid: spheres in the first cells,
in the last ones, or in both, so that empty tiles lie behind, before and
between; several steps, since each leaves the counts clear for the next."""
from dataclasses import replace

import numpy as np
import pytest

from oracle.oracle import OracleSystem
from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem
from tests.helpers import assert_step_matches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["first", "last", "both"])
@pytest.mark.parametrize("side", [131.0e-3, 150.0e-3])
def test_spheres_at_the_ends(gpu_lib, where, side):
    case = beds.lattice_cloud_case(1300, seed=95)
    lo, p = np.array(case.opts.minpoint), case.particles
    top = p.posR[:, :3].max(axis=0) + 0.8e-3
    hi = lo + side
    move = {"first": [], "last": range(p.n), "both": range(0, p.n, 2)}[where]
    p.posR[list(move), :3] += hi - top
    case = replace(case, opts=replace(case.opts, maxpoint=tuple(hi)))
    g, o = DEMSystem(case), OracleSystem(case)
    g.step(1)
    o.step(1)
    assert g.counters() == o.counters() and g.counters()["pp"] > 100
    assert_step_matches(g, o, what=where, pre=case.particles, case=case)
    for k in range(4):
        g.step(1)
        o.step(1)
        assert g.counters() == o.counters(), k
