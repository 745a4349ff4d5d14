"""The cell scan of very large grids, in three launches (more than 12,288 tiles of
4,096 cells): spheres in the first cells, the last ones and both, several steps;
and the surrogate's graph in a box of that many cells."""
from dataclasses import replace

import numpy as np
import pytest

from oracle.oracle import OracleSystem
from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem
from tests.helpers import assert_step_matches

pytestmark = pytest.mark.gpu


def wide_case(side, where):
    case = beds.lattice_cloud_case(1300, seed=95)
    lo, p = np.array(case.opts.minpoint), case.particles
    top = p.posR[:, :3].max(axis=0) + 0.8e-3
    hi = lo + side
    move = {"first": [], "last": range(p.n), "both": range(0, p.n, 2)}[where]
    p.posR[list(move), :3] += hi - top
    return replace(case, opts=replace(case.opts, maxpoint=tuple(hi)))


@pytest.mark.parametrize("where", ["first", "last", "both"])
def test_three_launches(gpu_lib, where):
    case = wide_case(np.array([0.46, 0.46, 0.47]), where)   # 386 x 386 x 394 cells: 14,332 tiles
    g, o = DEMSystem(case), OracleSystem(case)
    g.step(1)
    o.step(1)
    assert g.counters() == o.counters() and g.counters()["pp"] > 100
    assert_step_matches(g, o, what=where, pre=case.particles, case=case)
    for k in range(4):
        g.step(1)
        o.step(1)
        assert g.counters() == o.counters(), k


def test_launches_of_a_step(gpu_lib):
    """One launch more beyond the line: the work of a scan stays linear in the cells."""
    count = []
    for side in (0.40, 0.46):
        g = DEMSystem(wide_case(np.array([side] * 3), "first"))
        g.step(1)
        before = g.launch_count()
        g.step(2)
        count.append((g.launch_count() - before) // 2)
    assert count[1] == count[0] + 1


def test_graph_in_a_wide_box(gpu_lib):
    import torch
    from sdem_gb300 import surrogate as sg
    case = beds.lattice_cloud_case(1300, seed=103)
    p = case.particles
    d = 1.0e-3
    p.posR[::2, :3] += 0.58
    grid = sg.make_grid((0.0, 0.0, 0.0), (0.6, 0.6, 0.6), d)
    assert grid.dim[0] * grid.dim[1] * grid.dim[2] > 12288 * 4096
    x = torch.from_numpy(p.posR.copy()).cuda()
    a = sg.build_graph(x, grid, sender_order=False)
    row_off, dst, src, efeat, E = sg._edges_by_steps(x, grid)
    assert a.E == E > 5000
    for u, v in ((a.row_off, row_off), (a.dst, dst), (a.src, src), (a.efeat, efeat[:E])):
        assert torch.equal(u, v)
