"""The step's kernels at the sizes where their tiles and dispatch rules change,
against the oracle from identical inputs: the cell scan in one launch and in
two (up to 256 tiles of 4,096 cells and beyond), whole and ragged last tiles;
the image compaction's 1,024-candidate tiles; sums and update in one kernel and
in two (131,072 search positions); the near-wall list after deletes, which move
particles to other indices between two refreshes of the masks."""
from dataclasses import replace

import numpy as np
import pytest

from oracle.oracle import OracleSystem
from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem
from tests.helpers import assert_step_matches

pytestmark = pytest.mark.gpu


def both(case, steps=1):
    g, o = DEMSystem(case), OracleSystem(case)
    g.step(steps)
    o.step(steps)
    return g, o


# ncell = nx*ny*nz of the padded grid: 16 tiles whole, one cell over, 256 tiles
# (the last of one launch) and more (two launches), few cells
@pytest.mark.parametrize("side", [8.0e-3, 33.0e-3, 120.0e-3, 150.0e-3, 180.0e-3])
def test_cell_scan_forms(gpu_lib, side):
    case = beds.lattice_cloud_case(1200, seed=81)
    lo = case.opts.minpoint
    big = replace(case, opts=replace(case.opts, maxpoint=tuple(max(h, l + side) for h, l in
                                                               zip(case.opts.maxpoint, lo))))
    g, o = both(big)
    assert g.counters()["pp"] > 500
    assert_step_matches(g, o, what=f"side {side}", pre=case.particles, case=case)


@pytest.mark.parametrize("n", [4, 255, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("periodic", [(1, 0, 0), (0, 1, 0), (1, 1, 1)])
def test_image_compaction(gpu_lib, n, periodic):
    # a few spheres sit in a box wide enough for the GPU's two search cells
    case = beds.periodic_lattice_case(max(n, 4), 83, periodic)
    hi = tuple(max(h, l + 2.6e-3) if p else h for h, l, p in
               zip(case.opts.maxpoint, case.opts.minpoint, periodic))
    case = replace(case, opts=replace(case.opts, maxpoint=hi))
    g, o = both(case)
    assert g.counters() == o.counters()
    assert_step_matches(g, o, what=f"{n} {periodic}")
    g.step(3)
    o.step(3)
    assert g.counters() == o.counters()


@pytest.mark.parametrize("n", [131071, 131072, 131073])
def test_sums_and_update_together_or_apart(gpu_lib, n):
    case = beds.lattice_cloud_case(n, seed=85, nn=1.12e-3)
    g, o = both(case)
    assert g.counters()["pp"] > n // 10
    assert_step_matches(g, o, what=str(n), pre=case.particles, case=case)


def test_near_wall_list_after_deletes(gpu_lib):
    """Spheres fall out through the missing floor every few steps while the
    side walls' masks stay as they are (refreshed every 100 steps at most):
    wall contacts and their forces follow the particles to their new indices."""
    case = beds.lattice_cloud_case(900, seed=87, vmax=0.05)
    case.walls.walls = case.walls.walls[1:]
    case.walls.flags = case.walls.flags[1:]
    p = case.particles
    rng = np.random.default_rng(5)
    low = np.argsort(p.posR[:, 1])[:80]
    p.linVel[low, :, 1] = -rng.uniform(20.0, 200.0, len(low))[:, None]
    g, o = DEMSystem(case), OracleSystem(case)
    deleted = 0
    for k in range(25):
        g.step(1)
        o.step(1)
        cg, co = g.counters(), o.counters()
        assert cg == co, f"step {k}"
        np.testing.assert_array_equal(g.state().id, o.state().id)
        deleted = case.particles.n - cg["nlocal"]
    assert deleted > 20 and cg["pw"] > 20
    Fg, Fo = g.forces()[0], o.forces()[0]
    scale = np.maximum(np.abs(Fo).max(axis=1), 1e-6 * np.abs(Fo).max())
    assert (np.abs(Fg - Fo).max(axis=1) / scale).max() < 1e-6   # free run: rounding differences grow
