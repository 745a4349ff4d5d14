"""Steps whose pairs pass the contact capacity (SDEM_E_CL_FULL): the pairs of the
overflowing chunk are left out, the walls are not.  The reference is the same bed
with pair forces of zero stiffness, damping and friction, which moves by its
walls and gravity alone."""
from dataclasses import replace

import numpy as np
import pytest

from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem, SdemError

pytestmark = pytest.mark.gpu

E_CL_FULL = 3


def crowded(n):
    case = beds.lattice_cloud_case(n, seed=99)   # about 1.5 pairs a sphere, walls touched
    small = replace(case, opts=replace(case.opts, cntct_list_size=1))
    walls_only = replace(case, tables=replace(case.tables, bpp=np.zeros_like(case.tables.bpp)))
    return small, walls_only


def step_with_error(g):
    with pytest.raises(SdemError) as e:
        g.step(1)
    assert e.value.code == E_CL_FULL


# sums and update in one kernel, and in two
@pytest.mark.parametrize("n", [1500, 131500])
def test_walls_hold_when_pairs_overflow(gpu_lib, n):
    small, walls_only = crowded(n)
    g, w = DEMSystem(small), DEMSystem(walls_only)
    for k in range(3):   # the walls' histories pass from step to step
        step_with_error(g)
        w.step(1)
        assert w.counters()["pp"] > 1.2 * n and w.counters()["pw"] > 50
        a, b = g.state(), w.state()
        np.testing.assert_array_equal(a.id, b.id)
        for f in ("posR", "linVel", "linAcc", "theta", "rotVel", "rotAcc"):
            np.testing.assert_array_equal(getattr(a, f), getattr(b, f), err_msg=f"{f} step {k}")
        for x, y in zip(g.forces(), w.forces()):
            np.testing.assert_array_equal(x, y)


def records(s, base_wall_id):
    o, q, t, v = s.contacts()
    wall = q > base_wall_id
    return (np.stack([o[wall], q[wall]]), np.concatenate([t[wall], v[wall][:, None]], axis=1)), int((~wall).sum())


def test_records_after_an_overflow(gpu_lib):
    """The contact list holds what was computed: the walls', and the pairs of
    the chunks before the overflow."""
    small, walls_only = crowded(20000)
    g, w = DEMSystem(small), DEMSystem(walls_only)
    step_with_error(g)
    w.step(1)
    base = small.opts.base_wall_id
    (kg, hg), pairs = records(g, base)
    (kw, hw), _ = records(w, base)
    assert pairs == 0 and kg.shape[1] > 100
    np.testing.assert_array_equal(kg, kw)
    np.testing.assert_array_equal(hg, hw)
    # the first of four chunks holds a tenth of the targets: its pairs fit
    g = DEMSystem(small)
    g.set_launch(pipeline_chunks=4, first_chunk_percent=10)
    step_with_error(g)
    _, pairs = records(g, base)
    assert 0 < pairs <= 2 * 20000   # each under both its spheres
