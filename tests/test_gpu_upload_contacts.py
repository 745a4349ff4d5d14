"""A contact list uploaded between two steps: a wall record of a sphere that is
not near a wall belongs to no contact and is gone after the next step, for good;
the others go on as if nothing had been uploaded."""
import numpy as np
import pytest

from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem

pytestmark = pytest.mark.gpu


def test_wall_record_of_a_sphere_off_the_walls(gpu_lib):
    case = beds.lattice_cloud_case(2000, seed=101, vmax=0.02)
    g, c = DEMSystem(case), DEMSystem(case)
    for s in (g, c):
        s.step(3)
    o, q, t, v = g.contacts()
    base = case.opts.base_wall_id
    wall = int(q[q > base].min())
    x = g.state().posR[:, :3]
    far = int(np.argmin(np.abs(x - x.mean(axis=0)).max(axis=1)))
    assert not np.any((o == far) & (q > base))
    g.upload_contacts(np.append(o, far), np.append(q, wall), np.concatenate([t, [[1e-9, 2e-9, 3e-9]]]),
                      np.append(v, 0.25))
    for k in range(6):
        g.step(1)
        c.step(1)
        for a, b in zip(g.contacts(), c.contacts()):
            np.testing.assert_array_equal(a, b, err_msg=f"step {k}")
        np.testing.assert_array_equal(g.state().posR, c.state().posR)
