"""Spheres outside the padded search grid (SDEM_E_GRID), with sums and update in
one kernel and in two (131,072 search positions): the error is reported by the
step that meets them, every other sphere advances by exactly that step, to the
bits of a bed without the strays, and a stray outside the domain is deleted at
the end of it.  One with a NaN position stays, and is reported by every step."""
from dataclasses import replace

import numpy as np
import pytest

from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem, SdemError

pytestmark = pytest.mark.gpu

E_GRID = 6
SIZES = [900, 131500]


def beds_with_and_without(n, strays, where):
    case = beds.lattice_cloud_case(n, seed=97, nn=1.12e-3)
    p = case.particles
    keep = np.setdiff1d(np.arange(p.n), strays)
    clean = replace(case, particles=p.take(keep))
    q = p.copy()
    q.linVel[strays] = 0.0   # (the largest velocity sets the wall list's next refresh)
    q.posR[strays, :3] = np.array(case.opts.maxpoint) + 20e-3 if where == "outside" else np.nan
    return DEMSystem(replace(case, particles=q)), DEMSystem(clean, n_capacity=p.n, max_gid=int(p.id.max()))


def step_with_error(g):
    with pytest.raises(SdemError) as e:
        g.step(1)
    assert e.value.code == E_GRID


def assert_same(g, c, ids=None):
    a, b = g.state(), c.state()
    oa, ob = np.argsort(a.id), np.argsort(b.id)
    if ids is not None:
        oa = oa[np.isin(a.id[oa], ids)]
    np.testing.assert_array_equal(a.id[oa], b.id[ob])
    for f in ("posR", "linVel", "linAcc", "theta", "rotVel", "rotAcc"):
        np.testing.assert_array_equal(getattr(a, f)[oa], getattr(b, f)[ob], err_msg=f)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("count", [1, 2, 40])
def test_strays_at_the_end_are_deleted(gpu_lib, n, count):
    g, c = beds_with_and_without(n, np.arange(n - count, n), "outside")
    step_with_error(g)
    c.step(1)
    assert c.counters()["pp"] > n // 20
    assert_same(g, c)
    assert g.state().n == n - count
    for _ in range(3):   # no error any more: the indices are those of the clean bed
        g.step(1)
        c.step(1)
        assert g.counters() == c.counters()
        assert_same(g, c)


@pytest.mark.parametrize("n", SIZES)
def test_strays_among_the_others(gpu_lib, n):
    """The delete moves spheres from the end to the strays' indices."""
    g, c = beds_with_and_without(n, np.array([0, 5, n // 2]), "outside")
    step_with_error(g)
    c.step(1)
    assert_same(g, c)
    g.step(2)


@pytest.mark.parametrize("n", SIZES)
def test_a_nan_position(gpu_lib, n):
    g, c = beds_with_and_without(n, np.array([n - 1]), "nan")
    for _ in range(3):
        step_with_error(g)
        c.step(1)
        assert_same(g, c, ids=c.state().id)
        assert g.state().n == n


def test_off_grid_in_chunks(gpu_lib):
    """The same with the search in three chunks: the strays' positions fall into the last."""
    n = 40000
    g, c = beds_with_and_without(n, np.arange(n - 3, n), "outside")
    for s in (g, c):
        s.set_launch(pipeline_chunks=3)
    step_with_error(g)
    c.step(1)
    assert_same(g, c)
    g.step(2)
    c.step(2)
    assert_same(g, c)
