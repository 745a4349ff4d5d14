"""The device graph build against the library's single steps (every candidate
in FP64, sorts and prefix sums by torch), bit for bit: offsets, edges and their
order, features.  Beds of one sphere up to several scan tiles; pairs exactly at
the cutoff; more neighbours than the list between the two calls holds; spheres
outside the grid, NaN positions; grids of one cell, of cells wider than the
cutoff, and of more cells than one scan launch takes."""
import ctypes

import numpy as np
import pytest
import torch

from sdem_gb300 import build, surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 1.2e-3


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    return sg.load()


def bed(name, rng):
    """(posR, grid lo, grid hi)"""
    def cloud(n, side):
        return np.c_[rng.uniform(0, side, (n, 3)), rng.uniform(0.4e-3, 0.6e-3, n)], (0, 0, 0), (side,) * 3

    if name.startswith("n"):
        n = int(name[1:])
        return cloud(n, D * (n / 1.2) ** (1 / 3))
    if name == "lattice":              # 1.5 D is the cutoff: many pairs lie on it, or one rounding beside it
        g = np.stack(np.meshgrid(*[np.arange(12)] * 3, indexing="ij"), -1).reshape(-1, 3) * (0.75 * D)
        g = g + rng.integers(-1, 2, g.shape) * 2.0 ** -62
        return np.c_[g, np.full(len(g), 0.5e-3)], (0, 0, 0), tuple(g.max(0))
    if name == "dense":                # hundreds of neighbours
        return cloud(3000, 3.5 * D)
    if name == "outside":
        p, lo, hi = cloud(2500, 10 * D)
        p[:, :3] += rng.normal(0, 4 * D, (len(p), 3)) * (rng.random((len(p), 1)) < 0.3)
        p[7, 0] = np.nan
        p[11, 1] = np.inf
        return p, lo, hi
    if name == "one_cell":
        return cloud(40, 0.3 * D)
    if name == "wide_grid":            # 1.9M cells
        return cloud(4000, 14 * D)[0], (0, 0, 0), (0.22,) * 3
    raise ValueError(name)


@pytest.mark.parametrize("name", ["n1", "n2", "n255", "n257", "n4096", "n4097", "n20011", "lattice", "dense", "outside",
                                  "one_cell", "wide_grid"])
@pytest.mark.parametrize("wider", [1.0, 1.37])
def test_same_graph(name, wider):
    p, lo, hi = bed(name, np.random.default_rng(len(name)))
    posR = torch.from_numpy(p).to(DEV)
    grid = sg.make_grid(lo, hi, D)
    grid.cell = grid.cell * wider      # the cutoff stays
    a = sg._edges_on_device(posR, grid)
    b = sg._edges_by_steps(posR, grid)
    assert a[4] == b[4]
    if name in ("lattice", "dense"):
        assert a[4] > 10 * len(p)
    for x, y, what in zip(a[:4], b[:4], ("row_off", "dst", "src", "efeat")):
        assert torch.equal(x[:len(y)].view(torch.int16) if what == "efeat" and a[4] else x,
                           y.view(torch.int16) if what == "efeat" and a[4] else y) or a[4] == 0, what


def test_rows_of_a_larger_array():
    p, lo, hi = bed("n4096", np.random.default_rng(3))
    wide = torch.from_numpy(np.c_[p, p]).to(DEV)
    grid = sg.make_grid(lo, hi, D)
    a, b = sg.build_graph(wide[:, :4], grid), sg.build_graph(torch.from_numpy(p).to(DEV), grid)
    assert a.E == b.E and torch.equal(a.src, b.src) and torch.equal(a.efeat, b.efeat)


def test_refused_arguments(lib):
    p, lo, hi = bed("n255", np.random.default_rng(3))
    posR = torch.from_numpy(p).to(DEV)
    grid = sg.make_grid(lo, hi, D)
    work = torch.empty(int(lib.sdem_sg_graph_work(255, ctypes.byref(grid))) + 256, dtype=torch.uint8, device=DEV)
    row = torch.empty(264, dtype=torch.int32, device=DEV)

    def call(n=255, g=grid, w=0, r=0):
        return lib.sdem_sg_graph_count(n, sg._ptr(posR), ctypes.byref(g), sg._ptr(work, w), sg._ptr(row, r), sg._stream())

    assert call() == 0
    assert call(n=0) == 1 and call(n=-1) == 1 and call(w=16) == 1 and call(r=1) == 1
    bad = sg.make_grid(lo, hi, D)
    bad.cutoff = bad.cell * 1.01
    assert call(g=bad) == 1
    bad.dim[0] = 0
    assert call(g=bad) == 1 and lib.sdem_sg_graph_work(255, ctypes.byref(bad)) == 0
    torch.cuda.synchronize()
