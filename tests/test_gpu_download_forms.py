"""The state's download by one kernel into page-locked arrays against the copies
that pageable arrays take: one to three levels, ragged counts, fewer spheres
than rows, some of the arrays left out, arrays at an odd offset inside their
page-locked allocation, and page-locked and pageable arrays mixed."""
import ctypes as C
from dataclasses import replace

import numpy as np
import pytest
import torch

from sdem_gb300 import beds
from sdem_gb300.capi import DEMSystem

pytestmark = pytest.mark.gpu

NAMES = ("id", "ptype", "usrmark", "posR", "linVel", "linAcc", "theta", "rotVel", "rotAcc")


def arrays(g, pinned, offset=0):
    cap, ts, rs = g.cfg.n_capacity, g.cfg.tsize, g.cfg.rsize
    shapes = [(cap,)] * 3 + [(cap, 4), (cap, ts, 3), (cap, ts, 3), (cap, 3), (cap, rs, 3), (cap, rs, 3)]
    out = []
    for name, sh in zip(NAMES, shapes):
        dt = torch.int32 if len(sh) == 1 else torch.float64
        size = int(np.prod(sh))
        lock = pinned if isinstance(pinned, bool) else name in pinned
        buf = torch.full((size * (4 if dt == torch.int32 else 8) + 64,), 0x5a, dtype=torch.uint8, pin_memory=lock).numpy()
        shift = offset if dt == torch.float64 else 0
        raw = buf[shift:shift + size * (4 if dt == torch.int32 else 8)]
        out.append((buf, raw, sh, np.int32 if dt == torch.int32 else np.float64))
    return out


def download(g, arrs, skip=()):
    n = C.c_int()
    ptr = [C.c_void_p(None) if nm in skip else C.c_void_p(raw.ctypes.data) for nm, (_, raw, _, _) in zip(NAMES, arrs)]
    f = g.lib.sdem_download_particles
    keep, f.argtypes = f.argtypes, None
    try:
        assert f(g.h, C.byref(n), *ptr) == 0
    finally:
        f.argtypes = keep
    return n.value, {nm: raw.tobytes() for nm, (_, raw, _, _) in zip(NAMES, arrs)}, [b.tobytes() for b, *_ in arrs]


@pytest.mark.parametrize("n", [1, 31, 257, 5003])
@pytest.mark.parametrize("pi", [1, 2, 3])
def test_same_bytes_as_the_copies(gpu_lib, n, pi):
    case = beds.lattice_cloud_case(max(n, 8), seed=93, pi=pi, pri=pi)
    g = DEMSystem(case, n_capacity=max(n, 8) + 37)
    g.step(3)
    want = download(g, arrays(g, False))
    for offset in (0, 8, 16, 4):   # at 4 a double is misaligned for a kernel: the copies
        got = download(g, arrays(g, True, offset))
        assert got[0] == want[0]
        assert got[1] == want[1], offset
    mixed = download(g, arrays(g, ("posR", "linVel", "id")))
    assert mixed[:2] == want[:2]
    skip = ("ptype", "linAcc", "rotAcc", "theta")
    assert download(g, arrays(g, True), skip)[1] == download(g, arrays(g, False), skip)[1]


def test_bytes_past_the_rows_stay(gpu_lib):
    case = beds.lattice_cloud_case(500, seed=94)
    g = DEMSystem(case, n_capacity=640)
    g.step(1)
    arrs = arrays(g, True)
    n, _, whole = download(g, arrs)
    for (buf, raw, sh, dt), after in zip(arrs, whole):
        used = n * int(np.prod(sh[1:], dtype=np.int64)) * np.dtype(dt).itemsize
        assert set(after[used:]) == {0x5a}
