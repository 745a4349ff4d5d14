"""Waits that run out in the tensor-core kernels.  The library is compiled once
more with a limit of no polls, so that every bounded wait but the draining of
issued products ends at once: each kernel returns, counts its blocks, and leaves
zeros for its products (bias, ReLU and residual applied to them).  Blocks that
need no wait are not affected.  A network on that library raises where it looks."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

from sdem_gb300 import build, surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"
L = 128


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("waits") / "libsdem_surrogate_nowait.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-DSDEM_SG_WAIT_LIMIT=0", "-o", path, build.SG_SRC, "-lcudart"],
                   check=True)
    build.build()
    real = sg.load()
    sg._lib = None
    short = sg.load(path)
    sg._lib = real
    return short


def bf16(*shape, scale=0.5, seed=1):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


def lost(lib):
    c = ctypes.c_uint(0)
    assert lib.sdem_sg_tensor_timeouts(ctypes.byref(c)) == 0
    return c.value


def gemm(lib, I, J, R, a, b, splits=1, partial=None, **ep):
    assert lib.sdem_sg_gemm(I, J, R, ctypes.byref(a.o), ctypes.byref(b.o), ctypes.byref(sg._ep(**ep)), splits,
                            sg._ptr(partial), sg._stream()) == 0


# rows of the persistent kernel (R <= 384 with J = 128) and of the tiled one
@pytest.mark.parametrize("R", [128, 384, 512])
@pytest.mark.parametrize("reads", [False, True])
def test_rows(lib, R, reads):
    I = 300
    x, w = bf16(I, R), bf16(L, R, seed=2)
    bias, resid = torch.randn(L, device=DEV), torch.randn((I, L), device=DEV)
    out, res = torch.full((I, L), 7.0, device=DEV), torch.full((I, L), 7.0, device=DEV)
    more = dict(resid=resid, ld_resid=L, res_out=res, ld_res_out=L) if reads else {}
    before = lost(lib)
    gemm(lib, I, L, R, sg._Op(0, (x, 0, R, R, None)), sg._Op(0, (w, 0, R, R, None)), bias=bias, out=out, ld_out=L, **more)
    assert lost(lib) - before == 3          # row tiles
    assert torch.equal(out, bias.expand(I, L))
    if reads:
        assert torch.equal(res, resid + bias)


@pytest.mark.parametrize("splits", [1, 3])
def test_weight_gradient(lib, splits):
    R = 64 * 60                             # 60 slices, 20 a split: more than the ring holds
    x, y = bf16(R, L), bf16(R, L, seed=2)
    a, b = sg._Op(1, (x, 0, L, L, None)), sg._Op(1, (y, 0, L, L, None))
    out = torch.full((L, L), 7.0, device=DEV)
    partial = torch.full((splits * L * L,), 7.0, device=DEV)
    before = lost(lib)
    gemm(lib, L, L, R, a, b, splits=splits, partial=partial, out=out, ld_out=L)
    assert lost(lib) - before == splits
    assert torch.equal(out, torch.zeros_like(out))


def test_without_a_wait(lib):
    R = 192                                 # three slices: nothing to wait for but the products' end
    x, y = bf16(R, L), bf16(R, L, seed=2)
    out = torch.full((L, L), 7.0, device=DEV)
    before = lost(lib)
    gemm(lib, L, L, R, sg._Op(1, (x, 0, L, L, None)), sg._Op(1, (y, 0, L, L, None)), out=out, ld_out=L)
    want = x.double().T @ y.double()
    assert lost(lib) == before
    assert (out.double() - want).abs().max() <= 1e-4 * (x.double().abs().T @ y.double().abs()).max()


@pytest.mark.parametrize("agg", [False, True])
def test_two_layers(lib, agg):
    M, R, n = 2000, 3 * L, 100
    x, e = bf16(n, L), bf16(M, L, seed=2)
    dst = torch.arange(n, dtype=torch.int32, device=DEV).repeat_interleave(M // n)
    row_off = torch.arange(n + 1, dtype=torch.int32, device=DEV) * (M // n)
    w1, w2, b1, b2 = bf16(L, R, seed=3), bf16(L, L, seed=4), torch.randn(L, device=DEV), torch.randn(L, device=DEV)
    a = sg._Op(0, (x, 0, L, L, dst), (x, 0, L, L, dst), (e, 0, L, L, None))
    resid = torch.randn((M, L), device=DEV)
    z, out, outb = bf16(M, L, seed=5), torch.full((M, L), 7.0, device=DEV), bf16(M, L, seed=6)
    sums = bf16(n, L, seed=7)
    p = sg._ptr
    before = lost(lib)
    assert lib.sdem_sg_mlp(M, R, ctypes.byref(a.o), p(w1), p(b1), p(w2), p(b2), L, p(z), p(resid), p(out), p(outb),
                           n if agg else 0, p(row_off) if agg else None, p(dst) if agg else None,
                           p(sums) if agg else None, sg._stream()) == 0
    assert lost(lib) - before == 16         # blocks: 2000 rows in tiles of 128
    assert not z.any()
    assert torch.equal(out, resid) and torch.equal(outb, resid.to(torch.bfloat16))
    if agg:
        assert not sums.any()


def test_network_raises(lib, monkeypatch):
    monkeypatch.setattr(sg, "_lib", lib)
    rng = np.random.default_rng(3)
    n, d = 500, 1.2e-3
    p = np.c_[rng.uniform(0, 9e-3, (n, 3)), np.full(n, 0.5 * d)]
    g = sg.build_graph(torch.from_numpy(p).to(DEV), sg.make_grid((0, 0, 0), (9e-3,) * 3, d))
    net = sg.Network(seed=1)
    net.check_waits()                       # what ran out before the network was made is not its own
    net.forward(g, bf16(n, sg.NODE_IN), keep=False)
    with pytest.raises(RuntimeError, match="wait ran out"):
        net.check_waits()
    sample = sg.DeviceSample(g, bf16(n, sg.NODE_IN), torch.zeros((n, 6), device=DEV))
    with pytest.raises(RuntimeError, match="wait ran out"):
        sg.evaluate(sg.Network(seed=1), [sample])
