"""The two-layer kernel (sdem_sg_mlp) against the calls it stands for, bit for
bit: every optional output, both output widths, ragged row counts from one row
to several tiles per SM, and the per-receiver sums over graphs whose receivers
have no rows, a few, more than a tile of 128 and more than a CTA's share; then
the network's forward pass with and without it."""
import ctypes

import numpy as np
import pytest
import torch

from sdem_gb300 import build, surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def lib():
    build.build()
    return sg.load()


def bf16(g, *shape, scale=0.5):
    return (torch.randn(shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


def gemm(lib, M, J, R, a, b, **ep):
    assert lib.sdem_sg_gemm(M, J, R, ctypes.byref(a.o), ctypes.byref(b.o), ctypes.byref(sg._ep(**ep)), 1, None,
                            sg._stream()) == 0


@pytest.fixture(autouse=True)
def no_wait_ran_out(lib):
    yield
    c = ctypes.c_uint(9)
    assert lib.sdem_sg_tensor_timeouts(ctypes.byref(c)) == 0 and c.value == 0


def receivers(kind, rng):
    """rows per receiver"""
    return {"few": rng.integers(0, 4, 300), "one": np.array([1]), "none_then_many": np.array([0, 0, 700, 0, 129, 128, 0]),
            "packed": rng.integers(12, 30, 4000), "huge": np.array([3, 90000, 1, 0, 2]),
            "tile": np.full(500, 128)}[kind]


@pytest.mark.parametrize("kind", ["few", "one", "none_then_many", "packed", "huge", "tile"])
def test_edge_block(lib, kind):
    deg = receivers(kind, np.random.default_rng(5))
    n, M, L = len(deg), int(deg.sum()), 128
    g = torch.Generator(device=DEV).manual_seed(7)
    row_off = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    row_off[1:] = torch.from_numpy(np.cumsum(deg)).to(DEV)
    dst = torch.from_numpy(np.repeat(np.arange(n), deg).astype(np.int32)).to(DEV)
    src = torch.randint(0, n, (M,), device=DEV, generator=g, dtype=torch.int32)
    h, e, resid = bf16(g, n, L), bf16(g, M, L), torch.randn((M, L), device=DEV, generator=g)
    w1, w2 = bf16(g, L, 3 * L, scale=0.07), bf16(g, L, L, scale=0.1)
    b1, b2 = torch.randn(L, device=DEV, generator=g), torch.randn(L, device=DEV, generator=g)
    a = sg._Op(0, (h, 0, L, L, dst), (h, 0, L, L, src), (e, 0, L, L, None))
    z, zb = torch.empty((M, L), dtype=torch.bfloat16, device=DEV), torch.empty((M, L), dtype=torch.bfloat16, device=DEV)
    m, want, wantb = torch.empty((M, L), device=DEV), torch.empty((M, L), device=DEV), torch.empty_like(zb)
    agg = torch.zeros((n, L), dtype=torch.bfloat16, device=DEV)
    gemm(lib, M, L, 3 * L, a, sg._Op(0, (w1, 0, 3 * L, 3 * L, None)), bias=b1, relu=1, out_bf=z, ld_out_bf=L)
    gemm(lib, M, L, L, sg._Op(0, (z, 0, L, L, None)), sg._Op(0, (w2, 0, L, L, None)), bias=b2, out=m, ld_out=L,
         resid=resid, ld_resid=L, res_out=want, ld_res_out=L, res_out_bf=wantb, ld_res_out_bf=L)
    assert lib.sdem_sg_segsum(n, L, sg._ptr(row_off), None, sg._ptr(m), L, None, L, 0, sg._ptr(agg), L,
                              sg._stream()) == 0
    got, gotb, gagg = resid.clone(), torch.empty_like(wantb), torch.zeros_like(agg)
    p = sg._ptr
    assert lib.sdem_sg_mlp(M, 3 * L, ctypes.byref(a.o), p(w1), p(b1), p(w2), p(b2), L, p(zb), p(got), p(got), p(gotb),
                           n, p(row_off), p(dst), p(gagg), sg._stream()) == 0
    for x, y in ((zb, z), (got, want), (gotb, wantb), (gagg, agg)):
        assert torch.equal(x, y), kind
    for _ in range(20):              # the sums alone, often enough to meet another order of the warps
        only = torch.zeros_like(agg)
        assert lib.sdem_sg_mlp(M, 3 * L, ctypes.byref(a.o), p(w1), p(b1), p(w2), p(b2), L, None, None, None, None, n,
                               p(row_off), p(dst), p(only), sg._stream()) == 0
        assert torch.equal(only, agg)


@pytest.mark.parametrize("M", [1, 127, 128, 129, 19456, 19457, 40000])
@pytest.mark.parametrize("R,J", [(16, 128), (32, 128), (128, 16), (256, 128)])
def test_node_and_encoder_blocks(lib, M, R, J):
    L = 128
    g = torch.Generator(device=DEV).manual_seed(M + R)
    x, w1, w2 = bf16(g, M, R), bf16(g, L, R, scale=0.1), bf16(g, J, L, scale=0.1)
    b1, b2 = torch.randn(L, device=DEV, generator=g), torch.randn(J, device=DEV, generator=g)
    a = sg._Op(0, (x, 0, R, R, None))
    z, out, outb = (torch.empty((M, L), dtype=torch.bfloat16, device=DEV), torch.empty((M, J), device=DEV),
                    torch.empty((M, J), dtype=torch.bfloat16, device=DEV))
    gemm(lib, M, L, R, a, sg._Op(0, (w1, 0, R, R, None)), bias=b1, relu=1, out_bf=z, ld_out_bf=L)
    gemm(lib, M, J, L, sg._Op(0, (z, 0, L, L, None)), sg._Op(0, (w2, 0, L, L, None)), bias=b2, out=out, ld_out=J,
         out_bf=outb, ld_out_bf=J)
    got, gotb = torch.empty_like(out), torch.empty_like(outb)
    p = sg._ptr
    assert lib.sdem_sg_mlp(M, R, ctypes.byref(a.o), p(w1), p(b1), p(w2), p(b2), J, None, None, p(got), p(gotb), 0, None,
                           None, None, sg._stream()) == 0
    assert torch.equal(got, out) and torch.equal(gotb, outb)


def test_refused_arguments(lib):
    t, f = torch.zeros(4096, dtype=torch.bfloat16, device=DEV), torch.zeros(4096, device=DEV)
    p = sg._ptr

    def call(M=8, R=128, J=128, widths=(128,), z=None, resid=None, out=f, agg=None):
        a = sg._Op(0, *[(t, 0, w, w, None) for w in widths])
        return lib.sdem_sg_mlp(M, R, ctypes.byref(a.o), p(t), p(f), p(t), p(f), J, p(z), p(resid), p(out), None, 1, None,
                               None, p(agg), sg._stream())

    assert call(R=392, widths=(392,)) == 1 and call(J=32) == 1 and call(widths=(64, 32)) == 1
    assert call(R=128, widths=(72, 56)) == 1                    # a segment that ends inside a slice
    assert call(out=f[1:]) == 1 and call(out=None) == 1         # unaligned; nothing to write
    assert call(agg=t) == 1                                     # sums without receivers
    assert call(M=0) == 0


def test_forward_is_the_same_with_and_without(lib):
    rng = np.random.default_rng(3)
    for n, E in ((1, 0), (50, 0), (700, 9000), (3000, 70000)):
        deg = np.bincount(rng.integers(0, n, E), minlength=n)
        row_off = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
        row_off[1:] = torch.from_numpy(np.cumsum(deg)).to(DEV)
        dst = torch.from_numpy(np.repeat(np.arange(n), deg).astype(np.int32)).to(DEV)
        src = torch.from_numpy(rng.integers(0, n, max(E, 1)).astype(np.int32)).to(DEV)[:E]
        g = torch.Generator(device=DEV).manual_seed(n)
        graph = sg.Graph(n, E, row_off, dst, src, bf16(g, max(E, 1), 16)[:E], None, None)
        xn = bf16(g, n, 32)
        net = sg.Network(seed=4)
        assert net.fused
        ys, kept = [], []
        for fused in (True, False):
            net.fused = fused
            for keep in (True, False):
                ys.append(net.forward(graph, xn, keep=keep))
                if keep:
                    kept.append(net.saved)
        assert all(torch.equal(ys[0], y) for y in ys[1:])
        for key in ("zb_enc", "zd"):
            assert torch.equal(kept[0][key], kept[1][key]), key
        for key in ("ze", "zn", "agg", "hb"):
            for a, b in zip(kept[0][key], kept[1][key]):
                assert torch.equal(a[:E] if key == "ze" else a, b[:E] if key == "ze" else b), key
        for a, b in zip(kept[0]["eb"][:-1], kept[1]["eb"][:-1]):
            assert torch.equal(a[:E], b[:E])
