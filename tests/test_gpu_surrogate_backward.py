"""The backward pass's fused gathers and sums give the bits of the calls that they
stand for: the sphere gradient (gather_add and two segment sums), the message
gradient with its column sums (gather_add and colsum), the epilogues that read
(mask, residual in place) in both widths of access, and the split reduction."""
import ctypes as C

import numpy as np
import pytest
import torch

from sdem_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"
F32, BF = torch.float32, torch.bfloat16


@pytest.fixture(scope="module")
def lib(gpu_lib):
    return sg.load()


def p(t, off=0):
    return C.c_void_p(t.data_ptr() + off * t.element_size()) if t is not None else None


def randn(seed, *shape, dtype=F32):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


def edges(n, E, seed):
    rng = np.random.default_rng(seed)
    dst = np.sort(rng.integers(0, n, E)).astype(np.int32)
    src = rng.integers(0, max(1, n - n // 3), E).astype(np.int32)   # some spheres send nothing

    def off(x):
        return torch.from_numpy(np.concatenate([[0], np.cumsum(np.bincount(x, minlength=n))]).astype(np.int32)).to(DEV)
    perm = torch.from_numpy(np.argsort(src, kind="stable").astype(np.int32)).to(DEV)
    return torch.from_numpy(dst).to(DEV), off(dst), off(src), perm


@pytest.mark.parametrize("n,E", [(1, 0), (5, 0), (3, 200), (9, 7), (257, 4000), (1000, 33), (4001, 90001)])
def test_sphere_grad(lib, n, E):
    dst, ro, so, perm = edges(n, E, n + E)
    x, y, d = randn(1, n, 256), randn(2, n, 128), randn(3, max(E, 1), 256)
    st = sg._stream()
    want, want_bf = torch.empty(n, 128, device=DEV), torch.empty(n, 128, device=DEV, dtype=BF)
    assert lib.sdem_sg_gather_add(n, 128, None, p(x), 256, p(y), 128, p(want), 128, None, 128, st) == 0
    assert lib.sdem_sg_segsum(n, 128, p(ro), None, p(d), 256, p(want), 128, 1, None, 128, st) == 0
    assert lib.sdem_sg_segsum(n, 128, p(so), p(perm), p(d, 128), 256, p(want), 128, 1, p(want_bf), 128, st) == 0
    out, out_bf = torch.empty_like(want), torch.empty_like(want_bf)
    assert lib.sdem_sg_sphere_grad(n, p(ro), p(so), p(perm), p(x), 256, p(y), p(d), p(out), p(out_bf), st) == 0
    assert torch.equal(out, want) and torch.equal(out_bf, want_bf)


@pytest.mark.parametrize("E", [0, 1, 63, 64, 65, 160, 10239, 10240, 10241, 70001])
def test_gather_add_sum(lib, E):
    n = 300
    dst, *_ = edges(n, E, E)
    x, y = randn(4, n, 256), randn(5, max(E, 1), 128)
    st, part = sg._stream(), torch.empty(lib.sdem_sg_colsum_blocks() * 128, device=DEV)
    v, bf = torch.empty(max(E, 1), 128, device=DEV), torch.zeros(max(E, 1), 128, device=DEV, dtype=BF)
    want, got = randn(6, 128), randn(6, 128)
    assert lib.sdem_sg_gather_add(E, 128, p(dst), p(x, 128), 256, p(y), 128, p(v), 128, p(bf), 128, st) == 0
    assert lib.sdem_sg_colsum(E, 128, p(v), 128, p(want), 1, p(part), st) == 0
    bf2 = torch.zeros_like(bf)
    assert lib.sdem_sg_gather_add_sum(E, p(dst), p(x, 128), 256, p(y), p(bf2), p(got), p(part), st) == 0
    assert torch.equal(bf, bf2) and torch.equal(want, got)


def test_refused_arguments(lib):
    t, b = randn(7, 64, 256), torch.empty(64, 256, device=DEV, dtype=BF)
    i, st = torch.zeros(65, dtype=torch.int32, device=DEV), sg._stream()
    assert lib.sdem_sg_sphere_grad(4, p(i), p(i), p(i), p(t), 100, p(t), p(t), p(t), p(b), st) == 1
    assert lib.sdem_sg_sphere_grad(4, p(i), p(i), p(i), p(t, 1), 256, p(t), p(t), p(t), p(b), st) == 1
    assert lib.sdem_sg_sphere_grad(4, p(i), None, p(i), p(t), 256, p(t), p(t), p(t), p(b), st) == 1
    assert lib.sdem_sg_gather_add_sum(4, None, p(t), 256, p(t), p(b), p(t), p(t), st) == 1
    assert lib.sdem_sg_gather_add_sum(4, p(i), p(t), 256, p(t, 2), p(b), p(t), p(t), st) == 1
    assert lib.sdem_sg_gather_add_sum(4, p(i), p(t), 130, p(t), p(b), p(t), p(t), st) == 1


# rows around a tile, a ragged last tile, several tiles a block; columns of one
# and two blocks and a block's odd half
@pytest.mark.parametrize("I", [1, 127, 128, 129, 20001, 45000])
@pytest.mark.parametrize("J", [32, 96, 128, 256])
def test_epilogues_that_read(lib, I, J):
    R = 128
    a, w = randn(8, I, R, dtype=BF), randn(9, R, J, dtype=BF)
    mask, resid = randn(10, I, J, dtype=BF), randn(11, I, J)
    st = sg._stream()

    def gemm(ep, ld=J):
        A, B = sg._Op(0, (a, 0, R, R, None)), sg._Op(1, (w, 0, J, J, None))
        assert lib.sdem_sg_gemm(I, J, R, C.byref(A.o), C.byref(B.o), C.byref(ep), 1, None, st) == 0

    plain = torch.empty(I, J, device=DEV)
    gemm(sg._ep(out=p(plain), ld_out=J))
    masked = torch.where(mask > 0, plain, torch.zeros_like(plain))
    for pad in (0, 1):   # a padded leading dimension takes the narrow accesses
        def rows(dtype, fill=None):
            t = torch.empty(I, J + pad, device=DEV, dtype=dtype)
            if fill is not None:
                t[:, :J] = fill
            return t
        ld, out, bf = J + pad, rows(F32), rows(BF)
        m, r, rb = rows(BF, mask), rows(F32, resid), rows(BF)
        gemm(sg._ep(mask=p(m), ld_mask=ld, out=p(out), ld_out=ld, out_bf=p(bf), ld_out_bf=ld))
        assert torch.equal(out[:, :J], masked) and torch.equal(bf[:, :J], masked.to(BF))
        gemm(sg._ep(resid=p(r), ld_resid=ld, res_out=p(r), ld_res_out=ld, res_out_bf=p(rb), ld_res_out_bf=ld))
        assert torch.equal(r[:, :J], resid + plain) and torch.equal(rb[:, :J], (resid + plain).to(BF))
        r = rows(F32, resid)
        gemm(sg._ep(mask=p(m), ld_mask=ld, resid=p(r), ld_resid=ld, res_out=p(out), ld_res_out=ld))
        assert torch.equal(out[:, :J], resid + masked)


@pytest.mark.parametrize("splits", [2, 7, 152, 160, 161, 333])
@pytest.mark.parametrize("I,J", [(128, 128), (16, 24), (128, 384)])
def test_split_reduction(lib, splits, I, J):
    R = 32 * splits + 8
    a, b = randn(12, R, I, dtype=BF), randn(13, R, J, dtype=BF)
    A, B = sg._Op(1, (a, 0, I, I, None)), sg._Op(1, (b, 0, J, J, None))
    start = randn(14, I, J + 8)
    out, part = start.clone(), torch.zeros(splits + 1, I, J, device=DEV)
    ep = sg._ep(out=p(out), ld_out=J + 8, accumulate=1)
    assert lib.sdem_sg_gemm(I, J, R, C.byref(A.o), C.byref(B.o), C.byref(ep), splits, p(part), sg._stream()) == 0
    n = -(-R // (-(-(-(-R // splits)) // 32) * 32))   # chunks of whole steps of 32
    s = torch.zeros(I, J, device=DEV)
    for z in range(n):
        s = s + part[z]
    assert torch.equal(out[:, :J], start[:, :J] + s) and torch.equal(out[:, J:], start[:, J:])
