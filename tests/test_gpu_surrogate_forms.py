"""The tcgen05 GEMM kernels of the surrogate over the forms and edges of their
dispatch: whole and ragged row tiles, more tiles than SMs, one to three column
blocks, reductions below and across a 64-element slice, segments whose width
is no multiple of a slice, transposed B, accumulation and unaligned outputs,
and weight gradients with ragged splits.

Reference: float64 products of the same bf16 values.  Bound: fp32 accumulation
of R products loses at most R 2^-24 of their absolute sum (1e-4 covers R <= 1600;
the longer reductions here are split into chunks that are added in fp32)."""
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


def bf16(rng, shape, scale=1.0):
    return torch.from_numpy((rng.normal(size=shape) * scale).astype(np.float32)).to(torch.bfloat16).to(DEV)


def f64(t):
    return t.double().cpu().numpy()


def gemm(lib, I, J, R, a, b, splits=1, partial=None, **ep):
    assert lib.sdem_sg_gemm(I, J, R, ctypes.byref(a.o), ctypes.byref(b.o), ctypes.byref(sg._ep(**ep)), splits,
                            sg._ptr(partial), sg._stream()) == 0


def close(got, want, bound):
    err = np.abs(got - want)
    assert np.all(err <= 1e-4 * bound + 1e-30), float((err / (bound + 1e-30)).max())


def timeouts(lib):
    c = ctypes.c_uint(9)
    assert lib.sdem_sg_tensor_timeouts(ctypes.byref(c)) == 0
    return c.value


@pytest.mark.parametrize("M,J,widths", [
    (1, 128, (128,)), (127, 16, (16,)), (128, 128, (384,)), (129, 136, (72, 56)), (255, 384, (128,)),
    (300, 256, (128,)), (19457, 128, (128, 128, 128)), (40000, 32, (48, 80, 8)), (513, 48, (64, 40, 24))])
@pytest.mark.parametrize("trans_b", [0, 1])
def test_row_forms(lib, M, J, widths, trans_b):
    rng = np.random.default_rng(M + J)
    R, rows = sum(widths), 200
    segs, cols = [], []
    for k, w in enumerate(widths):
        gathered = k < len(widths) - 1 or len(widths) == 1
        src = bf16(rng, (rows if gathered else M, w))
        idx = torch.from_numpy(rng.integers(0, rows, M).astype(np.int32)).to(DEV) if gathered else None
        segs.append((src, 0, w, w, idx))
        cols.append(f64(src)[idx.cpu().numpy()] if gathered else f64(src))
    x = np.concatenate(cols, 1)
    W = bf16(rng, (R, J) if trans_b else (J, R), 0.1)
    w = f64(W) if trans_b else f64(W).T
    b_op = sg._Op(trans_b, (W, 0, J if trans_b else R, J if trans_b else R, None))
    bias = torch.from_numpy(rng.normal(size=J).astype(np.float32)).to(DEV)
    mask, resid = bf16(rng, (M, J)), torch.from_numpy(rng.normal(size=(M, J)).astype(np.float32)).to(DEV)
    bound = np.abs(x) @ np.abs(w) + np.abs(f64(bias))
    want = np.maximum(x @ w + f64(bias), 0.0) * (f64(mask) > 0)
    for ld, off in ((J, 0), (J + 8, 1)):   # aligned rows; odd start and stride: the scalar epilogue
        start = torch.from_numpy(rng.normal(size=M * ld + 8).astype(np.float32)).to(DEV)
        out, res = start.clone(), torch.zeros_like(start)
        outb = torch.zeros((M, J), dtype=torch.bfloat16, device=DEV)
        gemm(lib, M, J, R, sg._Op(0, *segs), b_op, bias=bias, relu=1, mask=mask, ld_mask=J, accumulate=1,
             out=sg._ptr(out, off), ld_out=ld, out_bf=outb, ld_out_bf=J, resid=resid, ld_resid=J,
             res_out=sg._ptr(res, off), ld_res_out=ld)
        view = lambda t: t[off:off + M * ld].view(M, ld)[:, :J]
        close(f64(view(out)) - f64(view(start)), want, bound + np.abs(f64(view(start))))
        close(f64(view(res)), want + f64(resid), bound + np.abs(f64(resid)))
        assert np.all(np.abs(f64(outb) - want) <= 2.0 ** -8 * np.abs(want) + 1e-4 * bound)
        keep = torch.ones_like(out, dtype=torch.bool)
        keep[off:off + M * ld].view(M, ld)[:, :J] = False
        assert torch.equal(out[keep], start[keep]), "written outside the rows"
    assert timeouts(lib) == 0


@pytest.mark.parametrize("I,widths,R,splits", [
    (128, (128,), 1, 1), (128, (128, 128, 128), 63, 1), (16, (128,), 65, 1), (128, (16,), 1500, 3),
    (128, (128, 128), 777, 5), (128, (72, 56, 16), 1300, 4), (256, (136,), 900, 2)])
def test_weight_gradient_forms(lib, I, widths, R, splits):
    rng = np.random.default_rng(I + R)
    J, rows = sum(widths), 150
    dy = bf16(rng, (R, I))
    segs, cols = [], []
    for k, w in enumerate(widths):
        src = bf16(rng, (rows if k == 0 else R, w))
        idx = torch.from_numpy(rng.integers(0, rows, R).astype(np.int32)).to(DEV) if k == 0 else None
        segs.append((src, 0, w, w, idx))
        cols.append(f64(src)[idx.cpu().numpy()] if k == 0 else f64(src))
    x = np.concatenate(cols, 1)
    start = torch.from_numpy(rng.normal(size=(I, J)).astype(np.float32)).to(DEV)
    out = start.clone()
    partial = torch.full((splits * I * J,), float("nan"), device=DEV)
    gemm(lib, I, J, R, sg._Op(1, (dy, 0, I, I, None)), sg._Op(1, *segs), splits, partial if splits > 1 else None,
         out=out, ld_out=J, accumulate=1)
    close(f64(out) - f64(start), f64(dy).T @ x, np.abs(f64(dy)).T @ np.abs(x) + np.abs(f64(start)))
    assert timeouts(lib) == 0
