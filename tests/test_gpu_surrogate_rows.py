"""Row-wise kernels of the backward pass at the edges of their vector forms,
against numpy in the same order of fp32 additions: the gathered sum (eight
columns a thread, or one where a width, stride or address does not allow it)
and the column sums (128-float rows through shared memory, or one thread per
column), for row counts around a chunk's and a tile's ends."""
import numpy as np
import pytest
import torch

from sdem_gb300 import build, surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"
CHUNKS = 160


@pytest.fixture(scope="module")
def lib():
    build.build()
    return sg.load()


@pytest.mark.parametrize("M", [1, 31, 32, 159, 160, 161, 5119, 5120, 5121, 20000])
@pytest.mark.parametrize("J,ld,off", [(128, 128, 0), (128, 256, 4), (128, 129, 0), (128, 128, 1), (16, 16, 0)])
def test_column_sums(lib, M, J, ld, off):
    rng = np.random.default_rng(M + ld)
    buf = rng.normal(size=M * ld + 8).astype(np.float32)
    x = buf[off:off + M * ld].reshape(M, ld)[:, :J]
    chunk = -(-M // CHUNKS)
    parts = np.zeros((CHUNKS, J), np.float32)
    for b in range(CHUNKS):
        for r in x[b * chunk:(b + 1) * chunk]:
            parts[b] += r
    total = np.zeros(J, np.float32)
    for b in range(CHUNKS):
        total += parts[b]
    start = rng.normal(size=J).astype(np.float32)
    xd, out = torch.from_numpy(buf).to(DEV), torch.from_numpy(start).to(DEV)
    partial = torch.full((CHUNKS * J,), float("nan"), device=DEV)
    assert lib.sdem_sg_colsum(M, J, sg._ptr(xd, off), ld, sg._ptr(out), 1, sg._ptr(partial), sg._stream()) == 0
    np.testing.assert_array_equal(out.cpu().numpy(), start + total)


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 4097])
@pytest.mark.parametrize("J,ldx,ldo,off", [(128, 256, 128, 0), (128, 128, 136, 0), (128, 128, 129, 0), (8, 8, 8, 1), (12, 12, 12, 0)])
def test_gathered_sum(lib, rows, J, ldx, ldo, off):
    rng = np.random.default_rng(rows + J)
    n = 37
    x, y = rng.normal(size=n * ldx + 8).astype(np.float32), rng.normal(size=(rows, J)).astype(np.float32)
    idx = rng.integers(0, n, rows).astype(np.int32)
    xs = x[off:off + n * ldx].reshape(n, ldx)[:, :J]
    xd, yd, id_ = (torch.from_numpy(a).to(DEV) for a in (x, y, idx))
    for with_idx in (True, False):
        if not with_idx and rows > n:
            continue
        for with_y in (True, False):
            want = xs[idx] if with_idx else xs[:rows]
            want = y + want if with_y else want
            out = torch.full((rows, ldo), 5.0, device=DEV)
            outb = torch.zeros((rows, J), dtype=torch.bfloat16, device=DEV)
            assert lib.sdem_sg_gather_add(rows, J, sg._ptr(id_) if with_idx else None, sg._ptr(xd, off), ldx,
                                          sg._ptr(yd) if with_y else None, J, sg._ptr(out), ldo, sg._ptr(outb), J,
                                          sg._stream()) == 0
            got = out.cpu().numpy()
            np.testing.assert_array_equal(got[:, :J], want)
            assert np.all(got[:, J:] == 5.0)
            assert torch.equal(outb, out[:, :J].to(torch.bfloat16))
