"""Kernels at the sizes where they can go wrong: edges of tiles, remainders of splits, the smallest and the largest of a range."""
import pytest
import torch

from tilerl_b200.ops import ref

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from tilerl_b200.ops.cuda import CudaOps
    return CudaOps(DEV)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("m,n,k,shift", [
    (1, 1, 32, 0), (2, 17, 96, 0), (8, 15, 544, 0), (9, 33, 512, 0), (16, 40, 1056, 0), (1, 16 * 149, 5120, 0), (3, 4100, 5120, 8),
    (5, 2500, 2592, 1), (8, 700, 13824, 0), (16, 900, 6240, 0), (16, 900, 6656, 0), (7, 64, 13856, 0), (16, 64, 6688, 0),
    (1, 19000, 1024, 0), (13, 19001, 1280, 0), (4, 10100, 2560, 0), (16, 9999, 2048, 4)])
def test_bf16_rows_for_every_split_of_k(ops, m, n, k, shift):
    """K shorter than the 16 warps that share it (4 or 8 with many rows), shared unevenly, and up to what shared memory holds with two, one and no
    reduction buffers; rows that are no multiple of a tile; activations that start off a 16-byte boundary.  Products of bf16
    values are exact in fp32, so sums differ from 64 bits by fp32 rounding alone: below k * 2^-24 of the summed magnitudes,
    and their square root's share of it on average."""
    g = torch.Generator().manual_seed(m * 7 + n + k)
    w = (torch.randn(n, k, generator=g) * 0.02).to(DEV, torch.bfloat16)
    x = torch.randn(m, k + shift, generator=g).to(DEV, torch.bfloat16)[:, shift:]
    res = torch.randn(m, n, generator=g).to(DEV, torch.bfloat16)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
    ops.gemv_now(x, w, y, epi=3)
    want = x.double() @ w.double().t()
    assert _rel(y, want) < 2e-6 * (1 + k ** 0.5 / 16)
    yr = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.gemv_now(x, w, yr, residual=res, epi=1)
    assert _rel(yr, want + res.double()) < 2 ** -8
    # a row's norm: one step of bf16 where the reciprocal root's last bit tips a rounding over (about one in 10^4 elements)
    nw = (1.0 + 0.1 * torch.randn(k, generator=g)).to(DEV)
    ops.gemv_now(x, w, y, norm_w=nw, eps=1e-6, epi=3)
    h = ref.rmsnorm(x, nw, 1e-6).to(torch.bfloat16)
    assert _rel(y, h.double() @ w.double().t()) < 2e-4 + 2 ** -8 / k ** 0.5
