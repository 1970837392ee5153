"""NVFP4 GEMM on pairs of SMs: outputs and residuals that are not whole vectors of eight rows (a tensor-parallel rank's 2060 rows), on a B200."""
import statistics

import pytest
import torch

from tilerl_b200 import formats as F
from tilerl_b200.ops import native
from tilerl_b200.ops.gemm_tc import gemm_nvfp4

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from tilerl_b200.ops.cuda import CudaOps
    return CudaOps()


def _rel(a, b):
    a, b = a.double().flatten(), b.double().flatten()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def _room(rows, width, stride, off, dtype):
    """``[rows, width]`` in a buffer of NaN, ``off`` values from its start, rows ``stride`` values apart; and the buffer."""
    buf = torch.full((off + rows * stride + 8,), float("nan"), dtype=dtype, device=DEV)
    return buf[off:off + rows * stride].view(rows, stride)[:, :width], buf


@pytest.mark.parametrize("tokens,terms", [(1, 4), (9, 4), (31, 2), (65, 2), (97, 1), (300, 2)])
@pytest.mark.parametrize("n,k,pad,off", [(2060, 5120, 0, 0), (1001, 544, 0, 0), (264, 544, 3, 0), (264, 544, 8, 1), (264, 544, 8, 0), (1030, 4128, 2, 0), (1288, 288, 4, 4)])
def test_outputs_that_are_not_whole_vectors(ops, tokens, terms, n, k, pad, off):
    """Rows that are no multiple of eight, strides and bases off the vectors, an output and a residual of unlike strides, every
    epilogue: against one CTA alone (the one-SM kernel), and nothing written beside the rows."""
    g = torch.Generator().manual_seed(tokens + n)
    w = F.quantize_nvfp4(torch.randn(n, k, generator=g) * 0.02).to(DEV)
    x = torch.randn(tokens, k, generator=g).to(DEV, torch.bfloat16)
    want = torch.empty(tokens, n, device=DEV)
    gemm_nvfp4(ops, x, w, want, terms=terms, epi=3, max_ctas=1, split=False)
    r, _ = _room(tokens, n, n + pad + 1, off, torch.bfloat16)
    r.copy_(torch.randn(tokens, n, generator=g))
    h = n // 2 * 2
    half = torch.nn.functional.silu(want[:, 0:h:2].double()) * want[:, 1:h:2].double()
    # fp32 sums in another order 1e-6; bf16 results half an ulp each, 2^-9, of values that the sums' order moves by less
    for epi, dtype, width, ref, tol in ((3, torch.float32, n, want, 1e-6), (0, torch.bfloat16, n, want, 2 ** -8), (1, torch.bfloat16, n, want.double() + r.double(), 2 ** -8),
                                        (2, torch.bfloat16, n // 2, half, 2 ** -8)):
        if epi == 2 and n % 2:
            continue
        y, buf = _room(tokens, width, width + pad, off, dtype)
        gemm_nvfp4(ops, x, w, y, terms=terms, epi=epi, residual=r if epi == 1 else None)
        assert _rel(y, ref) < tol, epi
        assert int(torch.isnan(buf).sum()) == buf.numel() - tokens * width, epi
    assert native.read_error()[0] == 0


@pytest.mark.parametrize("tokens", [128, 512, 2000])
def test_rows_that_are_no_multiple_of_eight_cost_little_more(ops, tokens):
    """2060 rows and a residual against 2064: the same tiles on the same kernel.  (As whole tiles on the one-SM kernel they took
    2.2, 1.9 and 1.7 times as long.)"""
    k, times, graphs, kept = 5120, {}, {}, []         # kept: what the graphs read and write
    x = torch.randn(tokens, k, device=DEV).to(torch.bfloat16)
    for n in (2060, 2064):
        ws, y = [F.quantize_nvfp4(torch.randn(n, k, device=DEV) * 0.02) for _ in range(4)], torch.zeros(tokens, n, dtype=torch.bfloat16, device=DEV)
        kept.append((ws, y))
        run = lambda: [gemm_nvfp4(ops, x, ws[j % 4], y, terms=2, epi=1, residual=y) for j in range(16)]
        run()
        torch.cuda.synchronize()
        kept.extend(ops.ws.bufs.values())              # (a larger buffer may take a name's place later)
        graphs[n], times[n] = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graphs[n]):
            run()
    for i in range(25):
        for n, g in graphs.items():
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            if i >= 5:
                times[n].append((a, b))
    torch.cuda.synchronize()
    us = {n: statistics.median(a.elapsed_time(b) for a, b in t) for n, t in times.items()}
    assert us[2060] < 1.45 * us[2064], us


def test_one_sm_as_asked_for(ops, monkeypatch):
    """``TRL_GEMM_PAIR=0``: by its own rules the one-SM kernel gives what it gives when asked for by the number of CTAs, and needs scratch
    where it splits tiles, which the form on pairs never does."""
    lib = ops.lib
    assert lib.trl_gemm_nvfp4_scratch_bytes(8, 4, 5120, 17408, 0, -1) == 0 < lib.trl_gemm_nvfp4_scratch_bytes(8, 4, 5120, 17408, 0, -2)
    assert lib.trl_gemm_nvfp4_scratch_bytes(8, 4, 5120, 17408, 0, 2) == 0
    g = torch.Generator().manual_seed(0)
    w = F.quantize_nvfp4(torch.randn(1288, 4128, generator=g) * 0.02).to(DEV)
    x = torch.randn(100, 4128, generator=g).to(DEV, torch.bfloat16)
    want, got = torch.empty(100, 1288, device=DEV), torch.empty(100, 1288, device=DEV)
    gemm_nvfp4(ops, x, w, want, terms=2, epi=3, max_ctas=1, split=False)
    monkeypatch.setattr("tilerl_b200.ops.gemm_tc._PAIR", False)
    gemm_nvfp4(ops, x, w, got, terms=2, epi=3, split=False)
    assert torch.equal(got, want)
    gemm_nvfp4(ops, x, w, got, terms=2, epi=3)
    assert _rel(got, want) < 1e-6
