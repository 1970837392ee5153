"""Kernels over many tensors of a training step (AdamW, clipping) with tensors of unlike lengths, on a B200."""
import math
import statistics

import pytest
import torch

from tilerl_b200 import optim

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths", [(1,), (3, 5, 1023, 1024, 1025, 2047, 2048, 2049), (70001, 2, 4099) * 11 + (6,), (5_000_003, 7)])
def test_lengths_that_fill_no_vector_and_no_block(lengths):
    """Against the loop over the names on the CPU, norms against 64 bits: tails of one to three values, one block and one more, more than
    a launch's tensors, a long one beside a short one.  Each value is the same few fp32 operations on both sides."""
    g = torch.Generator().manual_seed(len(lengths))
    p0 = {str(i): torch.randn(n, generator=g) for i, n in enumerate(lengths)}
    g0 = {k: torch.randn(v.shape, generator=g) * 3 for k, v in p0.items()}
    p1, g1 = ({k: v.to(DEV) for k, v in d.items()} for d in (p0, g0))
    o0, o1 = optim.AdamW(p0, lr=1e-2, weight_decay=0.1), optim.AdamW(p1, lr=1e-2, weight_decay=0.1)
    want = math.sqrt(sum(float(v.double().pow(2).sum()) for v in g0.values()))
    for clip in (1e9, 0.5):
        assert abs(optim.clip_grad_norm(g0, clip) / optim.clip_grad_norm(g1, clip) - 1) < 1e-12
    assert abs(math.sqrt(sum(float(v.double().pow(2).sum()) for v in g1.values())) / 0.5 - 1) < 1e-5 and want > 0.5
    for _ in range(2):
        o0.step(g0), o1.step(g1)
    for k in p0:
        for a, b in ((g0[k], g1[k]), (o0.m[k], o1.m[k]), (o0.v[k], o1.v[k]), (p0[k], p1[k])):
            assert torch.allclose(a, b.cpu(), rtol=2e-6, atol=1e-7), k


@pytest.mark.parametrize("what", ["adamw", "clip"])
def test_one_long_tensor_is_as_fast_as_many_short_ones(what):
    """The same 32 M values as one tensor and as 32.  (With as many blocks for each tensor of a launch, whatever its length, one took
    4.5 and 3.5 times as long.)"""
    sides = []
    for parts in (1, 32):
        p = {str(i): torch.zeros((1 << 25) // parts, device=DEV) for i in range(parts)}
        g = {k: torch.ones_like(v) for k, v in p.items()}
        opt = optim.AdamW(p)
        sides.append(((lambda o=opt, g=g: o.step(g)) if what == "adamw" else (lambda g=g: optim.clip_grad_norm(g, 1e9)), []))
    for i in range(20):
        for fn, times in sides:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
    one, many = (statistics.median(t[3:]) for _, t in sides)
    assert one < 1.5 * many + 0.05, (one, many)
