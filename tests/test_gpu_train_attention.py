"""The training attention block's softmax kernels at the widths of rows that each serves, on a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("t", [512, 513, 2048, 2049, 4096])
def test_softmax_of_long_rows_and_its_gradient(t):
    """Rows at and beside the lengths where a thread keeps more values (512, 2048) and the longest: positions in and out of order,
    against 64 bits.  A weight is an exponential of a score of up to 30, so a unit of fp32 in the score is 2e-6 of it; the sums over up to
    4096 terms add a few of 6e-8."""
    from tilerl_b200.ops import native
    from tilerl_b200.ops import train_kernels as K
    g = torch.Generator().manual_seed(t)
    b, heads, scale = 2, 3, 0.125
    for pos in (torch.arange(t)[None], torch.stack([torch.randperm(t, generator=g) for _ in range(b)])):
        pos = pos.to(DEV)
        s = (torch.randn(b, heads, t, t, generator=g) * 8 / scale / 4).to(DEV)
        want = (s.double() * scale).masked_fill(~(pos[:, None, None, :] <= pos[:, None, :, None]), float("-inf")).softmax(-1)
        p = s.clone()
        native.check(native.lib().trl_train_softmax(p.data_ptr(), pos.data_ptr(), pos.shape[0], b, heads, t, scale, native.stream()), "softmax")
        assert float((p.double() - want).norm() / want.norm()) < 5e-6
        assert bool((p[want == 0] == 0).all())
        dp = torch.randn(b, heads, t, t, generator=g).to(DEV)
        dwant = want * (dp.double() - (want * dp.double()).sum(-1, keepdim=True)) * scale
        native.check(native.lib().trl_train_softmax_grad(p.data_ptr(), dp.data_ptr(), b * heads * t, t, scale, native.stream()), "softmax_grad")
        assert float((dp.double() - dwant).norm() / dwant.norm()) < 1e-5
    assert K.there()


def test_attention_block_of_long_sequences():
    """The block at 700 and 2100 tokens against its torch form on the same device: the same products, fp32 sums in another order."""
    from tilerl_b200 import tape as T
    for t in (700, 2100):
        g = torch.Generator().manual_seed(t)
        dims = dict(n_q=4, n_kv=2, head_dim=64, rotary_dim=32, theta=1e4, eps=1e-6, gated=True)
        qkv = torch.randn(1, t, 4 * 64 * 2 + 2 * 2 * 64, generator=g).to(DEV)
        qw, kw = ((1 + 0.1 * torch.randn(64, generator=g)).to(DEV) for _ in range(2))
        pos, up = torch.arange(t, device=DEV), torch.randn(1, t, 256, generator=g).to(DEV)
        want, bwd = T._attention_torch(qkv, qw, kw, pos, **dims)
        tape = T.Tape()
        tape.watch(qkv)
        got = T.attention_block(tape, qkv, qw, kw, pos, **dims)
        assert float((got - want).norm() / want.norm()) < 2e-5
        d, dwant = tape.backward(got, up)[id(qkv)], bwd(up)[0]
        assert float((d - dwant).norm() / dwant.norm()) < 2e-5
