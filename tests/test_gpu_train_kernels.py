"""Training kernels on a B200 against the torch ops they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("b,t,nk,nv,taps", [(1, 1, 1, 2, 4), (2, 31, 1, 2, 4), (1, 32, 2, 2, 3), (2, 33, 2, 4, 4), (1, 200, 2, 6, 1), (3, 129, 4, 8, 4)])
def test_delta_rule_block_and_gradients(b, t, nk, nv, taps):
    """Lengths at, below and above a chunk of 32 and one token, several heads a key, convolutions down to one tap: output and every
    gradient against autograd through the chunked torch form.  Both are fp32 sums in another order; a gradient goes through up to
    200 steps of the recurrence: 1e-4."""
    from tilerl_b200 import tape as T
    from tilerl_b200.ops import gdn_train, native
    g = torch.Generator().manual_seed(t * 7 + nv)
    ch = (2 * nk + nv) * 128
    inp = torch.randn(b, t, ch + nv * 128 + 2 * nv, generator=g).to(DEV)
    params = [(torch.randn(ch, taps, generator=g) * 0.4).to(DEV), torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).mul(0.3).to(DEV),
              (1 + 0.1 * torch.randn(128, generator=g)).to(DEV)]
    up = torch.randn(b, t, nv * 128, generator=g).to(DEV)
    kw = dict(nk=nk, nv=nv, dk=128, dv=128, eps=1e-6)
    leaves = [x.clone().requires_grad_(True) for x in [inp] + params]
    want = T.gdn_block_torch(*leaves, **kw)
    grads = torch.autograd.grad(want, leaves, up)
    tape = T.Tape()
    tape.watch(inp, *params)
    before = native.launch_count
    got = T.gdn_block(tape, inp, *params, **kw)
    assert native.launch_count > before and gdn_train.takes(inp, *params, **kw)
    assert _rel(got, want) < 1e-5
    out = tape.backward(got, up)
    for x, w in zip([inp] + params, grads):
        assert out[id(x)].shape == x.shape and _rel(out[id(x)], w) < 1e-4, x.shape
    odd = inp.new_zeros(b, t, inp.shape[2] + 1)[..., 1:].copy_(inp)         # off a 16-byte boundary, strided
    assert torch.equal(T.gdn_block(T.Tape(), odd, *params, **kw), got)


def test_delta_rule_block_that_the_kernels_do_not_take():
    """An odd number of value heads and heads of 64 go through the torch form, as before."""
    from tilerl_b200 import tape as T
    for nk, nv, d in ((1, 1, 128), (1, 3, 128), (2, 2, 64)):
        g = torch.Generator().manual_seed(nv)
        ch = (2 * nk + nv) * d
        args = [torch.randn(1, 40, ch + nv * d + 2 * nv, generator=g).to(DEV), torch.randn(ch, 4, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV),
                torch.zeros(nv, device=DEV), torch.ones(d, device=DEV)]
        kw = dict(nk=nk, nv=nv, dk=d, dv=d, eps=1e-6)
        tape = T.Tape()
        tape.watch(args[0])
        y = T.gdn_block(tape, *args, **kw)
        assert torch.equal(y, T.gdn_block_torch(*args, **kw))
        assert tape.backward(y, torch.ones_like(y))[id(args[0])].shape == args[0].shape
