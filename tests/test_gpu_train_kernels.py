"""Training kernels on a B200 against the torch ops they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("b,t,nk,nv,taps", [(1, 1, 1, 2, 4), (2, 31, 1, 2, 4), (1, 32, 2, 2, 3), (2, 33, 2, 4, 4), (1, 200, 2, 6, 1), (3, 129, 4, 8, 4), (2, 45, 1, 4, 6)])
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


def _both(fn, *shapes, seed=0, scale=1.0):
    """The op and the gradients of its inputs by the torch form on the CPU and by the kernels: ``fn(tape, *inputs)``.  fp32 sums in
    another order."""
    from tilerl_b200 import tape as T
    from tilerl_b200.ops import native
    g = torch.Generator().manual_seed(seed)
    xs = [torch.randn(*s, generator=g) * scale for s in shapes]
    outs = []
    for dev in ("cpu", DEV):
        ins = [x.to(dev) for x in xs]
        tape = T.Tape()
        tape.watch(*ins)
        before = native.launch_count
        y = fn(tape, *ins)
        up = torch.randn(y.shape, generator=torch.Generator().manual_seed(1)).to(dev)
        gs = tape.backward(y, up)
        assert (native.launch_count > before) == (dev == DEV)
        outs.append([y] + [gs[id(x)] for x in ins if id(x) in gs])
    assert len(outs[0]) == len(outs[1])
    for want, got in zip(*outs):
        assert got.shape == want.shape and _rel(got.cpu(), want) < 2e-5, want.shape


@pytest.mark.parametrize("rows,h", [((1,), 4), ((3, 5), 1020), ((2, 7), 1028), ((9,), 8192)])
def test_rmsnorm_and_swiglu(rows, h):
    from tilerl_b200 import tape as T
    _both(lambda t, x, w: T.rmsnorm(t, x, w, 1e-6), (*rows, h), (h,), seed=h)
    _both(lambda t, x: T.swiglu(t, x), (*rows, 2 * h), seed=h)


@pytest.mark.parametrize("m,k,n,r", [((1,), 4, 4, 4), ((2, 17), 132, 260, 8), ((3, 100), 1024, 516, 16), ((1000,), 260, 4128, 32)])
def test_adapters(m, k, n, r):
    """Ranks of every form, rows and widths that fill no block, gradients summed over parts of the rows."""
    from tilerl_b200 import tape as T
    _both(lambda t, y, x, a, b: T.lora(t, y, x, a, b, 0.7), (*m, n), (*m, k), (r, k), (n, r), seed=n)


@pytest.mark.parametrize("m,k,n,r", [((3, 11), 64, 132, 16), ((700,), 1024, 516, 8)])
@pytest.mark.parametrize("quantised", [True, False])
def test_frozen_linear_with_adapter(m, k, n, r, quantised):
    """One op against the two it stands for, on the same device: the dense products are the same calls, sums around them in another
    order."""
    from tilerl_b200 import formats as F
    from tilerl_b200 import tape as T
    from tilerl_b200.ops.cuda import CudaOps
    CudaOps(DEV)                                      # installs the weights' decoder
    g = torch.Generator().manual_seed(n)
    w = torch.randn(n, k, generator=g) * 0.05
    w = F.quantize_nvfp4(w).to(DEV) if quantised else w.to(DEV)
    x, a, b, up = (torch.randn(*s, generator=g).to(DEV) for s in ((*m, k), (r, k), (n, r), (*m, n)))
    res = []
    for one in (True, False):
        tape = T.Tape()
        tape.watch(x, a, b)
        y = T.linear_lora(tape, x, w, True, a, b, 0.5) if one else T.lora(tape, T.linear(tape, x, w, frozen=True), x, a, b, 0.5)
        assert len(tape.nodes) == (1 if one else 2)
        gs = tape.backward(y, up)
        res.append([y] + [gs[id(t)] for t in (x, a, b)])
    for got, want in zip(*res):
        assert _rel(got, want) < 1e-6


@pytest.mark.parametrize("b,t,n_q,n_kv,d,rot,gated", [(1, 1, 1, 1, 4, 2, True), (2, 33, 4, 2, 64, 32, True), (1, 300, 6, 1, 256, 64, True), (2, 40, 2, 2, 512, 512, False)])
def test_attention_block(b, t, n_q, n_kv, d, rot, gated):
    """Positions as they come, shared and one row a sequence out of order; heads narrower than a warp and the widest."""
    from tilerl_b200 import tape as T
    g = torch.Generator().manual_seed(t)
    qw, kw = 1 + 0.1 * torch.randn(d, generator=g), 1 + 0.1 * torch.randn(d, generator=g)
    for pos in (torch.arange(t) + 3, torch.stack([torch.randperm(t, generator=g) for _ in range(b)])):
        def fn(tape, qkv):
            dev = qkv.device
            return T.attention_block(tape, qkv, qw.to(dev), kw.to(dev), pos.to(dev), n_q=n_q, n_kv=n_kv, head_dim=d, rotary_dim=rot, theta=1e4, eps=1e-6, gated=gated)
        _both(fn, (b, t, n_q * d * (2 if gated else 1) + 2 * n_kv * d), seed=t)


@pytest.mark.parametrize("rows,v", [((1,), 4), ((2, 3), 2048), ((5,), 32764)])
def test_cross_entropy(rows, v):
    from tilerl_b200 import tape as T
    from tilerl_b200.ops import train_kernels as K
    g = torch.Generator().manual_seed(v)
    tg, w = torch.randint(0, v, rows, generator=g), torch.rand(rows, generator=g)
    x, sides = torch.randn(*rows, v, generator=g) * 8, []
    for dev in ("cpu", DEV):
        lg, tape = x.to(dev), T.Tape()
        tape.watch(lg)
        loss = T.cross_entropy(tape, lg, tg.to(dev), w.to(dev))
        sides.append((loss.cpu(), tape.backward(loss, torch.tensor(2.0, device=dev))[id(lg)].cpu()))
    assert torch.allclose(sides[0][0], sides[1][0], rtol=1e-6)
    # probabilities up to 1 of a few roundings each, less 1 at the target, times the weight and 2
    assert float((sides[0][1] - sides[1][1]).abs().max()) < 8 * 2 ** -24 * 2
    x = torch.randn(6, 64, generator=g)
    x[0, 3], x[1, 5], x[2] = float("inf"), float("nan"), float("-inf")
    x[3, 1:], x[4, 0] = float("-inf"), torch.finfo(torch.float32).min
    assert torch.allclose(K.lse(x.to(DEV))[2].cpu(), torch.logsumexp(x, -1), rtol=1e-6, atol=1e-6, equal_nan=True)


def test_adamw_and_clipping_of_many_tensors():
    """More tensors than a launch takes, one without elements on a 16-byte boundary and one in bf16 among them: three steps against
    the torch form, state and all."""
    from tilerl_b200.optim import AdamW, clip_grad_norm
    g = torch.Generator().manual_seed(3)
    shapes = {f"p{i}": (i % 7 + 1, 4 * i + 1) if i % 3 else (2 * i + 1,) for i in range(40)}
    ps = {k: torch.randn(s, generator=g) for k, s in shapes.items()}
    ps["half"] = torch.randn(8, 8, generator=g).to(torch.bfloat16)
    sides = []
    for dev in ("cpu", DEV):
        p = {k: v.clone().to(dev) for k, v in ps.items()}
        if dev == DEV:
            p["p5"] = torch.zeros(p["p5"].numel() + 1, device=dev)[1:].view(p["p5"].shape).copy_(p["p5"])
        opt = AdamW(p, lr=1e-2, weight_decay=0.1)
        for step in range(3):
            gs = {k: (torch.randn(v.shape, generator=torch.Generator().manual_seed(step * 100 + i)) * 3).to(dev) for i, (k, v) in enumerate(p.items())}
            version = p["p1"]._version
            norm = clip_grad_norm(gs, 1.0)
            opt.step(gs)
            assert p["p1"]._version > version
        sides.append((norm, gs, p, opt))
    (n0, g0, p0, o0), (n1, g1, p1, o1) = sides
    assert abs(n0 - n1) < 1e-6 * n0 and o0.t == o1.t
    for k in p0:
        for a, b in ((g0[k], g1[k]), (o0.m[k], o1.m[k]), (o0.v[k], o1.v[k])):
            assert torch.allclose(a.float(), b.float().cpu(), rtol=2e-6, atol=1e-9), k
        assert torch.allclose(p0[k].float(), p1[k].float().cpu(), rtol=2 ** -8 if k == "half" else 2e-6, atol=1e-7), k


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs in one process")
def test_delta_rule_block_on_a_second_gpu_of_the_process():
    """Its kernels' shared-memory limits are raised on the device that they run on, not once for the process."""
    from tilerl_b200 import tape as T
    g = torch.Generator().manual_seed(1)
    args = [torch.randn(1, 40, 768 + 4, generator=g), torch.randn(512, 4, generator=g) * 0.4, torch.randn(2, generator=g), torch.randn(2, generator=g), torch.ones(128)]
    outs = []
    for dev in ("cuda:0", "cuda:1"):
        here = [a.to(dev) for a in args]
        tape = T.Tape()
        tape.watch(*here)
        y = T.gdn_block(tape, *here, nk=1, nv=2, dk=128, dv=128, eps=1e-6)
        outs.append([y.cpu()] + [tape.backward(y, torch.ones_like(y))[id(a)].cpu() for a in here[:1]])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
