"""What the tape hands to the training kernels, on the CPU: stand-ins that read as many values as the kernels do take their place."""
import types

import pytest
import torch

from tilerl_b200 import tape as T
from tilerl_b200.ops import gdn_train, ref, train_kernels


def _grad_of(fn, g, *xs):
    with torch.enable_grad():
        leaves = [x.clone().requires_grad_(True) for x in xs]
        y = fn(*leaves)
        return torch.autograd.grad(y, leaves, g)


@pytest.fixture
def kernels(monkeypatch):
    """A namespace in the place of ``ops.train_kernels``: its checks, and its functions in torch on flat memory of the sizes that the
    kernels go through.  ``calls`` counts what went to them."""
    calls = []

    def flat(t, n):
        calls.append(n)
        assert t.numel() >= n, "read past the end"
        return t.reshape(-1)[:n]

    def rmsnorm(x, w, eps, kept=None):
        if kept is not None:
            kept.copy_(x)
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w

    def swiglu(gu):
        return torch.nn.functional.silu(gu[..., 0::2]) * gu[..., 1::2]

    def lora(y, x, a, b, s):
        xa = x.reshape(-1, x.shape[-1]) @ a.t()
        return y.float() + (xa @ b.t()).view(y.shape) * s, xa

    def lora_grad(x, xa, a, b, s, g, dx16=None):
        m, n = xa.shape[0], b.shape[0]
        g2 = flat(g, m * n).view(m, n)
        dxa = g2 @ b * s
        dx = (dxa @ a).view(x.shape)
        return dx if dx16 is None else dx + dx16.float(), dxa.t() @ x.reshape(m, -1), g2.t() @ xa * s

    def attention(qkv, qw, kw, pos, **k):
        out, bwd = T._attention_torch(qkv, qw, kw, pos.to(torch.int64), **k)
        return out, lambda g: bwd(flat(g, out.numel()).view(out.shape))[0]

    def lse(lg):
        return torch.stack([lg.amax(-1), torch.exp(lg - lg.amax(-1, keepdim=True)).sum(-1), torch.logsumexp(lg, -1)])

    def cross_entropy_grad(lg, stats, tg, w):
        return ref.cross_entropy_grad(lg, tg, w)[1]

    K = types.SimpleNamespace(
        calls=calls, grad_takes=train_kernels.grad_takes, _grad=train_kernels._grad,
        rmsnorm_takes=lambda x, w: True, rmsnorm=rmsnorm,
        rmsnorm_grad=lambda x, w, g, eps: T._rmsnorm_torch(x, w, eps)[1](flat(g, x.numel()).view(x.shape))[0],
        swiglu_takes=lambda gu: True, swiglu=swiglu,
        swiglu_grad=lambda gu, g: _grad_of(swiglu, flat(g, gu.numel() // 2).view(*gu.shape[:-1], -1), gu)[0],
        lora_takes=lambda y, x, a, b: True, lora=lora, lora_grad=lora_grad,
        attention_takes=lambda *a, **k: True, attention=attention,
        cross_entropy_takes=lambda lg, tg, w: True, lse=lse,
        cross_entropy_grad=cross_entropy_grad, scale_by=lambda t, up: t.mul_(flat(up, 1)))
    monkeypatch.setattr(T, "_kernels", lambda x: K)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: None)        # (a CPU tensor's device has no index)
    return K


def _ops():
    g = torch.Generator().manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=g)
    pos = torch.arange(5)
    return {
        "rmsnorm": (lambda t, x, w: T.rmsnorm(t, x, w, 1e-6), [r(3, 8), r(8)]),
        "swiglu": (lambda t, x: T.swiglu(t, x), [r(3, 8)]),
        "lora": (lambda t, y, x, a, b: T.lora(t, y, x, a, b, 0.5), [r(3, 6), r(3, 8), r(4, 8), r(6, 4)]),
        "attention": (lambda t, x: T.attention_block(t, x, torch.ones(4), torch.ones(4), pos, n_q=2, n_kv=1, head_dim=4, rotary_dim=4, theta=1e4, eps=1e-6), [r(1, 5, 24)]),
    }


@pytest.mark.parametrize("op", ["rmsnorm", "swiglu", "lora"])
def test_gradient_that_broadcasts_is_not_read_past_its_end(op, kernels):
    """A root gradient of one row: no kernel gets it, and what comes back is what the torch form gives (the adapters' refuses it)."""
    fn, xs = _ops()[op]
    with torch.no_grad():
        tape = T.Tape()
        tape.watch(*xs)
        y = fn(tape, *xs)
        one = torch.randn(1, y.shape[-1], generator=torch.Generator().manual_seed(1))
        if op == "lora":
            with pytest.raises(RuntimeError):
                tape.backward(y, one)
            assert not kernels.calls
            return
        got = tape.backward(y, one)
        assert not kernels.calls
        whole = T.Tape()
        whole.watch(*xs)
        want = whole.backward(fn(whole, *xs), one.expand(y.shape).contiguous())
        assert kernels.calls
    for x in xs:
        assert got[id(x)].shape in (x.shape, one.shape)
        if got[id(x)].shape == x.shape:
            assert torch.allclose(got[id(x)], want[id(x)], rtol=1e-5, atol=1e-6)


def test_gradient_seen_in_another_shape(kernels):
    """The attention block's torch form takes a gradient of as many values in another shape."""
    fn, (x,) = _ops()["attention"]
    tape = T.Tape()
    tape.watch(x)
    y = fn(tape, x)
    up = torch.randn(y.shape, generator=torch.Generator().manual_seed(1))
    got = tape.backward(y, up.view(5, 8))[id(x)]
    assert not kernels.calls
    tape.watch(x)
    assert torch.allclose(got, tape.backward(fn(tape, x), up)[id(x)], rtol=1e-5, atol=1e-6)


def test_loss_gradient_of_another_shape(kernels):
    x, tg, w = torch.randn(4, 8, generator=torch.Generator().manual_seed(2)), torch.tensor([1, 7, 0, 3]), torch.rand(4)
    tape = T.Tape()
    tape.watch(x)
    rows = torch.tensor([[1.0], [2.0], [0.0], [4.0]])                    # one number a row: broadcasts over the gradient
    got = tape.backward(T.cross_entropy(tape, x, tg, w), rows)[id(x)]
    assert not kernels.calls and torch.allclose(got, ref.cross_entropy_grad(x, tg, w)[1] * rows)


def test_gradients_that_the_kernels_read():
    """Of the output's shape and device only; a number on the CPU for a loss elsewhere is not one."""
    out = torch.empty(2, 3, device="meta")
    for takes in (train_kernels.grad_takes, gdn_train.grad_takes):
        assert not takes(torch.empty(1, 3, device="meta"), out) and not takes(torch.empty(2, 3), out)
        assert not takes(torch.ones(()), torch.empty((), device="meta"))
    assert gdn_train.grad_takes(torch.empty(2, 3, device="meta"), out)


def test_positions_and_vectors_that_the_kernels_take(monkeypatch):
    """Fractional positions are rotated by their fraction (a cast to whole ones would drop it); vectors and taps of another rank
    mean something else to the torch form, or are refused there."""
    monkeypatch.setattr(train_kernels, "plain", lambda *t: True)
    qkv, w = torch.randn(1, 3, 24), torch.ones(4)
    dims = dict(n_q=2, n_kv=1, head_dim=4, rotary_dim=4, gated=True)
    pos = torch.arange(3)
    assert train_kernels.attention_takes(qkv, w, w, pos, **dims) and train_kernels.attention_takes(qkv, w, w, pos.int()[None], **dims)
    assert not train_kernels.attention_takes(qkv, w, w, pos * 0.5, **dims)
    nk, nv = 1, 2
    inp, conv, v, nw = torch.zeros(1, 3, (2 * nk + 2 * nv) * 128 + 2 * nv), torch.zeros((2 * nk + nv) * 128, 4), torch.zeros(nv), torch.ones(128)
    kw = dict(nk=nk, nv=nv, dk=128, dv=128, eps=1e-6)
    assert gdn_train.takes(inp, conv, v, v, nw, **kw)
    assert not gdn_train.takes(inp, conv[:, None], v, v, nw, **kw) and not gdn_train.takes(inp, conv, v[:, None], v, nw, **kw)
    assert not gdn_train.takes(inp, conv, v, v[None], nw, **kw) and not gdn_train.takes(inp, conv, v, v, nw[None], **kw)


@pytest.mark.parametrize("late", [False, True])
def test_weights_that_an_op_made_or_that_are_watched_later_get_their_gradient(late, kernels):
    """A norm's weight that comes out of another op on the tape passes its gradient on; a tensor may be watched after the ops that read it."""
    g = torch.Generator().manual_seed(3)
    x, qkv, base = torch.randn(3, 4, generator=g), torch.randn(1, 5, 24, generator=g), 1 + 0.1 * torch.randn(4, generator=g)
    dims = dict(n_q=2, n_kv=1, head_dim=4, rotary_dim=4, theta=1e4, eps=1e-6)
    for fn in (lambda t, w: T.rmsnorm(t, x, w, 1e-6), lambda t, w: T.attention_block(t, qkv, w, w, torch.arange(5), **dims)):
        res = []
        for K in (kernels, None):
            T._kernels = lambda x: K               # (the fixture puts the module's own back)
            tape = T.Tape()
            if not late:
                tape.watch(base)
            y = fn(tape, base if late else T.scale(tape, base, 2.0))
            tape.watch(base)
            res.append(tape.backward(y, torch.ones_like(y))[id(base)])
        assert torch.allclose(*res, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("late", [False, True])
def test_delta_rule_parameters_that_an_op_made_get_their_gradient(late, monkeypatch):
    asked = []
    monkeypatch.setattr(gdn_train, "takes", lambda *a, **k: True)
    monkeypatch.setattr(gdn_train, "forward", lambda inp, *a, **k: inp * 1.0)
    monkeypatch.setattr(gdn_train, "backward", lambda inp, *p, need, **k: asked.append(need) or (inp,) + tuple(q if n else None for q, n in zip(p, need)))
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)
    params = [torch.ones(2) for _ in range(4)]
    tape = T.Tape()
    if not late:
        tape.watch(params[0])
    used = params if late else [T.scale(tape, params[0], 2.0)] + params[1:]
    y = T.gdn_block(tape, torch.ones(2), *used, nk=1, nv=2, dk=128, dv=128, eps=1e-6)
    tape.watch(params[0])
    assert id(params[0]) in tape.backward(y, torch.ones_like(y)) and asked == [[True, False, False, False]]


def test_tensors_changed_between_the_passes(kernels):
    """Logits, targets, weights and a norm's rows may be written into after the forward pass: the gradient is that of the values
    that it saw.  An attention block's rows may not: both forms read some of them again."""
    g = torch.Generator().manual_seed(4)
    x, tg, w = torch.randn(4, 8, generator=g), torch.tensor([1, 7, 0, 3]), torch.rand(4, generator=g)
    want = ref.cross_entropy_grad(x, tg, w)[1]
    up = torch.randn(4, 8, generator=g)
    want_norm = T._rmsnorm_torch(x, torch.ones(8), 1e-6)[1](up)[0]
    for inference in (False, True):                  # (whose tensors keep no count of the writes)
        with torch.inference_mode(inference):
            lg, t, v = x * 1.0, tg * 1, w * 1.0
            tape = T.Tape()
            tape.watch(lg)
            loss = T.cross_entropy(tape, lg, t, v)
            lg.zero_(), t.zero_(), v.zero_()
            assert torch.allclose(tape.backward(loss)[id(lg)], want)
            rows = x * 1.0
            tape.watch(rows)
            y = T.rmsnorm(tape, rows, torch.ones(8), 1e-6)
            rows.zero_()
            assert torch.allclose(tape.backward(y, up * 1.0)[id(rows)], want_norm, rtol=1e-5, atol=1e-6)
    tape, qkv = T.Tape(), torch.randn(1, 5, 24, generator=g)
    tape.watch(qkv)
    y = _ops()["attention"][0](tape, qkv)
    qkv.mul_(2.0)
    with pytest.raises(RuntimeError, match="in place"):
        tape.backward(y)


def test_training_without_the_kernels(monkeypatch, tmp_path):
    """A library without these entry points (one that serves a single architecture), or none at all: the ops, clipping and the
    optimizer run in torch."""
    from tilerl_b200.ops import native
    from tilerl_b200.optim import AdamW, clip_grad_norm
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)

    class Device(str):                                # a "cuda" whose tensors live on the CPU
        type = "cuda"
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(3, 8, generator=g), torch.ones(8)
    params = [torch.zeros(4 * 128, 2), torch.zeros(2), torch.zeros(2), torch.ones(128)]
    inp = torch.randn(1, 3, 6 * 128 + 4, generator=g)
    for lib, path in ((object(), __file__), (None, str(tmp_path / "none.so"))):
        monkeypatch.setattr(native, "_LIB", lib), monkeypatch.setattr(native, "_PATH", path)
        assert not native.has("trl_train_adamw")
        tape = T.Tape()
        tape.watch(x)
        assert tape.backward(T.rmsnorm(tape, x, w, 1e-6), torch.ones(3, 8))[id(x)].shape == (3, 8)
        assert not gdn_train.takes(inp, *params, nk=1, nv=2, dk=128, dv=128, eps=1e-6)
        p, grads = {"w": torch.ones(4)}, {"w": torch.ones(4)}
        opt = AdamW(p, lr=0.1)
        opt.step(grads)
        assert float(p["w"][0]) < 1 and opt.t == {"w": 1}
        monkeypatch.setattr(torch.Tensor, "device", Device("cpu"), raising=False)
        assert abs(clip_grad_norm(grads, 10.0) - 2.0) < 1e-6
        monkeypatch.undo()
        monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)
    monkeypatch.setattr(native, "_LIB", type("L", (), {"trl_x": 1})())
    assert native.has("trl_x") and not native.has("trl_y")


def test_tensors_that_share_memory_are_not_in_one_launch(monkeypatch):
    """A weight under two names is updated by one after the other, as the loop over the names does; a gradient given twice is scaled
    by one after the other.  Gradients that only are read may be shared."""
    launches = []

    class Lib:
        def trl_train_adamw(self, p, m, v, g, n, decay, c1, c2, count, *rest):
            launches.append([int(p[i]) for i in range(count)])
            return 0

        def trl_train_scale(self, p, n, count, c, stream):
            launches.append([int(p[i]) for i in range(count)])
            return 0
    monkeypatch.setattr(train_kernels.N, "lib", lambda: Lib())
    monkeypatch.setattr(train_kernels.N, "stream", lambda: 0)
    t = [torch.ones(8) for _ in range(12)]
    item = lambda p, m, v, g: (p, m, v, g, 1.0, 0.1, 0.1)
    run = lambda *items: (launches.clear(), train_kernels.adamw(list(items), 0.1, (0.9, 0.99), 1e-8), [list(x) for x in launches])[2]
    at = lambda x: x.data_ptr()
    assert run(item(*t[:4]), item(*t[4:8])) == [[at(t[0]), at(t[4])]]
    assert run(item(*t[:4]), item(t[4], t[5], t[6], t[3])) == [[at(t[0]), at(t[4])]]
    assert run(item(*t[:4]), item(t[0], t[5], t[6], t[7])) == [[at(t[0])], [at(t[0])]]
    assert run(item(*t[:4]), item(t[4], t[5], t[6], t[0])) == [[at(t[0])], [at(t[4])]]
    whole = torch.ones(16)
    assert run(item(whole[:8], *t[1:4]), item(whole[8:], *t[5:8])) == [[at(whole), at(whole[8:])]]
    assert len(run(item(whole[:8], *t[1:4]), item(whole[4:12], *t[5:8]))) == 2
    for tensors, want in (([t[0], t[1]], [[at(t[0]), at(t[1])]]), ([t[0], t[1], t[0]], [[at(t[0])], [at(t[1])], [at(t[0])]])):
        launches.clear()
        train_kernels.scale(tensors, 0.5)
        assert launches == want


def test_adapters_go_to_the_kernels_where_they_are_faster(monkeypatch):
    """Few wide rows, and rank 32 over many, stay with the library's products."""
    monkeypatch.setattr(train_kernels, "plain", lambda *t: True)
    e = lambda *s: torch.empty(*s, device="meta")
    takes = lambda m, k, n, r: train_kernels.lora_takes(None, e(m, k), e(r, k), e(n, r))
    for m, k, n, r, want in ((1, 1024, 3072, 16, True), (1, 6144, 5120, 32, True), (31, 5120, 34816, 8, False), (32, 5120, 34816, 8, True), (16, 17408, 5120, 16, False),
                             (2048, 1024, 6144, 32, True), (4096, 1024, 3072, 32, True), (8192, 1024, 3072, 32, False), (1024, 17408, 5120, 32, True),
                             (2048, 17408, 5120, 32, False), (256, 5120, 34816, 32, False), (16384, 17408, 5120, 16, True), (64, 1024, 3072, 12, False)):
        assert takes(m, k, n, r) == want, (m, k, n, r)
        y = e(m, n)
        assert train_kernels.lora_takes(y, e(m, k), e(r, k), e(n, r)) == want


def test_narrow_rows_and_short_sequences_in_numbers_stay_with_torch(monkeypatch):
    monkeypatch.setattr(train_kernels, "plain", lambda *t: True), monkeypatch.setattr(gdn_train.N, "has", lambda name: True)
    e = lambda *s: torch.empty(*s, device="meta")
    for rows, h, want in ((65536, 64, True), (65537, 64, False), (262144, 252, False), (262144, 256, True), (512, 64, True)):
        assert train_kernels.rmsnorm_takes(e(rows, h), e(h)) == want
    for rows, v, want in ((8192, 128, True), (262144, 128, False), (65536, 512, True)):
        assert train_kernels.cross_entropy_takes(e(rows, v), e(rows), e(rows)) == want
    for m, k, want in ((16384, 64, True), (262144, 64, False), (65536, 512, True), (65537, 512, False), (131072, 1024, True), (65536, 256, False)):
        assert train_kernels.lora_takes(None, e(m, k), e(16, k), e(k, 16)) == want
    for b, t, nv, want in ((512, 1, 8, False), (512, 8, 8, True), (1, 1, 2, True), (256, 1, 8, True)):
        ch = (2 + nv) * 128
        assert gdn_train.takes(e(b, t, ch + nv * 130), e(ch, 4), e(nv), e(nv), e(128), nk=1, nv=nv, dk=128, dv=128, eps=1e-6) == want


def test_tensors_that_autograd_or_inference_mode_keeps_are_refused_as_before(monkeypatch):
    """A followed leaf, and an inference tensor outside that mode, are not written into by a kernel: torch refuses them."""
    from tilerl_b200 import optim
    monkeypatch.setattr(train_kernels, "there", lambda: True), monkeypatch.setattr(train_kernels, "plain", lambda *t: True)
    monkeypatch.setattr(train_kernels, "adamw", lambda items, *a: [it[0].data.zero_() for it in items])
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)
    with torch.inference_mode():
        kept = torch.ones(4)
    for p in (torch.ones(4, requires_grad=True), kept):
        with pytest.raises(RuntimeError):
            optim.AdamW({"w": p}).step({"w": torch.ones(4)})
    p = torch.ones(4, requires_grad=True)
    with torch.no_grad():
        optim.AdamW({"w": p}).step({"w": torch.ones(4)})
    assert float(p.detach().sum()) == 0.0
    assert not train_kernels.writable(kept) and train_kernels.writable(torch.ones(4))
    with torch.inference_mode():
        assert train_kernels.writable(kept)
