"""Gated delta rule block of the training tape on the kernels of ``csrc/gdn_train.cu``: fp32, heads of 128, whole sequences from an
empty state.  Parity: the same block as :func:`tilerl_b200.tape.gdn_block_torch`, which serves every other shape."""
from __future__ import annotations

import ctypes

import torch

from . import native as N

N.register("trl_gdn_train_workspace", [N.I] * 5)
N.register("trl_gdn_train_forward", [N.P] * 7 + [N.I] * 5 + [N.F, N.P])
N.register("trl_gdn_train_backward", [N.P] * 9 + [N.I] * 5 + [N.F, N.P])


def takes(inp, conv_w, dt_bias, a_log, norm_w, *, nk, nv, dk, dv, eps, chunk=64, state=None, cp=None) -> bool:
    if cp is not None or state is not None or dk != 128 or dv != 128 or nv % nk or nv % 2 or inp.dim() != 3 or inp.numel() == 0:
        return False
    # a sequence is a whole chunk of 32 tokens at least: 512 of one token with eight heads 4522 us with the gradient, 3634 as torch ops; of eight
    # tokens 4609 and 5520
    if inp.shape[1] < 8 and inp.shape[0] * nv > 2048:
        return False
    if not N.has("trl_gdn_train_forward"):           # (a library of one architecture)
        return False
    rows = 2 * nk * dk + 2 * nv * dv + 2 * nv
    return (inp.shape[2] == rows and inp.numel() < 1 << 29 and conv_w.dim() == 2 and conv_w.shape[0] == (2 * nk + nv) * dk
            and dt_bias.shape == a_log.shape == (nv,) and norm_w.shape == (dv,)
            and all(p.device == inp.device for p in (conv_w, dt_bias, a_log, norm_w)))


def grad_takes(g, out) -> bool:
    """A gradient of ``out``'s shape, on its device: what broadcasts to it (which autograd refuses) has fewer values than the kernels read."""
    return g.shape == out.shape and g.device == out.device


def _ready(*tensors):
    """fp32, contiguous and on a 16-byte boundary, as the kernels read them."""
    out = []
    for t in tensors:
        t = t.float().contiguous()
        out.append(t if t.data_ptr() % 16 == 0 else t.clone())
    return out


def _workspace(inp, nk: int, nv: int, grad: bool) -> torch.Tensor:
    f = N.lib().trl_gdn_train_workspace
    f.restype = ctypes.c_long
    return torch.empty(f(inp.shape[0], inp.shape[1], nk, nv, int(grad)), dtype=torch.float32, device=inp.device)


def forward(inp, conv_w, dt_bias, a_log, norm_w, *, nk, nv, dk, dv, eps, **_) -> torch.Tensor:
    x, cw, db, al, nw = _ready(inp, conv_w, dt_bias, a_log, norm_w)
    b, t, _ = x.shape
    with torch.cuda.device(x.device):
        out = torch.empty(b, t, nv * dv, dtype=torch.float32, device=x.device)
        ws = _workspace(x, nk, nv, False)
        N.check(N.lib().trl_gdn_train_forward(x.data_ptr(), cw.data_ptr(), db.data_ptr(), al.data_ptr(), nw.data_ptr(), out.data_ptr(),
                                              ws.data_ptr(), b, t, nk, nv, cw.shape[1], eps, N.stream()), "gdn_train_forward")
    N.count(4)
    return out


@torch.no_grad()
def backward(inp, conv_w, dt_bias, a_log, norm_w, grad, need, *, nk, nv, dk, dv, eps, **_):
    """Gradients of ``(inp, conv_w, dt_bias, a_log, norm_w)``; ``need``: which of the four parameters' are wanted."""
    x, cw, db, al, nw, g = _ready(inp, conv_w, dt_bias, a_log, norm_w, grad)
    b, t, _ = x.shape
    kw, ch = cw.shape[1], (2 * nk + nv) * dk
    where = (ctypes.c_long * 3)()
    with torch.cuda.device(x.device):
        dx = torch.empty_like(x)
        ws = _workspace(x, nk, nv, True)
        N.check(N.lib().trl_gdn_train_backward(x.data_ptr(), cw.data_ptr(), db.data_ptr(), al.data_ptr(), nw.data_ptr(), g.data_ptr(),
                                               dx.data_ptr(), ws.data_ptr(), where, b, t, nk, nv, kw, eps, N.stream()), "gdn_train_backward")
    N.count(8)
    tp = -(-t // 32) * 32
    d_conv = d_bias = d_log = d_norm = None
    if need[0]:
        dy = ws[where[2]:where[2] + b * t * ch].view(b, t, ch)
        xp = torch.nn.functional.pad(x[..., :ch], (0, 0, kw - 1, 0))
        d_conv = torch.stack([(dy * xp[:, j:j + t]).sum((0, 1)) for j in range(kw)], -1).view(conv_w.shape)
    if need[1]:
        d_bias = dx[..., ch + nv * dv:ch + nv * dv + nv].sum((0, 1)).view(dt_bias.shape)
    if need[2]:
        dg = ws[where[1]:where[1] + b * nv * tp].view(b, nv, tp)[:, :, :t].transpose(1, 2)
        decay = -torch.exp(al.view(-1)) * torch.nn.functional.softplus(x[..., ch + nv * dv:ch + nv * dv + nv] + db.view(-1))
        d_log = (dg * decay).sum((0, 1)).view(a_log.shape)
    if need[3]:
        o = ws[where[0]:where[0] + b * nv * tp * dv].view(b, nv, tp, dv)[:, :, :t].transpose(1, 2)
        z = x[..., ch:ch + nv * dv].view(b, t, nv, dv)
        d_norm = (g.view(b, t, nv, dv) * torch.nn.functional.silu(z) * o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + eps)).sum((0, 1, 2)).view(norm_w.shape)
    return dx, d_conv, d_bias, d_log, d_norm
