"""The training tape's elementwise and low-rank ops on the kernels of ``csrc/train.cu``.  Each function says what it takes with a
``*_takes`` of its own or returns ``None``; the tape runs its torch form where it does not."""
from __future__ import annotations

import ctypes
from typing import Dict, List, Optional, Sequence

import torch

from . import native as N

N.register("trl_train_rmsnorm", [N.P] * 4 + [N.I] * 2 + [N.F, N.P])
N.register("trl_train_rmsnorm_grad", [N.P] * 4 + [N.I] * 2 + [N.F, N.P])
N.register("trl_train_swiglu", [N.P] * 3 + [N.L, N.P])
N.register("trl_train_lowrank", [N.P] * 3 + [N.I] * 4 + [N.F, N.P])
N.register("trl_train_expand", [N.P, N.I] + [N.P] * 3 + [N.I] * 4 + [N.F, N.P])
N.register("trl_train_outer_parts", [N.I] * 2)
N.register("trl_train_outer", [N.P] * 4 + [N.I] * 4 + [N.F, N.P])
N.register("trl_train_attn_prep", [N.P] * 8 + [N.I] * 8 + [N.F, N.P])
N.register("trl_train_attn_prep_grad", [N.P] * 11 + [N.I] * 8 + [N.F, N.P])
N.register("trl_train_attn_gate", [N.P] * 3 + [N.I] * 7 + [N.P])
N.register("trl_train_softmax", [N.P] * 2 + [N.I] * 4 + [N.F, N.P])
N.register("trl_train_softmax_grad", [N.P] * 2 + [N.L, N.I, N.F, N.P])
N.register("trl_train_lse", [N.P] * 2 + [N.L] * 2 + [N.P])
N.register("trl_train_ce_grad", [N.P] * 5 + [N.L] * 2 + [N.P])
N.register("trl_train_scale_by", [N.P] * 2 + [N.L, N.P])
N.register("trl_train_adamw", [N.P] * 8 + [N.I] + [N.F] * 6 + [N.P])
N.register("trl_train_squares_blocks", [N.L])
N.register("trl_train_squares", [N.P, N.P, N.I, N.I, N.P, N.P])
N.register("trl_train_scale", [N.P, N.P, N.I, N.F, N.P])

INTEGERS = (torch.int64, torch.int32, torch.int16, torch.int8, torch.uint8)       # (positions between two tokens: the torch form)
MAX_TENSORS = 32          # a launch of the many-tensor kernels


def there() -> bool:
    """The library has these kernels: one of a single architecture does not, and training runs in torch as it does without one."""
    return N.has("trl_train_adamw")


def plain(*tensors) -> bool:
    """fp32, contiguous, not empty and on 16-byte boundaries, all on the current CUDA device."""
    here = torch.cuda.current_device() if tensors and tensors[0].is_cuda else None
    return all(t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.numel() and t.data_ptr() % 16 == 0
               and t.device.index == here for t in tensors)


def writable(*tensors) -> bool:
    """Tensors that torch would write into without a word: autograd refuses leaves that it follows (and records the others), inference
    mode its tensors outside it.  Kernels ask neither."""
    followed, outside = torch.is_grad_enabled(), not torch.is_inference_mode_enabled()
    return not any(followed and t.requires_grad or outside and t.is_inference() for t in tensors)


def grad_takes(g: torch.Tensor, out: torch.Tensor) -> bool:
    """A gradient that the kernels can read as that of ``out``: the same shape (torch ops also take one that broadcasts, or a number
    on the CPU; a kernel would read past its end), on the same device, which still is the current one."""
    return g.shape == out.shape and g.device == out.device and g.device.index == torch.cuda.current_device()


def _grad(g: torch.Tensor) -> torch.Tensor:
    g = g.float().contiguous()
    return g if g.data_ptr() % 16 == 0 else g.clone()


# ---- RMSNorm ---------------------------------------------------------------------------------------------
def rmsnorm_takes(x, w) -> bool:
    """Not many narrow rows, of which a block each is mostly idle: 262 144 x 64 722 us with its gradient, 570 as torch ops; 65 536 x 256 218 and 501."""
    h = x.shape[-1]
    if h < 256 and x.numel() > 65536 * h:
        return False
    return h % 4 == 0 and h <= 8192 and w.dim() == 1 and w.numel() == h and plain(x, w) and x.numel() // h < 1 << 31


def rmsnorm(x, w, eps, kept=None):
    """``kept``: gets a copy of ``x`` for the gradient, since the caller may write into ``x`` between the passes."""
    out = torch.empty_like(x)
    h = x.shape[-1]
    N.check(N.lib().trl_train_rmsnorm(x.data_ptr(), w.data_ptr(), out.data_ptr(), N.ptr(kept), x.numel() // h, h, eps, N.stream()), "train_rmsnorm")
    N.count()
    return out


def rmsnorm_grad(x, w, g, eps):
    g, dx, h = _grad(g), torch.empty_like(x), x.shape[-1]
    N.check(N.lib().trl_train_rmsnorm_grad(x.data_ptr(), w.data_ptr(), g.data_ptr(), dx.data_ptr(), x.numel() // h, h, eps, N.stream()), "train_rmsnorm_grad")
    N.count()
    return dx


# ---- SwiGLU ------------------------------------------------------------------------------------------------
def swiglu_takes(gu) -> bool:
    return gu.shape[-1] % 2 == 0 and gu.numel() % 8 == 0 and gu.numel() < 1 << 40 and plain(gu)


def swiglu(gu):
    out = torch.empty(*gu.shape[:-1], gu.shape[-1] // 2, dtype=torch.float32, device=gu.device)
    N.check(N.lib().trl_train_swiglu(gu.data_ptr(), None, out.data_ptr(), out.numel(), N.stream()), "train_swiglu")
    N.count()
    return out


def swiglu_grad(gu, g):
    g, d = _grad(g), torch.empty_like(gu)
    N.check(N.lib().trl_train_swiglu(gu.data_ptr(), g.data_ptr(), d.data_ptr(), g.numel(), N.stream()), "train_swiglu_grad")
    N.count()
    return d


# ---- adapters: y + s (x A^T) B^T -----------------------------------------------------------------------------
def lora_takes(y, x, a, b) -> bool:
    """``y`` may be ``None`` (a dense product's bf16 result to come)."""
    (r, k), n = a.shape, b.shape[0]
    return (r in (4, 8, 16, 32) and k % 4 == 0 and n % 4 == 0 and b.shape[1] == r and x.shape[-1] == k and _lora_pays(x.numel() // k, k, n, r) and plain(x, a, b)
            and x.numel() // k <= 16 * 65535 and (y is None or (y.shape[-1] == n and x.shape[:-1] == y.shape[:-1] and plain(y))))


def _lora_pays(m: int, k: int, n: int, r: int) -> bool:
    """Sizes where the kernels beat the torch ops (whose products are the library's).  Forward and gradient over a frozen weight, torch and
    here, us.  Few wide rows leave most of the GPU idle, a block going through all of them: 5120 -> 34 816, 16 rows of rank 16 271, 381, 32 rows 375,
    377; 16 480 16 rows 213, 231, 32 rows 273, 234; 6144 -> 5120 from one row on 194, 133.  Rank 32 passes over the rows twice, and a good GEMM does
    not: 1024 -> 3072, 4096 rows 407, 388, 8192 rows 658, 725; 6144 -> 5120 2048 rows 660, 610, 8192 1958, 2158; 17 408 -> 5120 1024 rows 706, 652,
    2048 rows 1226, 1223, 8192 4246, 4582; 34 816 at no length.  Many narrow rows: 262 144 x 256 rank 16 1273, 2216, 65 536 x 512 827, 782, 131 072 x 1024 rank 8 2004, 1748."""
    if m > (65536 if min(k, n) >= 512 else 16384) and min(k, n) < 1024:
        return False
    if m < 32 and max(k, n) > 8192:
        return False
    return r < 32 or (m <= 4096 and k + n <= 32768 and m * (k + n) <= 2048 * 16384)


def lora(y, x, a, b, s):
    """The result, and ``x A^T`` for the gradient.  ``y``: fp32, or bf16 as a dense product leaves it."""
    (r, k), n, m = a.shape, b.shape[0], x.numel() // x.shape[-1]
    xa, out = torch.empty(m, r, dtype=torch.float32, device=x.device), torch.empty(y.shape, dtype=torch.float32, device=y.device)
    N.check(N.lib().trl_train_lowrank(x.data_ptr(), a.data_ptr(), xa.data_ptr(), m, k, r, 0, 1.0, N.stream()), "train_lowrank")
    N.check(N.lib().trl_train_expand(y.data_ptr(), int(y.dtype == torch.bfloat16), xa.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, r, 0, s, N.stream()), "train_expand")
    N.count(2)
    return out, xa


def lora_grad(x, xa, a, b, s, g, dx16=None):
    """Gradients of (x, a, b) for that of the result; ``dx16``: what is to be added to x's (bf16)."""
    (r, k), n, m = a.shape, b.shape[0], x.numel() // x.shape[-1]
    lib, st = N.lib(), N.stream()
    dxa, dx, da, db = torch.empty_like(xa), torch.empty_like(x), torch.empty_like(a), torch.empty_like(b)
    part = torch.empty(r * max(lib.trl_train_outer_parts(m, n) * n, lib.trl_train_outer_parts(m, k) * k), dtype=torch.float32, device=x.device)
    N.check(lib.trl_train_lowrank(g.data_ptr(), b.data_ptr(), dxa.data_ptr(), m, n, r, 1, s, st), "train_lowrank")
    N.check(lib.trl_train_outer(g.data_ptr(), xa.data_ptr(), part.data_ptr(), db.data_ptr(), m, n, r, 0, s, st), "train_outer")
    N.check(lib.trl_train_outer(x.data_ptr(), dxa.data_ptr(), part.data_ptr(), da.data_ptr(), m, k, r, 1, 1.0, st), "train_outer")
    N.check(lib.trl_train_expand(N.ptr(dx16), int(dx16 is not None), dxa.data_ptr(), a.data_ptr(), dx.data_ptr(), m, k, r, 1, 1.0, st), "train_expand")
    N.count(6)
    return dx, da, db


# ---- attention block --------------------------------------------------------------------------------------------
def attention_takes(qkv, q_norm_w, k_norm_w, positions, *, n_q, n_kv, head_dim, rotary_dim, gated) -> bool:
    if qkv.dim() != 3 or n_q % n_kv or head_dim % 4 or head_dim > 512 or rotary_dim % 2 or rotary_dim > head_dim or rotary_dim < 2:
        return False
    b, t, rows = qkv.shape
    return (rows == n_q * head_dim * (2 if gated else 1) + 2 * n_kv * head_dim and t <= 4096 and b * n_q * t < 1 << 31
            and tuple(positions.shape) in ((t,), (b, t), (1, t)) and q_norm_w.numel() == head_dim and k_norm_w.numel() == head_dim
            and positions.device == qkv.device and positions.dtype in INTEGERS and plain(qkv, q_norm_w, k_norm_w))


def attention(qkv, q_norm_w, k_norm_w, positions, *, n_q, n_kv, head_dim, rotary_dim, theta, eps, gated):
    """Output ``[B, T, n_q * head_dim]`` and the function of its gradient that gives qkv's."""
    (b, t, rows), d, half, lib = qkv.shape, head_dim, rotary_dim // 2, N.lib()
    inv = theta ** (-torch.arange(half, dtype=torch.float64, device=qkv.device) * 2.0 / rotary_dim)
    pos = positions.reshape(-1, t).to(torch.int64).contiguous()
    ang = pos.to(torch.float64)[..., None] * inv
    cs, sn, pr = ang.cos().float(), ang.sin().float(), pos.shape[0]
    dims = (b, t, n_q, n_kv, d, half, int(gated), pr, eps)
    new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=qkv.device)
    head = (qkv.data_ptr(), q_norm_w.data_ptr(), k_norm_w.data_ptr(), cs.data_ptr(), sn.data_ptr())
    q, k, v = new(b * n_kv, n_q // n_kv * t, d), new(b * n_kv, t, d), new(b * n_kv, t, d)
    N.check(lib.trl_train_attn_prep(*head, q.data_ptr(), k.data_ptr(), v.data_ptr(), *dims, N.stream()), "train_attn_prep")
    sc = 1.0 / d ** 0.5
    p = torch.bmm(q, k.transpose(1, 2))
    N.check(lib.trl_train_softmax(p.data_ptr(), pos.data_ptr(), pr, b, n_q, t, sc, N.stream()), "train_softmax")
    o = torch.bmm(p, v)
    out = new(b, t, n_q * d)
    N.check(lib.trl_train_attn_gate(o.data_ptr(), qkv.data_ptr(), out.data_ptr(), b, t, n_q, d, rows, int(gated), 0, N.stream()), "train_attn_gate")
    N.count(3)

    def backward(gout):
        up, go, dqkv = _grad(gout), torch.empty_like(o), torch.empty_like(qkv)
        N.check(lib.trl_train_attn_gate(up.data_ptr(), qkv.data_ptr(), go.data_ptr(), b, t, n_q, d, rows, int(gated), 1, N.stream()), "train_attn_gate")
        dv = torch.bmm(p.transpose(1, 2), go)
        ds = torch.bmm(go, v.transpose(1, 2))
        N.check(lib.trl_train_softmax_grad(p.data_ptr(), ds.data_ptr(), b * n_q * t, t, sc, N.stream()), "train_softmax_grad")
        dq, dk = torch.bmm(ds, k), torch.bmm(ds.transpose(1, 2), q)
        N.check(lib.trl_train_attn_prep_grad(qkv.data_ptr(), q_norm_w.data_ptr(), k_norm_w.data_ptr(), cs.data_ptr(), sn.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                                             dv.data_ptr(), o.data_ptr(), up.data_ptr(), dqkv.data_ptr(), *dims, N.stream()), "train_attn_prep_grad")
        N.count(3)
        return dqkv

    return out, backward


# ---- cross-entropy ------------------------------------------------------------------------------------------------
def cross_entropy_takes(logits, targets, weights) -> bool:
    """Not many rows of few classes: 262 144 x 128 1714 us with its gradient, 830 as torch ops; 65 536 x 1000 601 and 986."""
    if logits.shape[-1] < 512 and logits.numel() > 8192 * logits.shape[-1]:
        return False
    return logits.shape[-1] % 4 == 0 and plain(logits) and targets.device == logits.device and weights.device == logits.device \
        and targets.numel() == weights.numel() == logits.numel() // logits.shape[-1] < 1 << 31


def lse(lg):
    """``[3, rows]``: largest value, sum of exponentials below it, log-sum-exp."""
    out = torch.empty(3, lg.shape[0], dtype=torch.float32, device=lg.device)
    N.check(N.lib().trl_train_lse(lg.data_ptr(), out.data_ptr(), lg.shape[0], lg.shape[1], N.stream()), "train_lse")
    N.count()
    return out


def cross_entropy_grad(lg, stats, targets, weights):
    g = torch.empty_like(lg)
    N.check(N.lib().trl_train_ce_grad(lg.data_ptr(), stats.data_ptr(), targets.data_ptr(), weights.data_ptr(), g.data_ptr(),
                                      lg.shape[0], lg.shape[1], N.stream()), "train_ce_grad")
    N.count()
    return g


def scale_by(t, up):
    """``t`` times a number on the device, in place (nothing is touched where it is 1)."""
    up = up.reshape(1).float()
    N.check(N.lib().trl_train_scale_by(t.data_ptr(), up.data_ptr(), t.numel(), N.stream()), "train_scale_by")
    torch.autograd.graph.increment_version(t)
    N.count()
    return t


# ---- many tensors at a time -------------------------------------------------------------------------------------------
def _addresses(tensors: Sequence[torch.Tensor]) -> List[int]:
    return [t.data_ptr() for t in tensors]


def _pointers(addresses: Sequence[int]):
    return (ctypes.c_void_p * len(addresses))(*addresses)


def _lengths(lengths: Sequence[int]):
    return (ctypes.c_long * len(lengths))(*lengths)


def _floats(v: Sequence[float]):
    return (ctypes.c_float * len(v))(*v)


def apart(written: Sequence[tuple], read: Sequence[tuple] = ()) -> bool:
    """Of (address, values) of fp32 tensors: none that is written shares memory with another one (a weight under two names, a gradient given
    twice), since the tensors of a launch are worked on at the same time."""
    spans = sorted([(a, a + 4 * n, True) for a, n in written] + [(a, a + 4 * n, False) for a, n in read])
    if all(x[1] <= y[0] for x, y in zip(spans, spans[1:])):
        return True
    any_end = written_end = 0
    for start, end, w in spans:
        if start < (any_end if w else written_end):
            return False
        any_end = max(any_end, end)
        written_end = max(written_end, end) if w else written_end
    return True


def adamw(items: List[tuple], lr: float, betas, eps: float) -> None:
    """``items``: (parameter, m, v, gradient, decay factor, 1 - b1^t, 1 - b2^t), tensors plain.  One after the other where some share memory."""
    p, m, v, g, decay, c1, c2 = zip(*items)
    n, at = [t.numel() for t in p], [_addresses(ts) for ts in (p, m, v, g)]
    most = MAX_TENSORS if apart([x for a in at[:3] for x in zip(a, n)], list(zip(at[3], n))) else 1
    for i in range(0, len(items), most):
        part = slice(i, i + most)
        ptrs = [_pointers(a[part]) for a in at]
        N.check(N.lib().trl_train_adamw(*ptrs, _lengths(n[part]), _floats(decay[part]), _floats(c1[part]), _floats(c2[part]),
                                        len(n[part]), lr, betas[0], 1 - betas[0], betas[1], 1 - betas[1], eps, N.stream()), "train_adamw")
        N.count()
    torch.autograd.graph.increment_version(p + m + v)             # written in place, as ``copy_`` says it


def squares(grads: Dict[str, torch.Tensor]) -> Optional[torch.Tensor]:
    """Parts of the sum of squares of every gradient in fp64, a row each, in the order of the dict; ``None`` where the kernel does not
    take them all."""
    gs = list(grads.values())
    if not gs or not plain(*gs):
        return None
    n, at = [g.numel() for g in gs], _addresses(gs)
    blocks = N.lib().trl_train_squares_blocks(max(n))
    part = torch.empty(len(gs), blocks, dtype=torch.float64, device=gs[0].device)
    for i in range(0, len(gs), MAX_TENSORS):
        some = slice(i, i + MAX_TENSORS)
        N.check(N.lib().trl_train_squares(_pointers(at[some]), _lengths(n[some]), len(n[some]), blocks, part[i:].data_ptr(), N.stream()), "train_squares")
        N.count()
    return part


def scale(tensors: Sequence[torch.Tensor], c: float) -> None:
    """All of them times ``c``, in place (plain ones), one after the other where some share memory."""
    tensors = list(tensors)
    n, at = [t.numel() for t in tensors], _addresses(tensors)
    most = MAX_TENSORS if apart(list(zip(at, n))) else 1
    for i in range(0, len(n), most):
        some = slice(i, i + most)
        N.check(N.lib().trl_train_scale(_pointers(at[some]), _lengths(n[some]), len(n[some]), c, N.stream()), "train_scale")
        N.count()
    torch.autograd.graph.increment_version(tensors)
