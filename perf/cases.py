"""Workloads by which the speed of the serving and training paths is followed.

The product serves the 27B hybrid (Gated DeltaNet and gated grouped-query attention, NVFP4 weights) on one GPU, so most
cases are ticks of that model: captured decode ticks of one to many sequences, prompts, ticks that mix both, a speculative
verify tick, an fp8 KV pool, and one whole request.  They run a sixteenth of it: 4 of the 64 layers at full width (one
round of the pattern of three recurrent layers and one attention layer) and a sixteenth of the vocabulary, so that every
kernel has the sizes and the share of a tick that it has in the whole model.  At full depth a random-init network spreads
the rounding of one layer over tens of percent of its logits, and a wrong result could not be told from a rounded one.  The
small model of the same head geometry stands for calls whose time is launches, and for a training step with adapters.  Weights are random-init (N(0, 0.02) quantised to NVFP4), token ids are
uniform, KV pages and recurrent states of sequences in flight are drawn with the spread that such weights give them.

``exact`` repeats a pass in plain torch, 64 bits, from the served weights.
"""
import math
from dataclasses import replace

import torch

from tilerl_b200 import rl
from tilerl_b200.batch import Batch
from tilerl_b200.config import ATTN, get_config
from tilerl_b200.factory import build_engine, build_model, make_ops
from tilerl_b200.graph import VerifyGraphRunner
from tilerl_b200.kv import GdnStatePool, make_kv_pool
from tilerl_b200.optim import AdamW

PAGE = 16
BIG, SMALL = "qwen38-27b/16", "small-gpu"
#: the longest prompt whose pass is repeated in 64 bits: the recurrence runs token by token there
EXACT_TOKENS = 10000


def listed():
    return [
        # the smallest call: one token of one short chat on the small model; launches and host work count
        dict(name="decode-small", kind="decode", model=SMALL, seqs=1, context=100, kv="bf16"),
        # one whole interactive request, the headline: 512 tokens in, 64 out, through the engine tick by tick
        dict(name="request-512-64", kind="request", model=BIG, prompt=512, gen=64),
        # one user far into a long document: the KV read shows beside the weights
        dict(name="decode-1x32k", kind="decode", model=BIG, seqs=1, context=32749, kv="bf16"),
        # a small server, and the rollout of one group in RL: eight conversations of unlike length
        dict(name="decode-8x4k", kind="decode", model=BIG, seqs=8, context=4100, kv="bf16"),
        # a busy server, rollouts of several groups
        dict(name="decode-32x1k", kind="decode", model=BIG, seqs=32, context=1200, kv="bf16"),
        # the same with the e4m3 pool that long contexts of many users are kept in
        dict(name="decode-12x6k-fp8kv", kind="decode", model=BIG, seqs=12, context=6000, kv="fp8"),
        # speculative decoding: windows of eight drafted tokens of two sequences
        dict(name="verify-2x8", kind="verify", model=BIG, seqs=2, width=8, context=1500),
        # a short question: the first token's latency, rows not a multiple of any tile
        dict(name="prefill-37", kind="prefill", model=BIG, tokens=37, chunk=512),
        # an agent's prompt in one tick
        dict(name="prefill-2000", kind="prefill", model=BIG, tokens=2000, chunk=2048),
        # a long document in chunks, the later ones attending to the earlier
        dict(name="prefill-8192", kind="prefill", model=BIG, tokens=8192, chunk=2048),
        # continuous batching: prompts of unlike length enter while others decode
        dict(name="mixed-6+3", kind="mixed", model=BIG, seqs=6, context=900, prompts=3, tokens=330),
        # RL and fine-tuning: a supervised step on adapters over the frozen NVFP4 base
        dict(name="train-lora-4x512", kind="train", model=SMALL, seqs=4, tokens=512),
    ]


def _config(name):
    name, _, part = name.partition("/")
    cfg = get_config(name)
    if not part:
        return cfg
    return replace(cfg, name=name + "-part", layer_types=cfg.layer_types[:cfg.n_layers // int(part)], vocab=cfg.vocab // int(part))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "request", "verify", "prefill", "prefill", "mixed", "train"])
    model = BIG if rng.random() < 0.85 else SMALL
    if kind == "decode":
        seqs = _log(rng, 1, 40)
        return dict(kind=kind, model=model, seqs=seqs, context=_log(rng, 60, 32768 // seqs + 800),
                    kv="fp8" if rng.random() < 0.25 else "bf16")
    if kind == "request":
        return dict(kind=kind, model=model, prompt=_log(rng, 20, 600), gen=rng.randint(4, 64))
    if kind == "verify":
        return dict(kind=kind, model=model, seqs=rng.randint(1, 4), width=rng.randint(2, 8), context=_log(rng, 100, 4000))
    if kind == "prefill":
        return dict(kind=kind, model=model, tokens=_log(rng, 17, 6000), chunk=rng.choice([512, 1024, 2048]))
    if kind == "mixed":
        return dict(kind=kind, model=model, seqs=rng.randint(1, 12), context=_log(rng, 100, 2000), prompts=rng.randint(1, 4),
                    tokens=_log(rng, 40, 500))
    return dict(kind=kind, model=SMALL, seqs=rng.randint(1, 4), tokens=_log(rng, 60, 512))


# ---- what a program has in hand ------------------------------------------------------------------------
def _contexts(case):
    """Lengths of the sequences in flight: the longest first, the others down to about half of it."""
    c = case["context"]
    return [max(1, c - i * 389 % max(1, c // 2)) for i in range(case["seqs"])]


def _prompts(case):
    n = case["tokens"]
    return [max(1, n - i * 131 % max(1, n // 2)) for i in range(case["prompts"])]


def _ids(n, vocab, seed):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _fill(pool, states, seed):
    """Pages and states as sequences in flight have them: K rows normed to unit size, V rows and convolution inputs of
    the spread that a projection of a normed row has, states of some dozens of decayed outer products."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    for i in range(pool.k.shape[0]):
        shape = pool.k[i].shape
        for store, scale, std in ((pool.k, "k_scale", 1.0), (pool.v, "v_scale", 1.4)):
            x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).mul_(std)
            if pool.fp8:
                s = x.abs().amax(-1).clamp_min(1e-8) / 448.0
                getattr(pool, scale)[i].copy_(s)
                x.div_(s.unsqueeze(-1))
            store[i].copy_(x)
    states.states.normal_(0.0, 0.05, generator=g)
    for i in range(states.ring.shape[1]):
        states.ring[:, i].copy_(torch.randn(states.ring[:, i].shape, generator=g, device="cuda") * 1.4)


def _in_flight(case, cfg, need, planes=1):
    """Pools with the sequences of the case in them, pages scattered as after some hours of serving.  ``need``: positions
    each sequence's pages have to reach."""
    pages = [(n + PAGE - 1) // PAGE for n in need]
    pool = make_kv_pool(cfg, sum(pages) + 1, torch.device("cuda"), torch.bfloat16, n_kv_heads=cfg.n_kv_heads,
                        fp8=case.get("kv") == "fp8")
    states = GdnStatePool(cfg, len(need) + 1, "cuda", planes=planes)
    g = torch.Generator().manual_seed(case["seed"])
    order = (torch.randperm(sum(pages), generator=g) + 1).tolist()
    blocks, o = [], 0
    for n in pages:
        blocks.append(order[o:o + n])
        o += n
    _fill(pool, states, case["seed"] + 1)
    return pool, states, blocks


def prepare(case, seed):
    cfg = _config(case["model"])
    case = dict(case, seed=seed)
    ops = make_ops("cuda")
    model = build_model(cfg, "cuda", seed=seed & 0xFFFF, ops=ops)
    ops.vocab = cfg.vocab
    st = dict(case=case, cfg=cfg, ops=ops, model=model)
    kind = case["kind"]
    if kind in ("request", "prefill"):
        n = case["prompt"] + case["gen"] if kind == "request" else case["tokens"]
        st["ids"] = _ids(n, cfg.vocab, seed)
        st["engine"] = build_engine(model, ops, blocks=(n + PAGE - 1) // PAGE + 1, slots=1, max_ctx=n + PAGE, prefix=False)
        if kind == "request":
            st["engine"].precapture((1,))
    elif kind == "train":
        model.add_lora(rank=16, targets=("qkv", "in", "gate_up", "down"), seed=seed & 0xFFFF)
        g = torch.Generator(device="cuda").manual_seed(seed)
        for k, v in model.trainable().items():
            if k.endswith("lora_b"):
                v.normal_(0.0, 0.02, generator=g)
        st["ids"] = torch.tensor(_ids(case["seqs"] * case["tokens"], cfg.vocab, seed), device="cuda").view(case["seqs"], -1)
        st["opt"] = AdamW(model.trainable(), lr=1e-5)
    else:
        ctx = _contexts(case)
        if kind == "mixed":
            new = _prompts(case)
            toks = [_ids(1, cfg.vocab, seed + 7 * i) for i in range(len(ctx))] + [_ids(n, cfg.vocab, seed + 1009 * (i + 1)) for i, n in enumerate(new)]
            start = ctx + [0] * len(new)
        else:
            w = case.get("width", 1)
            toks = [_ids(w, cfg.vocab, seed + 7 * i) for i in range(len(ctx))]
            start = ctx
        planes = case.get("width", 1)
        pool, states, blocks = _in_flight(case, cfg, [s + len(t) for s, t in zip(start, toks)], planes)
        if kind == "mixed":
            for i in range(len(ctx), len(start)):      # a request that enters starts from an empty state
                states.states[i + 1].zero_()
                states.ring[i + 1].zero_()
        seqs = [dict(tokens=t, start=s, blocks=b, slot=i + 1, keep=kind == "verify")
                for i, (t, s, b) in enumerate(zip(toks, start, blocks))]
        st.update(pool=pool, states=states, seqs=seqs)
        longest = max(start) + case.get("width", 1) + PAGE
        if kind == "decode":
            from tilerl_b200.graph import DecodeGraphRunner
            st["runner"] = DecodeGraphRunner(model, ops, pool, states, max_ctx=longest)
            st["runner"].precapture((len(seqs),))
        elif kind == "verify":
            st["runner"] = VerifyGraphRunner(model, ops, pool, states, max_ctx=longest, width=case["width"])
    return st


# ---- one pass -------------------------------------------------------------------------------------------
def _kept(pool, states, n):
    """The caches that the pass wrote into (views)."""
    out = {"states": states.states[1:n + 1], "ring": states.ring[1:n + 1]}
    if pool.fp8:
        out.update(k_scale=pool.k_scale[:, 1:], v_scale=pool.v_scale[:, 1:])
    else:
        out.update(k=pool.k[:, 1:], v=pool.v[:, 1:])     # page 0 takes the writes of padding rows
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "train":
        m = rl.train_step(st["model"], st["ids"], st["opt"], checkpoint_layers=True)
        return {"loss": m["loss"], "grad_norm": m["grad_norm"], "weights": st["model"].trainable(), "moments": st["opt"].m}
    if kind == "prefill":
        eng, ids, c = st["engine"], st["ids"], case["chunk"]
        for a in range(0, len(ids), c):
            part = ids[a:a + c]
            last = a + len(part) == len(ids)
            logits = eng.feed([("r", part, [len(part) - 1] if last else [])], end=["r"] if last else [])
        return {"logits": logits, **_kept(eng.kv, eng.states, 1)}
    if kind == "request":
        eng, ids, p = st["engine"], st["ids"], case["prompt"]
        out = [eng.feed([("r", ids[:p], [p - 1])]).clone()]
        for i in range(p, len(ids) - 1):
            out.append(eng.feed([("r", ids[i:i + 1], [0])], end=["r"] if i == len(ids) - 2 else []))
        return {"logits": torch.cat(out), **_kept(eng.kv, eng.states, 1)}
    pool, states, n = st["pool"], st["states"], len(st["seqs"])
    if kind == "decode":
        logits = st["runner"].run(st["seqs"]).logits
    elif kind == "verify":
        logits = st["runner"].run(st["seqs"], need_logits=True).logits
    else:
        batch = Batch.build(st["seqs"], "cuda")
        logits = st["model"].forward(batch, st["ops"], pool, states)
    return {"logits": logits, **_kept(pool, states, n)}


# ---- what a pass cannot do without ------------------------------------------------------------------------
def _tokens(case):
    """(new tokens, wanted logits rows, sum over new tokens of the keys they see, keys read, sequences, times the weights
    are read)."""
    kind = case["kind"]
    if kind == "prefill":
        n = case["tokens"]
        return n, 1, n * (n + 1) // 2, n, 1, (n + case["chunk"] - 1) // case["chunk"]
    if kind == "request":
        n = case["prompt"] + case["gen"] - 1
        return n, case["gen"], n * (n + 1) // 2, n * case["gen"], 1, case["gen"]
    ctx = _contexts(case)
    w = case.get("width", 1)
    new, rows, seen, read = w * len(ctx), w * len(ctx), sum(w * c + w * (w + 1) // 2 for c in ctx), sum(c + w for c in ctx)
    seqs = len(ctx)
    if kind == "mixed":
        for n in _prompts(case):
            new, rows, seen, read, seqs = new + n, rows + 1, seen + n * (n + 1) // 2, read + n, seqs + 1
    return new, rows, seen, read, seqs, 1


def _projection_params(cfg):
    h, n = cfg.hidden, 0
    for t in cfg.layer_types:
        n += 3 * h * cfg.ffn
        n += cfg.qkv_rows * h + h * cfg.attn_out_dim if t == ATTN else cfg.gdn_in_rows * h + h * cfg.gdn_v_dim
    return n


def work(case):
    cfg = _config(case["model"])
    proj, head = _projection_params(cfg), cfg.vocab * cfg.hidden
    if case["kind"] == "train":
        t = case["seqs"] * case["tokens"]
        # forward, its repetition and the gradient of the inputs; the frozen base has no gradient of its own
        return {"bytes": 3 * 0.5625 * proj + 2 * 2 * head + 4.0 * t * cfg.vocab, "flops": 2.0 * t * (3 * proj + 2 * head)}
    new, rows, seen, read, seqs, times = _tokens(case)
    kv = 2 * cfg.n_kv_heads * (cfg.head_dim + 4 if case.get("kv") == "fp8" else 2 * cfg.head_dim) * cfg.n_attn_layers
    state = 4 * cfg.gdn_v_heads * cfg.gdn_head_dim ** 2 * cfg.n_gdn_layers
    ticks = times if case["kind"] == "request" else 1
    nbytes = times * 0.5625 * proj + ticks * 2 * head + kv * (read + new) + state * 2 * seqs * times \
        + (state * (case["width"] - 1) * seqs if case["kind"] == "verify" else 0) + 4 * rows * cfg.vocab
    flops = 2.0 * new * proj + 2.0 * rows * head + 4.0 * seen * cfg.n_q_heads * cfg.head_dim * cfg.n_attn_layers \
        + 8.0 * new * cfg.gdn_v_heads * cfg.gdn_head_dim ** 2 * cfg.n_gdn_layers
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    # Measured against exact(): logits 0.01 to 0.02 off with up to 8 rows (bf16 stream and projections), 0.05 to 0.07 with
    # more, where activations are kept as two NVFP4 terms.  Two correct implementations share that rounding and part where
    # sums in another order tip a rounding over.  Gradients of the adapters are 0.02 off (bf16 products).
    return {"rel": 0.03}


# ---- the same in 64 bits ------------------------------------------------------------------------------------
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _w64(w):
    """A served weight in 64 bits: NVFP4 (two e2m1 codes a byte, the low nibble first, an e4m3 scale for 16 weights, one
    scale for the tensor) or plain."""
    if isinstance(w, torch.Tensor):
        return w.double()
    lut = torch.tensor(_E2M1 + tuple(-v for v in _E2M1), dtype=torch.float64, device=w.wq.device)
    v = torch.stack([lut[(w.wq & 15).int()], lut[(w.wq >> 4).int()]], -1).flatten(-2)
    n, k = v.shape
    return (v.view(n, k // 16, 16) * w.scale.float().double().unsqueeze(-1) * w.tscale.double()).view(n, k)


def _norm(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _rope(x, pos, cfg):
    half = cfg.rotary_dim // 2
    inv = cfg.rope_theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) * 2.0 / cfg.rotary_dim)
    a = (pos.double()[:, None] * inv)[:, None]
    x1, x2, rest = x[..., :half], x[..., half:2 * half], x[..., 2 * half:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin(), rest], -1)


def _attend(qkv, p, cfg, start, past):
    """Gated attention of one sequence's new tokens: ``past`` = its (K, V) so far, ``[n, kv heads, dim]`` each."""
    t, d, nq, nkv = qkv.shape[0], cfg.head_dim, cfg.n_q_heads, cfg.n_kv_heads
    pos = torch.arange(start, start + t, device=qkv.device)
    qg = qkv[:, :2 * nq * d].view(t, nq, 2, d)
    q = _rope(_norm(qg[:, :, 0], p["q_norm"], cfg.rms_eps), pos, cfg)
    k = _rope(_norm(qkv[:, 2 * nq * d:(2 * nq + nkv) * d].view(t, nkv, d), p["k_norm"], cfg.rms_eps), pos, cfg)
    v = qkv[:, (2 * nq + nkv) * d:].view(t, nkv, d)
    if past is not None:
        k, v = torch.cat([past[0], k]), torch.cat([past[1], v])
    hidden = torch.arange(k.shape[0], device=q.device)[None] > pos[:, None]
    out = []
    for h in range(nkv):
        s = torch.einsum("tgd,nd->gtn", q[:, h * (nq // nkv):(h + 1) * (nq // nkv)], k[:, h]) / math.sqrt(d)
        out.append(torch.einsum("gtn,nd->tgd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), v[:, h]))
    return (torch.cat(out, 1) * torch.sigmoid(qg[:, :, 1])).reshape(t, nq * d)


def _delta(inp, p, cfg, before, s, each=False):
    """Gated delta rule of one sequence's new tokens: ``before`` = the convolution's last inputs, ``s`` = the state.
    Returns the rows, and the state after the last token (after each of them)."""
    t, d, nk, nv, w = inp.shape[0], cfg.gdn_head_dim, cfg.gdn_k_heads, cfg.gdn_v_heads, cfg.gdn_conv
    c = (2 * nk + nv) * d
    rows = torch.cat([before, inp[:, :c]])
    conv = p["conv"].double()
    y = torch.nn.functional.silu(sum(rows[j:j + t] * conv[:, j] for j in range(w)))
    q, k, v = y[:, :nk * d].view(t, nk, d), y[:, nk * d:2 * nk * d].view(t, nk, d), y[:, 2 * nk * d:].view(t, nv, d)
    unit = lambda x: (x / torch.sqrt(x.pow(2).sum(-1, keepdim=True) + 1e-12)).repeat_interleave(nv // nk, 1)
    q, k = unit(q) / math.sqrt(d), unit(k)
    z, a, b = inp[:, c:c + nv * d].view(t, nv, d), inp[:, c + nv * d:c + nv * d + nv], inp[:, c + nv * d + nv:]
    decay = torch.exp(-torch.exp(p["a_log"].double()) * torch.nn.functional.softplus(a + p["dt_bias"].double(), threshold=700.0))
    beta = torch.sigmoid(b)
    out, steps = [], []
    for i in range(t):
        s = s * decay[i][:, None, None]
        u = (v[i] - torch.bmm(k[i][:, None], s)[:, 0]) * beta[i][:, None]
        s = s + k[i][:, :, None] * u[:, None]
        out.append(torch.bmm(q[i][:, None], s)[:, 0])
        if each:
            steps.append(s)
    o = torch.stack(out)
    return (_norm(o, p["gdn_norm"], cfg.rms_eps) * torch.nn.functional.silu(z)).reshape(t, nv * d), steps if each else s


def _layers(cfg, params, x, seqs, linear):
    """The decoder's layers over rows ``x`` of several sequences, each ``{"n", "start", "past": f(attention layer),
    "before": f(recurrent layer), "state": f(recurrent layer), "each"}``.  Returns rows and states by recurrent layer."""
    states, ai, gi = [], 0, 0
    for i, t in enumerate(cfg.layer_types):
        pre = "L%d." % i
        p = {k[len(pre):]: v for k, v in params.items() if k.startswith(pre)}
        h = _norm(x, p["norm1"], cfg.rms_eps)
        y = linear(h, pre + ("qkv" if t == ATTN else "in"))
        rows, o, kept = [], 0, []
        for s in seqs:
            part = y[o:o + s["n"]]
            o += s["n"]
            if t == ATTN:
                rows.append(_attend(part, p, cfg, s["start"], s["past"](ai)))
            else:
                r, after = _delta(part, p, cfg, s["before"](gi), s["state"](gi), s.get("each", False))
                rows.append(r)
                kept.append(torch.stack(after) if s.get("each") else after)
        if t == ATTN:
            ai += 1
        else:
            gi += 1
            states.append(kept)
        x = x + linear(torch.cat(rows), pre + ("o" if t == ATTN else "out"))
        gu = linear(_norm(x, p["norm2"], cfg.rms_eps), pre + "gate_up")
        x = x + linear(torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2], pre + "down")
    return x, states


def _head(cfg, params, x):
    h = _norm(x, params["final_norm"], cfg.rms_eps)
    return torch.cat([h @ w.double().t() for w in params["lm_head"].split(16384)], 1)


def _exact_train(st):
    cfg, params, ids = st["cfg"], st["model"].params, st["ids"]
    leaves = {k: v.double().requires_grad_() for k, v in st["model"].trainable().items()}
    scale = {k: v[2] for k, v in st["model"].lora.items()}

    def linear(x, name):
        y = x @ _w64(params[name]).t()
        return y + (x @ leaves[name + ".lora_a"].t()) @ leaves[name + ".lora_b"].t() * scale[name] if name in scale else y

    b, t = ids.shape
    empty = dict(past=lambda i: None, before=lambda i: torch.zeros(cfg.gdn_conv - 1, cfg.gdn_conv_dim, dtype=torch.float64, device="cuda"),
                 state=lambda i: torch.zeros(cfg.gdn_v_heads, cfg.gdn_head_dim, cfg.gdn_head_dim, dtype=torch.float64, device="cuda"))
    loss = 0.0
    for row in ids:                                  # one sequence at a time: the graph of a recurrence is large
        x, _ = _layers(cfg, params, params["embed"][row].double(), [dict(empty, n=t, start=0)], linear)
        part = torch.nn.functional.cross_entropy(_head(cfg, params, x)[:-1], row[1:], reduction="sum") / (b * (t - 1))
        part.backward()
        loss += float(part.detach())
    norm = math.sqrt(sum(float(v.grad.pow(2).sum()) for v in leaves.values()))
    o = st["opt"]
    c = 1.0 / (norm + 1e-6) if norm > 1.0 else 1.0
    weights, moments = {}, {}
    for k, v in leaves.items():
        g = v.grad * c
        moments[k] = (1 - o.betas[0]) * g
        weights[k] = v.detach() - o.lr * g / (g.abs() + o.eps)
    return {"loss": loss, "grad_norm": norm, "weights": weights, "moments": moments}


def exact(case, seed):
    if case["kind"] != "train" and _tokens(case)[0] > EXACT_TOKENS:
        return None
    st = prepare(case, seed)
    if case["kind"] == "train":
        return _exact_train(st)
    with torch.no_grad():
        return _exact_tick(st)


def _exact_tick(st):
    cfg, params, kind = st["cfg"], st["model"].params, st["case"]["kind"]
    nothing = lambda i: None
    if kind in ("prefill", "request"):
        ids = st["ids"] if kind == "prefill" else st["ids"][:-1]
        states = st["engine"].states
        seqs = [dict(tokens=ids, start=0, blocks=[], slot=1)]
        want = [len(ids) - 1] if kind == "prefill" else list(range(st["case"]["prompt"] - 1, len(ids)))
        fresh = True
    else:
        pool, states, seqs, fresh = st["pool"], st["states"], st["seqs"], False
        want, o = [], 0
        for s in seqs:
            n = len(s["tokens"])
            want += list(range(o, o + n)) if kind == "verify" else [o + n - 1]
            o += n
    w = cfg.gdn_conv - 1

    def past(s):
        if s["start"] == 0:
            return nothing
        n, b = s["start"], torch.tensor(s["blocks"], device="cuda")

        def rows(store, scale, i):
            x = store[i][b].float()
            if pool.fp8:
                x = x * scale[i][b].unsqueeze(-1)
            return x.transpose(1, 2).reshape(-1, cfg.n_kv_heads, cfg.head_dim)[:n].double()
        return lambda i: (rows(pool.k, getattr(pool, "k_scale", None), i), rows(pool.v, getattr(pool, "v_scale", None), i))

    def before(s):
        at = [p % states.ring.shape[2] for p in range(s["start"] - w, s["start"])]

        def rows(i):
            r = states.ring[s["slot"], i][at].double()
            for j in range(w):
                if fresh or s["start"] - w + j < 0:
                    r[j] = 0.0
            return r
        return rows

    def state(s):
        return lambda i: torch.zeros_like(states.states[1, i, 0], dtype=torch.float64) if fresh else states.states[s["slot"], i, 0].double()

    todo = [dict(n=len(s["tokens"]), start=s["start"], past=past(s), before=before(s), state=state(s), each=kind == "verify") for s in seqs]
    flat = torch.tensor([t for s in seqs for t in s["tokens"]], device="cuda")
    x, after = _layers(cfg, params, params["embed"][flat].double(), todo, lambda a, name: a @ _w64(params[name]).t())
    logits = _head(cfg, params, x[want])
    # [sequence, recurrent layer, plane, head, key, value], as the pool keeps them
    kept = torch.stack([torch.stack([(layer[i] if kind == "verify" else layer[i][None]) for layer in after]) for i in range(len(seqs))])
    return {"logits": logits, "states": kept, "ring": None}
