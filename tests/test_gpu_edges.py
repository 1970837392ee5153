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
    (1, 19000, 1024, 0), (13, 19001, 1280, 0), (4, 10100, 2560, 0), (16, 9999, 2048, 4),
    (4, 32761, 1024, 0), (8, 19001, 1280, 0), (5, 9999, 2048, 0), (12, 32761, 1024, 0), (16, 9999, 2560, 0)])
def test_bf16_rows_for_every_split_of_k(ops, m, n, k, shift):
    """K shared by 4, 8 and 16 warps in sets of 4 and 5 loads, with one and two tiles of activation rows; K shorter than the 16
    warps, shared unevenly, and up to what shared memory holds with two, one and no
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


@pytest.mark.parametrize("k", [32, 256, 288, 5120, 10240, 10496, 17408, 18432, 18464])
@pytest.mark.parametrize("tokens,terms,swiglu", [(1, 4, False), (3, 2, True), (130, 2, False), (17, 1, False)])
def test_activation_quantiser_row_kernel_gives_the_general_kernels_bits(ops, k, tokens, terms, swiglu):
    """Rows on a 16-byte boundary up to 18 432 values take the kernel that keeps the row in registers, others the general one:
    the same values in both alignments, the same bytes, zero scales in the padding of K (without a norm; with one, sums in
    another order move the reciprocal root by its last bit, and single codes with it)."""
    from tilerl_b200.ops.gemm_tc import quant_act
    g = torch.Generator().manual_seed(k + tokens)
    width = 2 * k if swiglu else k
    x = (torch.randn(tokens, width, generator=g) * torch.exp(torch.randn(tokens, 1, generator=g))).to(DEV, torch.bfloat16)
    x[0, :16] = 0
    off = torch.zeros(tokens, width + 8, dtype=torch.bfloat16, device=DEV)[:, 4:4 + width]
    off.copy_(x)
    if swiglu:       # pairs are read 16 bytes at a time in both kernels
        off = x
    nk = (k + 255) // 256
    cols = tokens * terms
    xq, sf, rs = (a.clone() for a in quant_act(ops, x, k, terms, swiglu_in=swiglu))
    yq, tf, ts = quant_act(ops, off, k, terms, swiglu_in=swiglu)
    c = torch.arange(cols, device=DEV)
    rows = lambda s: s.view(-1, nk * 4, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(-1, nk * 16)[c]
    assert torch.equal(xq, yq) and torch.equal(rs, ts) and torch.equal(rows(sf), rows(tf))
    assert int(rows(sf)[:, k // 16:].sum()) == 0
    if swiglu:
        return
    nw = (1.0 + 0.1 * torch.randn(k, generator=g)).to(DEV)
    xq, sf, rs = (a.clone() for a in quant_act(ops, x, k, terms, norm_w=nw, eps=1e-6))
    yq, tf, ts = quant_act(ops, off, k, terms, norm_w=nw, eps=1e-6)
    assert float((xq != yq).float().mean()) < 2e-3 and _rel(rs, ts) < 2 ** -7
    assert float((rows(sf) != rows(tf)).float().mean()) < 2e-3


@pytest.mark.parametrize("g_heads,splits", [(1, 1), (6, 1), (6, 5), (8, 3)])
@pytest.mark.parametrize("scale_v", [1.0, 1e-25, 1e12])
def test_fp8_attention_on_tensor_cores(ops, g_heads, splits, scale_v):
    """Contexts at the edges of pages and splits, bytes past the sequence's end that are NaN, V of any magnitude, query rows far
    from one, against 64 bits.  The split's partial sums are fp32: weights in two f16 parts leave 2^-22 of each, sums over up
    to 1 100 keys their fp32 rounding; the finished row is bf16."""
    from tilerl_b200.ops import native as N
    import math
    n_kv, d = 2, 256
    n_q = n_kv * g_heads
    lens = [1, 2, 15, 16, 17, 127, 128, 129, 511, 1100]
    g = torch.Generator(device=DEV).manual_seed(g_heads * 10 + splits)
    t = len(lens)
    mb = (max(lens) + 15) // 16
    pages = t * mb + 1
    e4 = lambda x: x.clamp(-448, 448).to(torch.float8_e4m3fn)
    k8 = e4(torch.randn(pages, n_kv, 16, d, generator=g, device=DEV) * 40)
    v8 = e4(torch.randn(pages, n_kv, 16, d, generator=g, device=DEV) * 100)
    ks = torch.rand(pages, n_kv, 16, generator=g, device=DEV) * 0.02 + 0.01
    vs = torch.exp(torch.randn(pages, n_kv, 16, generator=g, device=DEV)) * scale_v
    table = (torch.randperm(pages - 1, generator=g, device=DEV)[:t * mb] + 1).int().view(t, mb)
    kd, vd = k8.double() * ks.double().unsqueeze(-1), v8.double() * vs.double().unsqueeze(-1)
    for i, n in enumerate(lens):                        # what lies past the sequence's end must not matter
        if n % 16:
            b = int(table[i, n // 16])
            for s in (k8, v8):
                s[b].view(torch.uint8)[:, n % 16:] = 0x7f
            ks[b, :, n % 16:] = vs[b, :, n % 16:] = float("nan")
    q = torch.randn(t, n_q, d, generator=g, device=DEV)
    q[1] *= 2.0 ** 20
    q[2] *= 2.0 ** -30
    q[3] = 0
    q = q.to(torch.bfloat16)
    gate = torch.randn(t, n_q * 2 * d, generator=g, device=DEV).to(torch.bfloat16)
    po = torch.full((t, n_q, splits, d), float("nan"), device=DEV)
    pm, pl = (torch.full((t, n_q, splits), float("nan"), device=DEV) for _ in range(2))
    out = torch.full((t, n_q * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    sid = torch.arange(t, dtype=torch.int32, device=DEV)
    N.check(ops.lib.trl_attn_paged_fp8(q.data_ptr(), gate.data_ptr(), gate.stride(0), k8.data_ptr(), v8.data_ptr(), ks.data_ptr(),
                                       vs.data_ptr(), table.data_ptr(), mb, sid.data_ptr(), pos.data_ptr(), po.data_ptr(),
                                       pm.data_ptr(), pl.data_ptr(), out.data_ptr(), t, n_q, n_kv, d, splits, 1 / math.sqrt(d), 1,
                                       N.stream()), "attn_paged_fp8")
    for i, n in enumerate(lens):
        b = table[i].long()
        kk = kd[b].transpose(1, 2).reshape(-1, n_kv, d)[:n]
        vv = vd[b].transpose(1, 2).reshape(-1, n_kv, d)[:n]
        s = torch.einsum("hgd,nhd->hgn", q[i].double().view(n_kv, g_heads, d), kk) / math.sqrt(d)
        want = torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), vv).reshape(n_q, d)
        if splits > 1:
            c = torch.exp2(pm[i].double() - pm[i].double().amax(-1, keepdim=True))
            got = (po[i].double() * c.unsqueeze(-1)).sum(1) / (pl[i].double() * c).sum(1, keepdim=True)
            tol = 2e-2 if i == 1 else 2e-5             # scores of 10^8: the last bit of an fp32 score is a factor in a weight
            assert _rel(got, want) < tol, (n, _rel(got, want))
        final = want * torch.sigmoid(gate[i].double().view(n_q, 2, d)[:, 1])
        assert _rel(out[i].view(n_q, d), final) < (2e-2 if i == 1 else 2 ** -8), n


@pytest.mark.parametrize("tokens,n,k", [(3, 20000, 512), (9, 700, 5120), (40, 19000, 288), (129, 128, 256), (130, 130, 288), (200, 384, 2048), (256, 1000, 5120), (257, 4130, 1056), (700, 640, 6144),
                                        (1111, 5120, 1024), (2100, 5120, 256)])
@pytest.mark.parametrize("split", [False, True, None])
def test_gemm_tiles_whole_and_split_equal_one_cta_alone(ops, tokens, n, k, split):
    """Tiles that several CTAs and one go through (their accumulator is given back before the values are stored), rows and K that
    fill no tile, tiles whole and split, every epilogue, against the same kernel on one CTA.  The same products in
    fp32, summed in another order where tiles are split."""
    from tilerl_b200 import formats as F
    from tilerl_b200.ops import native
    from tilerl_b200.ops.gemm_tc import gemm_nvfp4
    g = torch.Generator().manual_seed(tokens + n)
    w = F.quantize_nvfp4(torch.randn(n, k, generator=g) * 0.02).to(DEV)
    x = torch.randn(tokens, k, generator=g).to(DEV, torch.bfloat16)
    got, want = (torch.full((tokens, n), float("nan"), device=DEV) for _ in range(2))
    gemm_nvfp4(ops, x, w, want, terms=2, epi=3, max_ctas=1, split=False)
    for _ in range(2):
        gemm_nvfp4(ops, x, w, got, terms=2, epi=3, split=split)
        assert _rel(got, want) < 1e-6
    a = torch.full((tokens, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    gemm_nvfp4(ops, x, w, a, terms=2, split=split)
    assert _rel(a, want) < 2 ** -8
    if n % 2 == 0:
        h = torch.full((tokens, n // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
        gemm_nvfp4(ops, x, w, h, terms=2, epi=2, split=split)
        assert _rel(h, torch.nn.functional.silu(want[:, 0::2].double()) * want[:, 1::2].double()) < 2 ** -8
    r = torch.randn(tokens, n, generator=g).to(DEV, torch.bfloat16)
    acc = r.clone()
    gemm_nvfp4(ops, x, w, acc, terms=2, epi=1, residual=acc, split=split)
    assert _rel(acc, want.double() + r.double()) < 2 ** -8
    assert native.read_error()[0] == 0


@pytest.mark.parametrize("nk,nv,d,taps", [(2, 4, 128, 4), (1, 3, 128, 4), (2, 2, 64, 4), (2, 4, 128, 3)])
def test_delta_rule_prep_over_runs_of_tokens(ops, nk, nv, d, taps):
    """Convolution, norms and gates of tokens taken in runs of 8 (thousands of tokens), 4, 2 and 1: sequences that begin inside a
    run, at position 0 and later (their window then comes from the ring), shorter than the window, and a last run that is not
    full.  Scratch rows against 64 bits."""
    from tilerl_b200.ops import native as N
    c = (2 * nk + nv) * d
    for lens in ([1], [3, 1, 2], [7, 40, 1, 9, 300], [1500, 2, 3, 1, 1700], [5000]):
        g = torch.Generator().manual_seed(sum(lens) + d)
        t, b = sum(lens), len(lens)
        starts = [0 if i % 2 else 5 + 13 * i for i in range(b)]
        inp = torch.randn(t, c + nv * d + 2 * nv, generator=g).to(DEV, torch.bfloat16)
        conv = (torch.randn(c, taps, generator=g) * 0.3).to(DEV)
        dt, al = torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV)
        ring = torch.randn(b + 1, 16, c, generator=g).to(DEV, torch.bfloat16)
        keep = ring.clone()
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        q0 = [sum(lens[:i]) for i in range(b)]
        pos = i32([s + j for s, n in zip(starts, lens) for j in range(n)])
        seq = i32([i for i, n in enumerate(lens) for _ in range(n)])
        states = torch.zeros(b + 1, 1, 1, nv, d, d, device=DEV)
        f = lambda *s: torch.full(s, float("nan"), device=DEV)
        qn, kn, vc, gg, bb, o = f(t, nk, d), f(t, nk, d), f(t, nv, d), f(t, nv), f(t, nv), f(t, nv, d)
        out = torch.empty(t, nv * d, dtype=torch.bfloat16, device=DEV)
        cur = torch.zeros(b + 1, dtype=torch.int32, device=DEV)
        nw, qs, ql, slots = torch.ones(d, device=DEV), i32(q0), i32(lens), i32(list(range(1, b + 1)))
        N.check(ops.lib.trl_gdn(inp.data_ptr(), inp.stride(0), conv.data_ptr(), dt.data_ptr(), al.data_ptr(), nw.data_ptr(),
                                states.data_ptr(), cur.data_ptr(), ring.data_ptr(), pos.data_ptr(), seq.data_ptr(), qs.data_ptr(),
                                ql.data_ptr(), slots.data_ptr(), None, states.stride(0), states.stride(2),
                                ring.stride(0), qn.data_ptr(), kn.data_ptr(), vc.data_ptr(), gg.data_ptr(), bb.data_ptr(), o.data_ptr(),
                                out.data_ptr(), t, b, nk, nv, d, taps, 1, 1e-6, N.stream()), "gdn")
        x = inp.double()
        want = []
        for i, n in enumerate(lens):
            halo = torch.stack([keep[i + 1, (starts[i] - taps + 1 + j) % 16].double() if starts[i] - taps + 1 + j >= 0 else
                                torch.zeros(c, dtype=torch.float64, device=DEV) for j in range(taps - 1)])
            rows = torch.cat([halo, x[q0[i]:q0[i] + n, :c]])
            want.append(torch.nn.functional.silu(sum(rows[j:j + n] * conv[:, j].double() for j in range(taps))))
        want = torch.cat(want)
        unit = lambda a: a / torch.sqrt(a.pow(2).sum(-1, keepdim=True) + 1e-12)
        assert _rel(qn, unit(want[:, :nk * d].view(t, nk, d)) / d ** 0.5) < 1e-5
        assert _rel(kn, unit(want[:, nk * d:2 * nk * d].view(t, nk, d))) < 1e-5
        assert _rel(vc, want[:, 2 * nk * d:].view(t, nv, d)) < 1e-5
        assert _rel(bb, torch.sigmoid(x[:, c + nv * d + nv:])) < 1e-5
        assert _rel(gg, -torch.exp(al.double()) * torch.nn.functional.softplus(x[:, c + nv * d:c + nv * d + nv] + dt.double())) < 1e-5


@pytest.mark.parametrize("nk,nv,b,taps", [(16, 48, 5, 4), (16, 48, 32, 4), (1, 3, 75, 4), (2, 6, 37, 3), (8, 8, 149, 4)])
def test_decode_step_of_many_heads_equals_one_sequence_at_a_time(ops, nk, nv, b, taps):
    """Items that the blocks share evenly and unevenly, as few as the kernel of many items takes, positions before the
    convolution's window is full and past the ring's end, live planes other than the first.  The same arithmetic as the
    kernel of one item a block (which a single sequence takes), except for the order of the sum q.k."""
    from tilerl_b200.ops import native as N
    d, planes = 128, 2
    g = torch.Generator().manual_seed(b + nv)
    c = (2 * nk + nv) * d
    ld = c + nv * d + 2 * nv
    inp = torch.randn(b, ld, generator=g).to(DEV, torch.bfloat16)
    conv = (torch.randn(c, taps, generator=g) * 0.3).to(DEV)
    dt, al, nw = torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV), torch.rand(d, generator=g).to(DEV)
    ring = torch.randn(b + 1, 16, c, generator=g).to(DEV, torch.bfloat16)
    states = torch.randn(b + 1, 1, planes, nv, d, d, device=DEV) * 0.05
    cur = torch.randint(0, planes, (b + 1,), generator=g).to(DEV, torch.int32)
    pos = torch.tensor([(0, 1, 2, 3, 15, 16, 17, 40)[i % 8] for i in range(b)], dtype=torch.int32, device=DEV)
    qs = torch.arange(b, dtype=torch.int32, device=DEV)
    slots = (torch.randperm(b, generator=g) + 1).to(DEV, torch.int32)

    def step(s, r, o, rows):
        for i, n in rows:
            N.check(ops.lib.trl_gdn_decode(inp.data_ptr(), ld, conv.data_ptr(), dt.data_ptr(), al.data_ptr(), nw.data_ptr(), s.data_ptr(),
                                           cur.data_ptr(), r.data_ptr(), pos.data_ptr(), qs[i:].data_ptr(), slots[i:].data_ptr(), s.stride(0),
                                           s.stride(2), r.stride(0), o.data_ptr(), n, nk, nv, d, taps, 1e-6, N.stream()), "gdn_decode")
    s1, r1, o1 = states.clone(), ring.clone(), torch.zeros(b, nv * d, dtype=torch.bfloat16, device=DEV)
    s2, r2, o2 = states.clone(), ring.clone(), torch.zeros(b, nv * d, dtype=torch.bfloat16, device=DEV)
    step(s1, r1, o1, [(0, b)])
    step(s2, r2, o2, [(i, 1) for i in range(b)])
    assert torch.equal(s1, s2) and torch.equal(r1, r2)
    assert _rel(o1, o2) < 2e-4                        # a bf16 step where the sum's last bit tips a rounding over
    assert not torch.equal(s1, states) and N.read_error()[0] == 0


@pytest.mark.parametrize("g_heads", [1, 6, 7, 8])
@pytest.mark.parametrize("fp8", [False, True])
def test_prefill_attention_pairs_of_warps(ops, g_heads, fp8):
    """Queries and histories at the edges of 16-row tiles, 32-key halves and 64-key tiles, pool rows past a sequence's end that are
    NaN, both thread counts (up to six heads a group, and more), against 64 bits.  Weights and the result are bf16: 2^-9 each of
    what they carry, in the rms over rows whose keys are independent."""
    from tilerl_b200.ops import native as N
    import math
    n_kv, d = 2, 256
    n_q = n_kv * g_heads
    seqs = [(1, 0), (16, 0), (17, 15), (32, 0), (15, 49), (33, 31), (64, 1), (5, 123), (2, 127), (40, 500)]
    g = torch.Generator(device=DEV).manual_seed(g_heads * 2 + fp8)
    b, t = len(seqs), sum(n for n, _ in seqs)
    mb = max((n + h + 15) // 16 for n, h in seqs)
    pages = b * mb + 1
    k, v = (torch.randn(pages, n_kv, 16, d, generator=g, device=DEV) for _ in range(2))
    scales = [torch.ones(pages, n_kv, 16, device=DEV) for _ in range(2)]
    if fp8:
        scales = [torch.rand(pages, n_kv, 16, generator=g, device=DEV) * 0.02 + 0.01 for _ in range(2)]
        k, v = ((x * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for x in (k, v))
    else:
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
    kd, vd = (x.double() * s.double().unsqueeze(-1) for x, s in zip((k, v), scales))
    table = (torch.randperm(pages - 1, generator=g, device=DEV)[:b * mb] + 1).int().view(b, mb)
    for i, (n, h) in enumerate(seqs):                   # what lies past the sequence's end must not matter
        if (n + h) % 16:
            pg, r = int(table[i, (n + h) // 16]), (n + h) % 16
            for x in (k, v):
                x[pg].view(torch.uint8 if fp8 else torch.int16)[:, r:] = 0x7f if fp8 else 0x7fc0
            if fp8:
                scales[0][pg, :, r:] = scales[1][pg, :, r:] = float("nan")
    q = torch.randn(t, n_q, d, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(t, n_q * 2 * d, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((t, n_q * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(n for n, _ in seqs[:i]) for i in range(b)]
    qs, ql, pos = i32(starts), i32([n for n, _ in seqs]), i32([h + j for n, h in seqs for j in range(n)])
    tail = (qs.data_ptr(), ql.data_ptr(), pos.data_ptr(), out.data_ptr(), b, max(n for n, _ in seqs), n_q, n_kv, d,
            1 / math.sqrt(d), 1, N.stream())
    head = (q.data_ptr(), gate.data_ptr(), gate.stride(0), k.data_ptr(), v.data_ptr())
    if fp8:
        N.check(ops.lib.trl_attn_prefill_fp8(*head, scales[0].data_ptr(), scales[1].data_ptr(), table.data_ptr(), mb, *tail), "prefill_fp8")
    else:
        N.check(ops.lib.trl_attn_prefill(*head, table.data_ptr(), mb, pages, *tail), "prefill")
    for i, (n, h) in enumerate(seqs):
        blocks = table[i].long()
        kk, vv = (x[blocks].transpose(1, 2).reshape(-1, n_kv, d)[:n + h] for x in (kd, vd))
        rows = slice(starts[i], starts[i] + n)
        s = torch.einsum("thgd,nhd->thgn", q[rows].double().view(n, n_kv, g_heads, d), kk) / math.sqrt(d)
        s.masked_fill_((torch.arange(n + h, device=DEV) > (h + torch.arange(n, device=DEV)).view(n, 1)).view(n, 1, 1, -1), -math.inf)
        want = torch.einsum("thgn,nhd->thgd", torch.softmax(s, -1), vv).reshape(n, n_q, d)
        want = (want * torch.sigmoid(gate[rows].double().view(n, n_q, 2, d)[:, :, 1])).reshape(n, -1)
        assert _rel(out[rows], want) < 2 ** -7, (n, h, _rel(out[rows], want))


@pytest.mark.parametrize("nk,nv,d", [(2, 4, 128), (1, 3, 128), (2, 2, 64)])
def test_delta_rule_scan_of_kept_states(ops, nk, nv, d):
    """The state after every token, from states at even float addresses (the scan of two columns a lane) and at odd ones (the plain
    recurrence), against the rule in 64 bits on the rows that the preparation left; fp32 sums over up to 17 tokens."""
    from tilerl_b200.ops import native as N
    lens, taps, planes = [8, 1, 17, 16], 4, 18
    c, t, b = (2 * nk + nv) * d, sum(lens), len(lens)
    g = torch.Generator().manual_seed(d + nv)
    inp = torch.randn(t, c + nv * d + 2 * nv, generator=g).to(DEV, torch.bfloat16)
    conv = (torch.randn(c, taps, generator=g) * 0.3).to(DEV)
    dt, al, nw = torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV), torch.ones(d, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q0 = [sum(lens[:i]) for i in range(b)]
    pos, seq = i32([j for n in lens for j in range(n)]), i32([i for i, n in enumerate(lens) for _ in range(n)])
    qs, ql, slots, keep = i32(q0), i32(lens), i32(list(range(1, b + 1))), i32([1] * b)
    first = (torch.randn(b + 1, planes, nv, d, d, generator=g) * 0.05).to(DEV)
    for odd in (0, 1):
        states = torch.empty(first.numel() + 2, device=DEV)[odd:odd + first.numel()].view(first.shape)
        states.copy_(first)
        ring = torch.zeros(b + 1, 16, c, dtype=torch.bfloat16, device=DEV)
        f = lambda *s: torch.full(s, float("nan"), device=DEV)
        qn, kn, vc, gg, bb, o = f(t, nk, d), f(t, nk, d), f(t, nv, d), f(t, nv), f(t, nv), f(t, nv, d)
        out = torch.empty(t, nv * d, dtype=torch.bfloat16, device=DEV)
        cur = torch.full((b + 1,), planes - 1, dtype=torch.int32, device=DEV)
        N.check(ops.lib.trl_gdn(inp.data_ptr(), inp.stride(0), conv.data_ptr(), dt.data_ptr(), al.data_ptr(), nw.data_ptr(),
                                states.data_ptr(), cur.data_ptr(), ring.data_ptr(), pos.data_ptr(), seq.data_ptr(), qs.data_ptr(),
                                ql.data_ptr(), slots.data_ptr(), keep.data_ptr(), states.stride(0), states.stride(1),
                                ring.stride(0), qn.data_ptr(), kn.data_ptr(), vc.data_ptr(), gg.data_ptr(), bb.data_ptr(), o.data_ptr(),
                                out.data_ptr(), t, b, nk, nv, d, taps, planes, 1e-6, N.stream()), "gdn")
        rep = nv // nk
        for i, n in enumerate(lens):
            s = first[i + 1, planes - 1].double()
            for j in range(n):
                r = q0[i] + j
                k, q, v = kn[r].double().repeat_interleave(rep, 0), qn[r].double().repeat_interleave(rep, 0), vc[r].double()
                s = s * torch.exp(gg[r].double()).view(nv, 1, 1)
                s = s + k.unsqueeze(2) * (bb[r].double().unsqueeze(1) * (v - torch.einsum("hd,hdc->hc", k, s))).unsqueeze(1)
                assert _rel(states[i + 1, j], s) < 1e-5, (odd, n, j)
                x = torch.einsum("hd,hdc->hc", q, s)
                z = inp[r, c:c + nv * d].double().view(nv, d)
                want = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * torch.nn.functional.silu(z)
                assert _rel(out[r].view(nv, d), want) < 2 ** -7, (odd, n, j)


def _fp8_decode(ops, q, k8, v8, ks, vs, table, ctx, splits, gate=None):
    """(partial rows, maxima, sums, finished rows) of ``trl_attn_paged_fp8``: a row of ``q [t, heads, 256]`` a sequence."""
    from tilerl_b200.ops import native as N
    t, n_q, d = q.shape
    po = torch.full((t, n_q, splits, d), float("nan"), device=DEV)
    pm, pl = (torch.full((t, n_q, splits), float("nan"), device=DEV) for _ in range(2))
    out = torch.full((t, n_q * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pos, sid = i32([n - 1 for n in ctx]), i32(list(range(t)))
    g = torch.zeros(t, n_q * 2 * d, dtype=torch.bfloat16, device=DEV) if gate is None else gate
    N.check(ops.lib.trl_attn_paged_fp8(q.data_ptr(), g.data_ptr(), g.stride(0), k8.data_ptr(), v8.data_ptr(), ks.data_ptr(),
                                       vs.data_ptr(), table.data_ptr(), table.shape[1], sid.data_ptr(), pos.data_ptr(), po.data_ptr(),
                                       pm.data_ptr(), pl.data_ptr(), out.data_ptr(), t, n_q, k8.shape[1], d, splits, 1 / d ** 0.5,
                                       int(gate is not None), N.stream()), "attn_paged_fp8")
    return po, pm, pl, out


@pytest.mark.parametrize("kind,splits,bound", [
    ("typical", 9, 1e-6), ("long", 2, 1e-6), ("tail 14", 2, 1e-6), ("tail 20", 2, 1e-6), ("tail 20", 9, 1e-6), ("tail 25", 2, 2 ** -14)])
def test_fp8_attention_keeps_its_sums_in_fp32(ops, kind, splits, bound):
    """Partial sums against 64 bits, with contexts that a long chain of MMAs or weights cut to f16's range would show in: up to
    32 000 keys, and a flat tail of 30 000 keys that each weigh 2^-14 to 2^-25 of the first key, seen in the columns where that
    one's V is zero.  Scores of up to 20 are rounded to 2^-20 of a power of two in fp32, 7e-7 of a weight.  A weight of 2^-25
    of the largest keeps what is above 2^-39 of that, 2^-14 of itself."""
    d, n_kv, gh = 256, 2, 6
    t, ctx = (3, 6000) if kind == "typical" else (1, 32000 if kind == "long" else 30000)
    g = torch.Generator(device=DEV).manual_seed(5)
    mb = (ctx + 15) // 16
    k, v = (torch.randn(t * mb + 1, n_kv, 16, d, generator=g, device=DEV) for _ in range(2))
    v *= torch.exp(torch.randn(t * mb + 1, n_kv, 16, 1, generator=g, device=DEV))
    table = (torch.randperm(t * mb, generator=g, device=DEV) + 1).int().view(t, mb)
    q = torch.randn(t, n_kv * gh, d, generator=g, device=DEV)
    cols = slice(None)
    if kind.startswith("tail"):
        cols = slice(1, None)
        q.zero_()
        q[..., 0], k[..., 0] = 16.0, 0.0
        first = int(table[0, 0])
        k[first, :, 0, 0] = int(kind.split()[1]) * 0.6931471805599453
        v[..., 1:] += 1.0
        v[first, :, 0], v[first, :, 0, 0] = 0.0, 3.0
    q = q.to(torch.bfloat16)
    ks, vs = k.abs().amax(-1).clamp_min(1e-8) / 448, v.abs().amax(-1).clamp_min(1e-8) / 448
    k8, v8 = ((x / s.unsqueeze(-1)).clamp(-448, 448).to(torch.float8_e4m3fn) for x, s in ((k, ks), (v, vs)))
    po, pm, pl, _ = _fp8_decode(ops, q, k8, v8, ks, vs, table, [ctx] * t, splits)
    c = torch.exp2(pm.double() - pm.double().amax(-1, keepdim=True))
    got = (po.double() * c.unsqueeze(-1)).sum(2) / (pl.double() * c).sum(-1, keepdim=True)
    for i in range(t):
        b = table[i].long()
        kk, vv = ((x[b].double() * s[b].double().unsqueeze(-1)).transpose(1, 2).reshape(-1, n_kv, d)[:ctx] for x, s in ((k8, ks), (v8, vs)))
        s = torch.einsum("hgd,nhd->hgn", q[i].double().view(n_kv, gh, d), kk) / d ** 0.5
        want = torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), vv).reshape(n_kv * gh, d)
        assert _rel(got[i][:, cols], want[:, cols]) < bound, _rel(got[i][:, cols], want[:, cols])


@pytest.mark.parametrize("off_q,off_kv", [(1, 0), (0, 8), (4, 8)])
def test_fp8_attention_takes_rows_off_a_16_byte_boundary(ops, off_q, off_kv):
    """Queries on any element, K and V on any 8 bytes, as the kernel for one key a warp takes them, against the aligned call
    (the same weights and sums in fp32, in another order)."""
    d, n_kv, gh, t, ctx = 256, 2, 6, 3, 300
    g = torch.Generator(device=DEV).manual_seed(off_q + off_kv)
    mb = (ctx + 15) // 16
    pages = t * mb + 1
    k8, v8 = ((torch.randn(pages, n_kv, 16, d, generator=g, device=DEV) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for _ in range(2))
    ks, vs = (torch.rand(pages, n_kv, 16, generator=g, device=DEV) * 0.02 + 0.01 for _ in range(2))
    table = (torch.randperm(pages - 1, generator=g, device=DEV) + 1).int().view(t, mb)
    q = torch.randn(t, n_kv * gh, d, generator=g, device=DEV).to(torch.bfloat16)

    def moved(x, off):
        room = torch.empty(x.numel() + 64, dtype=x.dtype, device=DEV)
        y = room[off:off + x.numel()].view(x.shape)
        y.copy_(x)
        assert y.data_ptr() % 16 == off * x.element_size() % 16
        return y
    for splits in (1, 3):
        a = _fp8_decode(ops, q, k8, v8, ks, vs, table, [ctx, 17, 128], splits)[3]
        b = _fp8_decode(ops, moved(q, off_q), moved(k8, off_kv), moved(v8, off_kv), ks, vs, table, [ctx, 17, 128], splits)[3]
        assert _rel(b, a) < 2e-4                       # a bf16 step where the sum's last bits tip a rounding over


@pytest.mark.parametrize("ctx", [[5], [128, 129, 40], [1100, 16]])
def test_fp8_attention_of_short_contexts_in_many_splits(ops, ctx):
    """More splits than the contexts have groups of eight pages for: the empty ones are neutral partials, the merge gives what
    one split gives (the same weights, sums in another order)."""
    d, n_kv, gh, t = 256, 2, 6, len(ctx)
    g = torch.Generator(device=DEV).manual_seed(sum(ctx))
    mb = (max(ctx) + 15) // 16
    k8, v8 = ((torch.randn(t * mb + 1, n_kv, 16, d, generator=g, device=DEV) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for _ in range(2))
    ks, vs = (torch.rand(t * mb + 1, n_kv, 16, generator=g, device=DEV) * 0.02 + 0.01 for _ in range(2))
    table = (torch.randperm(t * mb, generator=g, device=DEV) + 1).int().view(t, mb)
    q = torch.randn(t, n_kv * gh, d, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(t, n_kv * gh * 2 * d, generator=g, device=DEV).to(torch.bfloat16)
    one = _fp8_decode(ops, q, k8, v8, ks, vs, table, ctx, 1, gate)[3]
    for splits in (2, 9, 64):
        po, pm, pl, out = _fp8_decode(ops, q, k8, v8, ks, vs, table, ctx, splits, gate)
        assert _rel(out, one) < 2e-4
        for i, n in enumerate(ctx):
            used = min(splits, ((n + 15) // 16 + 7) // 8)
            assert bool((pm[i, :, used:] == -float("inf")).all()) and float(pl[i, :, used:].abs().sum() + po[i, :, used:].abs().sum()) == 0


def test_explicit_split_count_is_taken_for_the_e4m3_pool(ops):
    """``attn_splits`` as set: with one split the rows are finished in one launch, without a merge."""
    from tilerl_b200.batch import Batch
    from tilerl_b200.config import get_config
    from tilerl_b200.kv import make_kv_pool
    from tilerl_b200.ops import native
    cfg = get_config("small-gpu")
    pool = make_kv_pool(cfg, 40, torch.device(DEV), fp8=True)
    batch = Batch.build([dict(tokens=[3], start=500, blocks=list(range(1, 36)), slot=1)], DEV)
    qkv = torch.randn(1, 2 * cfg.n_q_heads * 256 + 2 * cfg.n_kv_heads * 256, device=DEV).to(torch.bfloat16)
    lp = dict(q_norm=torch.ones(256, device=DEV), k_norm=torch.ones(256, device=DEV))
    outs = {}
    try:
        for splits, launches in ((0, 3), (1, 2), (2, 3)):
            ops.attn_splits = splits
            before = native.launch_count
            outs[splits] = ops.attention(qkv, lp, batch, pool, 0, cfg, cfg.n_q_heads, cfg.n_kv_heads).clone()
            assert native.launch_count - before == launches, splits
    finally:
        ops.attn_splits = 0
    assert _rel(outs[0], outs[1]) < 2e-4 and _rel(outs[2], outs[1]) < 2e-4


@pytest.mark.parametrize("tokens,n,k", [(3, 19001, 2080), (10, 19001, 2304), (20, 20000, 2048), (40, 19074, 2304), (128, 9999, 2080), (200, 19072, 2048),
                                        (900, 5120, 2304), (600, 6000, 1056)])
def test_gemm_stores_beside_the_next_tile(ops, tokens, n, k):
    """More tiles than CTAs and K long enough that a tile's stores run beside the next one's MMAs, in every tile width, with rows
    and columns that fill no tile: every epilogue, against the same kernel on one CTA per tile in chunks (split: one tile a
    CTA at a time)."""
    from tilerl_b200 import formats as F
    from tilerl_b200.ops import native
    from tilerl_b200.ops.gemm_tc import gemm_nvfp4
    g = torch.Generator().manual_seed(tokens + n)
    w = F.quantize_nvfp4(torch.randn(n, k, generator=g) * 0.02).to(DEV)
    x = torch.randn(tokens, k, generator=g).to(DEV, torch.bfloat16)
    want = torch.full((tokens, n), float("nan"), device=DEV)
    for a in range(0, n, 2560):                       # at most 20 tiles of rows: the form for few tiles
        part = F.NVFP4Tensor(w.wq[a:a + 2560].contiguous(), w.scale[a:a + 2560].contiguous(), w.tscale)
        y = torch.empty(tokens, part.wq.shape[0], device=DEV)
        gemm_nvfp4(ops, x[:60], part, y[:60], terms=2, epi=3, split=False)
        for b in range(60, tokens, 60):
            gemm_nvfp4(ops, x[b:b + 60], part, y[b:b + 60], terms=2, epi=3, split=False)
        want[:, a:a + 2560] = y
    for split in (False, True, None):
        f32, bf16 = torch.full((tokens, n), float("nan"), device=DEV), torch.full((tokens, n), float("nan"), dtype=torch.bfloat16, device=DEV)
        gemm_nvfp4(ops, x, w, f32, terms=2, epi=3, split=split)
        assert _rel(f32, want) < 1e-6
        gemm_nvfp4(ops, x, w, bf16, terms=2, split=split)
        assert _rel(bf16, want) < 2 ** -8
        r = torch.randn(tokens, n, generator=g).to(DEV, torch.bfloat16)
        acc = r.clone()
        gemm_nvfp4(ops, x, w, acc, terms=2, epi=1, residual=acc, split=split)
        assert _rel(acc, want.double() + r.double()) < 2 ** -8
        if n % 2 == 0:
            h = torch.full((tokens, n // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
            gemm_nvfp4(ops, x, w, h, terms=2, epi=2, split=split)
            assert _rel(h, torch.nn.functional.silu(want[:, 0::2].double()) * want[:, 1::2].double()) < 2 ** -8
    assert native.read_error()[0] == 0


@pytest.mark.parametrize("tokens,terms", [(1, 4), (8, 4), (9, 4), (16, 2), (17, 2), (32, 2), (33, 2), (64, 2), (65, 2), (96, 2), (97, 2), (31, 1), (193, 1), (500, 2)])
@pytest.mark.parametrize("n,k", [(264, 544), (1288, 4128), (5120, 6144), (19072, 288)])
def test_gemm_on_pairs_of_sms(ops, tokens, terms, n, k):
    """Every width of a tile with columns that fill it, one more and one less, rows that leave the second SM of a pair half or
    nothing, tiles that one pair and two or three go through, every epilogue, against one CTA alone (the one-SM kernel).  The
    same products in fp32, summed in another order."""
    from tilerl_b200 import formats as F
    from tilerl_b200.ops import native
    from tilerl_b200.ops.gemm_tc import gemm_nvfp4
    g = torch.Generator().manual_seed(tokens + n)
    w = F.quantize_nvfp4(torch.randn(n, k, generator=g) * 0.02).to(DEV)
    x = torch.randn(tokens, k, generator=g).to(DEV, torch.bfloat16)
    got, want = (torch.full((tokens, n), float("nan"), device=DEV) for _ in range(2))
    gemm_nvfp4(ops, x, w, want, terms=terms, epi=3, max_ctas=1, split=False)
    for _ in range(2):
        gemm_nvfp4(ops, x, w, got, terms=terms, epi=3)
        assert _rel(got, want) < 1e-6
    a, r = torch.full((tokens, n), float("nan"), dtype=torch.bfloat16, device=DEV), torch.randn(tokens, n, generator=g).to(DEV, torch.bfloat16)
    gemm_nvfp4(ops, x, w, a, terms=terms)
    assert _rel(a, want) < 2 ** -8
    acc = r.clone()
    gemm_nvfp4(ops, x, w, acc, terms=terms, epi=1, residual=acc)
    assert _rel(acc, want.double() + r.double()) < 2 ** -8
    h = torch.full((tokens, n // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
    gemm_nvfp4(ops, x, w, h, terms=terms, epi=2)
    assert _rel(h, torch.nn.functional.silu(want[:, 0::2].double()) * want[:, 1::2].double()) < 2 ** -8
    assert native.read_error()[0] == 0


@pytest.mark.parametrize("k", [1040, 18464, 24576, 28672])
@pytest.mark.parametrize("terms,swiglu", [(1, False), (2, False), (2, True), (4, False)])
def test_activation_quantiser_with_the_row_staged(ops, k, terms, swiglu):
    """Rows that the row kernel does not take: a block a row, the row staged in shared memory (128 rows and more), against blocks
    of slices (fewer rows): the same values, the same bytes."""
    from tilerl_b200.ops.gemm_tc import quant_act
    g = torch.Generator().manual_seed(k)
    width = 2 * k if swiglu else k
    room = torch.zeros(130, width + 8, dtype=torch.bfloat16, device=DEV)
    x = room[:, :width] if swiglu or k > 18432 else room[:, 4:4 + width]
    x.copy_(torch.randn(130, width, generator=g) * torch.exp(torch.randn(130, 1, generator=g)))
    nw = None if swiglu else (1.0 + 0.1 * torch.randn(k, generator=g)).to(DEV)
    nk = (k + 255) // 256

    def codes(rows):
        xq, sf, rs = quant_act(ops, rows, k, terms, norm_w=nw, eps=1e-6, swiglu_in=swiglu)
        c = torch.arange(rows.shape[0] * terms, device=DEV)
        return xq.clone(), rs.clone(), sf.view(-1, nk * 4, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(-1, nk * 16)[c].clone()
    many, few = codes(x), codes(x[:100])
    assert all(torch.equal(a[:100 * terms], b) for a, b in zip(many, few))
    assert int(many[2][:, k // 16:].sum()) == 0


@pytest.mark.parametrize("nk,nv,d,lens,keep,odd", [
    (8, 24, 128, [3, 1, 8, 17], True, 0), (8, 24, 128, [3, 1, 8, 17], True, 1), (2, 4, 64, [8, 1, 5], True, 0), (2, 4, 64, [8, 1, 5], True, 1),
    (16, 48, 64, [40, 1, 17, 5, 16, 33, 2], False, 0), (16, 48, 64, [40, 1, 17, 5, 16, 33, 2], False, 1)])
def test_delta_rule_scan_forms_equal_one_sequence_at_a_time(ops, nk, nv, d, lens, keep, odd):
    """Two columns a lane (many heads, kept states of short ones) and one (few heads, states at odd float addresses) do the same
    arithmetic on a column: the same states and rows as each sequence alone, bit for bit."""
    from tilerl_b200.ops import native as N
    c, t, b, planes = (2 * nk + nv) * d, sum(lens), len(lens), max(lens) + 1 if keep else 1
    g = torch.Generator().manual_seed(d + nv + odd)
    inp = torch.randn(t, c + nv * d + 2 * nv, generator=g).to(DEV, torch.bfloat16)
    conv = (torch.randn(c, 4, generator=g) * 0.3).to(DEV)
    dt, al, nw = torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV), torch.rand(d, generator=g).to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q0 = [sum(lens[:i]) for i in range(b)]
    first = torch.randn(b + 1, planes, nv, d, d, generator=torch.Generator(device=DEV).manual_seed(d), device=DEV) * 0.05

    def run(groups):
        states = torch.empty(first.numel() + 2, device=DEV)[odd:odd + first.numel()].view(first.shape)
        states.copy_(first)
        out = torch.zeros(t, nv * d, dtype=torch.bfloat16, device=DEV)
        ring = torch.zeros(b + 1, 16, c, dtype=torch.bfloat16, device=DEV)
        cur = torch.full((b + 1,), planes - 1, dtype=torch.int32, device=DEV)
        for seqs in groups:
            n = [lens[i] for i in seqs]
            a, m = q0[seqs[0]], sum(n)
            f = lambda *s: torch.full(s, float("nan"), device=DEV)
            sc = [f(m, nk, d), f(m, nk, d), f(m, nv, d), f(m, nv), f(m, nv), f(m, nv, d)]
            pos, seq = i32([j for x in n for j in range(x)]), i32([i for i, x in enumerate(n) for _ in range(x)])
            qs, ql, slots, kp = i32([sum(n[:i]) for i in range(len(n))]), i32(n), i32([i + 1 for i in seqs]), i32([1] * len(n))
            rows = inp[a:a + m]
            N.check(ops.lib.trl_gdn(rows.data_ptr(), rows.stride(0), conv.data_ptr(), dt.data_ptr(), al.data_ptr(), nw.data_ptr(),
                                    states.data_ptr(), cur.data_ptr(), ring.data_ptr(), pos.data_ptr(), seq.data_ptr(), qs.data_ptr(),
                                    ql.data_ptr(), slots.data_ptr(), kp.data_ptr() if keep else None, states.stride(0), states.stride(1),
                                    ring.stride(0), *(x.data_ptr() for x in sc), out[a:].data_ptr(), m, len(n), nk, nv, d, 4, planes,
                                    1e-6, N.stream()), "gdn")
        return states, out
    s1, o1 = run([list(range(b))])
    s2, o2 = run([[i] for i in range(b)])
    assert torch.equal(s1, s2) and torch.equal(o1, o2)
    assert not torch.equal(s1, first) and bool(torch.isfinite(o1.float()).all())


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_delta_rule_prep_does_not_read_past_a_short_window(ops, taps):
    """A row that is not finite is seen by the ``taps`` tokens whose window it is in, and by none after them, where tokens are
    taken in runs too."""
    from tilerl_b200.ops import native as N
    nk, nv, d, t = 2, 4, 128, 3000
    c = (2 * nk + nv) * d
    g = torch.Generator().manual_seed(taps)
    inp = torch.randn(t, c + nv * d + 2 * nv, generator=g).to(DEV, torch.bfloat16)
    bad = [0, 9, 1203, 2998]
    for i, r in enumerate(bad):
        inp[r, :c] = float("nan") if i % 2 else float("inf")
    conv = torch.rand(c, taps, generator=g).to(DEV) + 0.1
    dt, al, nw = torch.randn(nv, generator=g).to(DEV), torch.randn(nv, generator=g).to(DEV), torch.ones(d, device=DEV)
    ring = torch.zeros(2, 16, c, dtype=torch.bfloat16, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, seq, qs, ql, slots, cur = i32(list(range(t))), i32([0] * t), i32([0]), i32([t]), i32([1]), i32([0, 0])
    states = torch.zeros(2, 1, nv, d, d, device=DEV)
    f = lambda *s: torch.zeros(s, device=DEV)
    qn, kn, vc, gg, bb, o = f(t, nk, d), f(t, nk, d), f(t, nv, d), f(t, nv), f(t, nv), f(t, nv, d)
    out = torch.empty(t, nv * d, dtype=torch.bfloat16, device=DEV)
    N.check(ops.lib.trl_gdn(inp.data_ptr(), inp.stride(0), conv.data_ptr(), dt.data_ptr(), al.data_ptr(), nw.data_ptr(), states.data_ptr(),
                            cur.data_ptr(), ring.data_ptr(), pos.data_ptr(), seq.data_ptr(), qs.data_ptr(), ql.data_ptr(), slots.data_ptr(),
                            None, states.stride(0), states.stride(1), ring.stride(0), qn.data_ptr(), kn.data_ptr(), vc.data_ptr(), gg.data_ptr(),
                            bb.data_ptr(), o.data_ptr(), out.data_ptr(), t, 1, nk, nv, d, taps, 1, 1e-6, N.stream()), "gdn")
    seen = torch.zeros(t, dtype=torch.bool)
    for r in bad:
        seen[r:r + taps] = True
    assert torch.equal(torch.isfinite(vc).all(-1).all(-1).cpu(), ~seen)


@pytest.mark.parametrize("g_heads", [1, 3, 4])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("form", [-1, 0, 1, 2])
def test_prefill_attention_forms(ops, g_heads, fp8, form):
    """The forms for up to four heads a group: queries and histories at the edges of 16-row tiles and of tiles of 32 and 64 keys,
    sequences of one row (first in the grid) among longer ones, pool rows past a sequence's end that are NaN, against 64
    bits.  Weights and the result are bf16: 2^-9 each of what they carry, in the rms over rows whose keys are independent."""
    from tilerl_b200.ops import native as N
    import math
    n_kv, d = 2, 256
    n_q = n_kv * g_heads
    seqs = [(1, 0), (1, 700), (16, 0), (17, 15), (32, 0), (15, 49), (33, 31), (64, 1), (5, 123), (2, 127), (70, 500)]
    g = torch.Generator(device=DEV).manual_seed(g_heads * 2 + fp8)
    b, t = len(seqs), sum(n for n, _ in seqs)
    mb = max((n + h + 15) // 16 for n, h in seqs)
    pages = b * mb + 1
    k, v = (torch.randn(pages, n_kv, 16, d, generator=g, device=DEV) for _ in range(2))
    scales = [torch.ones(pages, n_kv, 16, device=DEV) for _ in range(2)]
    if fp8:
        scales = [torch.rand(pages, n_kv, 16, generator=g, device=DEV) * 0.02 + 0.01 for _ in range(2)]
        k, v = ((x * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for x in (k, v))
    else:
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
    kd, vd = (x.double() * s.double().unsqueeze(-1) for x, s in zip((k, v), scales))
    table = (torch.randperm(pages - 1, generator=g, device=DEV)[:b * mb] + 1).int().view(b, mb)
    for i, (n, h) in enumerate(seqs):                   # what lies past the sequence's end must not matter
        if (n + h) % 16:
            pg, r = int(table[i, (n + h) // 16]), (n + h) % 16
            for x in (k, v):
                x[pg].view(torch.uint8 if fp8 else torch.int16)[:, r:] = 0x7f if fp8 else 0x7fc0
            if fp8:
                scales[0][pg, :, r:] = scales[1][pg, :, r:] = float("nan")
    q = torch.randn(t, n_q, d, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(t, n_q * 2 * d, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((t, n_q * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(n for n, _ in seqs[:i]) for i in range(b)]
    qs, ql, pos = i32(starts), i32([n for n, _ in seqs]), i32([h + j for n, h in seqs for j in range(n)])
    tail = (qs.data_ptr(), ql.data_ptr(), pos.data_ptr(), out.data_ptr(), b, max(n for n, _ in seqs), n_q, n_kv, d,
            1 / math.sqrt(d), 1, form, N.stream())
    head = (q.data_ptr(), gate.data_ptr(), gate.stride(0), k.data_ptr(), v.data_ptr())
    if fp8:
        N.check(ops.lib.trl_attn_prefill_fp8_form(*head, scales[0].data_ptr(), scales[1].data_ptr(), table.data_ptr(), mb, *tail), "prefill_fp8")
    else:
        N.check(ops.lib.trl_attn_prefill_form(*head, table.data_ptr(), mb, pages, *tail), "prefill")
    for i, (n, h) in enumerate(seqs):
        blocks = table[i].long()
        kk, vv = (x[blocks].transpose(1, 2).reshape(-1, n_kv, d)[:n + h] for x in (kd, vd))
        rows = slice(starts[i], starts[i] + n)
        s = torch.einsum("thgd,nhd->thgn", q[rows].double().view(n, n_kv, g_heads, d), kk) / math.sqrt(d)
        s.masked_fill_((torch.arange(n + h, device=DEV) > (h + torch.arange(n, device=DEV)).view(n, 1)).view(n, 1, 1, -1), -math.inf)
        want = torch.einsum("thgn,nhd->thgd", torch.softmax(s, -1), vv).reshape(n, n_q, d)
        want = (want * torch.sigmoid(gate[rows].double().view(n, n_q, 2, d)[:, :, 1])).reshape(n, -1)
        assert _rel(out[rows], want) < 2 ** -7, (n, h, _rel(out[rows], want))
    assert N.read_error()[0] == 0


@pytest.mark.parametrize("lens", [[2], [16, 1], [17, 1, 15], [33, 2, 1, 48, 31, 100], [1] * 40 + [2]])
@pytest.mark.parametrize("nk,nv", [(2, 2), (1, 3)])
def test_delta_rule_chunk_kernel_with_and_without_preparing_groups(ops, lens, nk, nv):
    """The two forms of the chunk kernel take the same steps in the same order: the same bits in outputs, states and ring,
    over one chunk, a slot's reuse, rows that fill no chunk and sequences of one token."""
    from tilerl_b200.batch import Batch
    from tilerl_b200.config import GDN, ModelConfig
    from tilerl_b200.kv import GdnStatePool
    from tilerl_b200.ops import native as N
    d = 128
    cfg = ModelConfig("t", hidden=64, ffn=64, vocab=64, layer_types=(GDN,), n_q_heads=2, n_kv_heads=1, head_dim=64, rotary_dim=64,
                      rope_theta=1e6, gdn_k_heads=nk, gdn_v_heads=nv, gdn_head_dim=d)
    g = torch.Generator().manual_seed(sum(lens) + nv)
    lp = dict(conv=(torch.randn(cfg.gdn_conv_dim, 4, generator=g) * 0.3).to(DEV), dt_bias=torch.rand(nv, generator=g).to(DEV),
              a_log=torch.log(1 + 3 * torch.rand(nv, generator=g)).to(DEV), gdn_norm=(1 + 0.1 * torch.randn(d, generator=g)).to(DEV))
    batch = Batch.build([dict(tokens=[0] * n, start=7, blocks=list(range(1 + 8 * i, 9 + 8 * i)), slot=i + 1) for i, n in enumerate(lens)], DEV)
    inp = torch.randn(batch.n_tokens, cfg.gdn_in_rows, generator=g).to(DEV, torch.bfloat16)
    got = []
    try:
        for form in (0, 1, -1):
            pool = GdnStatePool(cfg, len(lens) + 1, DEV, planes=1, ring_dtype=torch.bfloat16)
            for i, x in enumerate((pool.states, pool.ring)):
                x.copy_(torch.randn(x.shape, generator=torch.Generator().manual_seed(i)))
            before = pool.states.clone()
            ops.gdn_form = form
            out = ops.gdn(inp, lp, batch, pool, 0, cfg, nk, nv).clone()
            got.append((out, pool.states.clone(), pool.ring.clone()))
    finally:
        ops.gdn_form = -1
    assert not torch.equal(got[0][1], before) and N.read_error()[0] == 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("m", [9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n,k", [(130, 72), (999, 1032), (15520, 5120), (40003, 640)])
def test_logits_of_many_rows(ops, m, n, k):
    """Every width of a tile, vocabularies that fill none of 128, K that fills no stage and one of many accumulators, more tiles than
    CTAs, against fp64 from the same normed rows: fp32 sums over K."""
    from tilerl_b200.ops import native
    g = torch.Generator().manual_seed(m + n)
    w, nw = (torch.randn(n, k, generator=g) * 0.02).to(DEV, torch.bfloat16), (1 + 0.1 * torch.randn(k, generator=g)).to(DEV)
    x = torch.randn(m, k, generator=g).to(DEV, torch.bfloat16)
    before = native.launch_count
    got = ops.lm_head(x, nw, w, 1e-6).clone()
    assert native.launch_count - before == 2 and got.dtype == torch.float32
    want = ops._rmsnorm(x, nw, 1e-6).double() @ w.double().t()
    assert _rel(got, want) < 2e-6
    # few rows and many: within the few roundings of the normed rows' bf16
    assert _rel(ops.lm_head(x[:4].contiguous(), nw, w, 1e-6), want[:4]) < 2 ** -8
    assert native.read_error()[0] == 0
