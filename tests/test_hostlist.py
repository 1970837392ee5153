"""Python lists into int32 staging memory (``csrc/hostlist.cu``): the same values as numpy's conversion, and everything that is
not a plain list of integers left to it."""
import numpy as np
import pytest
import torch

from tilerl_b200.batch import Batch
from tilerl_b200.graph import _Bucket, take_rows
from tilerl_b200.ops import native

needs_lib = pytest.mark.skipif(not native.loadable(), reason="the kernel library is not built")


def _fill(b, mb, seqs, general):
    bk = _Bucket(b, mb, torch.device("cpu"))
    bk.np[:] = 7
    keep = native.fill_decode
    if general:
        native.fill_decode = lambda *a: False
    try:
        bk.fill(seqs)
    finally:
        native.fill_decode = keep
    return bk.np.copy(), bk.h2d_bytes


@needs_lib
@pytest.mark.parametrize("b,n,mb", [(1, 1, 1), (4, 3, 9), (8, 8, 130), (2, 0, 4)])
def test_decode_inputs_equal_the_general_fill(b, n, mb):
    rng = np.random.RandomState(b + mb)
    seqs = []
    for i in range(n):
        nb = int(rng.randint(1, mb + 1))
        seqs.append(dict(tokens=[int(rng.randint(1 << 17))], start=int(rng.randint(16 * nb)), slot=i + 1, keep=True,
                         blocks=[int(v) for v in rng.randint(1, 1 << 20, nb)]))
    if seqs:
        assert native.fill_decode(seqs, np.empty(5 * b + b * mb, np.int32).ctypes.data, b, mb, 16)
    got, want = _fill(b, mb, seqs, False), _fill(b, mb, seqs, True)
    assert (got[0] == want[0]).all() and got[1] == want[1]


@needs_lib
def test_other_forms_go_the_general_way():
    plain = dict(tokens=[3], start=20, blocks=[4, 5], slot=1)
    room = np.empty(64, np.int32)
    ok = lambda s: native.fill_decode(s, room.ctypes.data, 2, 4, 16)
    assert ok([plain])
    for change in (dict(tokens=torch.tensor([3])), dict(tokens=[3, 4]), dict(start=np.int64(20)), dict(start=-1), dict(start=32), dict(blocks=(4, "x")),
                   dict(blocks=np.array([4, 5])), dict(blocks=[1] * 5), dict(blocks=[-1, 2]), dict(slot=None), dict(slot=True)):
        assert not ok([dict(plain, **change)]), change
    assert not ok([plain] * 3) and not ok((plain,)) and not ok([plain, 5])
    # what the general way takes it still takes, and what it refuses it still refuses
    a = _fill(2, 4, [dict(plain, blocks=np.array([4, 5]), start=np.int64(20))], False)[0]
    assert (a == _fill(2, 4, [plain], True)[0]).all()
    with pytest.raises(IndexError):
        _fill(2, 4, [dict(plain, start=40)], False)


@needs_lib
def test_list_conversion_checks_type_range_and_room():
    out = np.full(8, -7, np.int32)
    conv = lambda x, cap=8, lo=-(1 << 31), hi=1 << 31: native.list_i32(x, out.ctypes.data, cap, lo, hi)
    assert conv([5, -(1 << 31), (1 << 31) - 1]) == 3 and out[:4].tolist() == [5, -(1 << 31), (1 << 31) - 1, -7]
    assert conv((9, 8)) == 2 and out[:2].tolist() == [9, 8] and conv([]) == 0
    for bad in ([1.0], ["1"], [True], [1 << 31], [1 << 80], [None], np.arange(3), "12", {1: 2}):
        assert conv(bad) == -1, bad
    assert conv([1, 10], hi=10) == -1 and conv([-1], lo=0) == -1 and conv([1] * 9) == -2


@pytest.mark.parametrize("rows", [[0], [3], [1, 2, 3], [0, 2], [2, 1], [1, 1], [-1], [-2, -1], []])
def test_rows_that_are_a_range_equal_an_index(rows):
    x = torch.arange(20.0).view(5, 4)
    got = take_rows(x, rows)
    assert torch.equal(got, x[torch.tensor(rows, dtype=torch.long)])
    assert got.data_ptr() != x.data_ptr() or not len(rows)
    r = Batch.row_range(rows)
    assert r is None or list(range(5))[r] == rows


@pytest.mark.parametrize("rows", [[5], [4, 5], [0, 5], [7, 8], [-6], [-6, -5], [1, 9, 2]])
def test_rows_that_are_not_there_are_refused(rows):
    """As an index refuses them; a slice would return what there is of them."""
    x = torch.arange(20.0).view(5, 4)
    with pytest.raises(IndexError):
        take_rows(x, rows)


def _forward(lens, **kw):
    from tilerl_b200.factory import build_model, make_ops
    from tilerl_b200.kv import GdnStatePool, make_kv_pool
    ops = make_ops("cpu")
    model = build_model("tiny", "cpu", seed=0, ops=ops)
    cfg = model.cfg
    seqs = [dict(tokens=list(range(3 + i, 3 + i + n)), start=0, blocks=[i + 1], slot=i + 1) for i, n in enumerate(lens)]
    pool = make_kv_pool(cfg, len(lens) + 1, torch.device("cpu"), torch.float32)
    states = GdnStatePool(cfg, len(lens) + 1, "cpu", ring_dtype=torch.float32)
    return model.forward(Batch.build(seqs, "cpu"), ops, pool, states, **kw)


@pytest.mark.parametrize("lens", [[2, 0], [1, 1], [0, 2, 1], [3]])
def test_last_rows_are_each_sequences_last(lens):
    """As many tokens as sequences is not one token each: a sequence may bring none."""
    every = _forward(lens, last_only=False)
    last = [sum(lens[:i + 1]) - 1 for i in range(len(lens))]
    torch.testing.assert_close(_forward(lens), every[last], rtol=0, atol=1e-5)     # (the head of other row counts sums in another order)


@pytest.mark.parametrize("rows", [[4], [3, 4], [-5]])
def test_wanted_rows_that_are_not_there_are_refused(rows):
    with pytest.raises(IndexError):
        _forward([1, 3], rows=rows)


def test_library_of_another_interpreter_is_not_current(monkeypatch):
    """The host sources read the interpreter's lists in place: its version and headers are part of what was built."""
    import os
    import sys
    from tilerl_b200 import build
    src = os.path.join(build.CSRC, "hostlist.cu")
    here = build._stamp(src)
    assert here == build._stamp(src)
    with monkeypatch.context() as m:
        m.setattr(sys, "version_info", (3, 99, 0, "final", 0))
        assert build._stamp(src) != here
    with monkeypatch.context() as m:
        m.setattr(build, "_include", lambda: "/nowhere")
        assert build._stamp(src) != here


@pytest.mark.parametrize("rows,n_kv,pages,want", [(1, 4, 1, 1), (1, 4, 8, 1), (1, 4, 9, 2), (1, 4, 4000, 64), (12, 4, 400, 25), (12, 4, 24, 3), (32, 4, 400, 10),
                                                  (500, 8, 400, 1), (0, 4, 400, 50)])
def test_splits_of_attention_over_an_e4m3_pool(rows, n_kv, pages, want):
    """Four splits a block slot, none of them under eight pages, 64 at most."""
    from tilerl_b200.ops.cuda import fp8_splits
    assert fp8_splits(148, rows, n_kv, pages) == want


def test_captured_ticks_choose_their_splits_once():
    """One rule for the runners: the e4m3 one for pools of head dim 256, the bf16 kernel's for others."""
    from types import SimpleNamespace as NS
    from tilerl_b200.graph import _splits
    runner = lambda fp8, dim, mb: NS(ops=NS(sms=148), model=NS(dims=NS(n_kv=4), cfg=NS(head_dim=dim)), kv=NS(fp8=fp8), max_blocks=mb)
    assert _splits(runner(False, 256, 400), 12, 64) == 3 and _splits(runner(True, 128, 400), 12, 64) == 3
    assert _splits(runner(True, 256, 400), 12, 64) == 25 and _splits(runner(True, 256, 24), 12, 64) == 3
    assert _splits(runner(False, 256, 400), 1, 32) == 32


@pytest.mark.parametrize("q,kv,n_kv,g,want", [
    ([2000], [2000], 2, 4, 0), ([2000], [2000], 4, 4, 2), ([512], [512], 4, 3, 0), ([512], [512], 8, 4, 2), ([100] * 8, [100] * 8, 4, 1, 2),
    ([2048], [8192], 2, 4, 1), ([1000], [4000], 2, 4, 0), ([1000], [4000], 4, 4, 1), ([300], [3300], 8, 2, 1), ([64], [8064], 8, 4, 0),
    ([1] * 12 + [64], [4001] * 12 + [64], 8, 4, 0), ([2048], [8192], 4, 6, 0), ([1], [1], 1, 1, 0)])
def test_form_of_prefill_attention(q, kv, n_kv, g, want):
    """One block an SM while the blocks are through with the longest one; else two, by the length of the contexts."""
    from tilerl_b200.ops.cuda import prefill_form
    assert prefill_form(q, kv, n_kv, g, 148) == want
