"""Host side of the CUDA ops, on the CPU: what goes to which entry point."""
import types

import pytest
import torch

from tilerl_b200.ops import cuda


def _head(x, w):
    """``CudaOps.lm_head`` on tensors of the CPU, entry points as stand-ins: what was called."""
    calls = []
    ws = cuda.Workspace("cpu")
    lib = types.SimpleNamespace(trl_head_bf16=lambda *a: calls.append("head") or 0)
    ops = types.SimpleNamespace(settle=lambda: None, ws=ws, lib=lib, _f32=lambda t: t, use_tc_gemm=False,
                                _rmsnorm=lambda x, w, eps, name=None: x, _gemv=lambda x, w, *a, **k: calls.append("rows"))
    cuda.CudaOps.lm_head(ops, x, torch.ones(x.shape[1]), w, 1e-6)
    return calls


def test_head_of_another_width_is_not_read_past_its_rows(monkeypatch):
    """The tensor-core head takes its number of columns from the weights: activations of another width are refused by the product
    that they go to, as for rows that it does not take."""
    monkeypatch.setattr(cuda.N, "stream", lambda: 0)
    w = torch.zeros(40, 64, dtype=torch.bfloat16)
    x = lambda m, k: torch.zeros(m, k, dtype=torch.bfloat16)
    assert _head(x(32, 64), w) == ["head"] and _head(x(8, 64), w) == ["rows"] and _head(x(65, 64), w) == []
    with pytest.raises(RuntimeError):
        _head(x(32, 48), w)
    assert _head(x(12, 48), w) == ["rows"]


def test_workspace_takes_shapes_of_every_form(monkeypatch):
    """Lists as well as tuples; a buffer that was replaced gives no old view."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    ws = cuda.Workspace("cpu")
    a = ws.get("a", [2, 3], torch.float32)
    assert a.shape == (2, 3) and ws.get("a", (2, 3), torch.float32) is a and ws.get("a", torch.Size([2, 3]), torch.float32) is a
    b = ws.get("a", (4, 3), torch.float32)
    assert ws.get("a", (2, 3), torch.float32).data_ptr() == b.data_ptr() != a.data_ptr() and ws.retired[0].data_ptr() == a.data_ptr()


def test_gemm_on_one_sm_as_asked_for(monkeypatch):
    """``TRL_GEMM_PAIR=0`` keeps every layout off the kernel on pairs; without it nothing changes."""
    from tilerl_b200.ops import gemm_tc
    from tilerl_b200.ops.gemm_tc import _want_split
    for pair, forms in ((True, {None: -1, False: 0, True: 1}), (False, {None: -2, False: 2, True: 1})):
        monkeypatch.setattr(gemm_tc, "_PAIR", pair)
        for split, want in forms.items():
            assert _want_split(split) == want
    monkeypatch.setenv("TRL_SPLITK", "0")
    assert _want_split() == 2 and _want_split(True) == 1
    monkeypatch.setattr(gemm_tc, "_PAIR", True)
    assert _want_split() == 0
