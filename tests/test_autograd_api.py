"""Differentiable front end, CPU part: the torch.library operators exist, carry fake (meta)
implementations with the right shapes, and refuse CPU tensors (there is no CPU fallback)."""
from __future__ import annotations

import pytest
import torch

from min_fa3_demo_b200 import autograd as ag


def test_operators_are_registered_with_schemas():
    assert str(torch.ops.b200attn.fwd.default._schema).startswith("b200attn::fwd(Tensor q, Tensor k, Tensor v, bool is_causal)")
    assert "bool deterministic" in str(torch.ops.b200attn.bwd.default._schema)


def test_fake_implementations_give_shapes_and_dtypes():
    q = torch.empty(2, 384, 8, 128, dtype=torch.bfloat16, device="meta")
    k = torch.empty(2, 512, 2, 128, dtype=torch.bfloat16, device="meta")
    out, lse = torch.ops.b200attn.fwd(q, k, k, True)
    assert out.shape == q.shape and out.dtype == torch.bfloat16
    assert lse.shape == (2, 8, 384) and lse.dtype == torch.float32
    dq, dk, dv = torch.ops.b200attn.bwd(out, q, k, k, out, lse, True, False)
    assert dq.shape == q.shape and dk.shape == k.shape and dv.shape == k.shape


def test_cpu_tensors_are_rejected():
    q = torch.zeros(1, 128, 2, 128, dtype=torch.bfloat16, requires_grad=True)
    with pytest.raises(RuntimeError, match="no CPU implementation"):
        ag.attention(q, q, q, True)
    cu = torch.tensor([0, 128], dtype=torch.int32)
    with pytest.raises(RuntimeError, match="no CPU implementation"):
        ag.attention_varlen(q[0], q[0], q[0], cu, cu, 128, 128, True)


def _stand_ins(monkeypatch):
    """Lets CPU tensors pass for CUDA ones, with cheap functions in the kernels' place; records direct calls."""
    direct = []
    monkeypatch.setattr(ag, "_require_cuda", lambda t, name: None)
    monkeypatch.setattr(ag, "_plain_tensors", lambda tensors: all(type(t) in ag._PLAIN_TYPES for t in tensors))
    monkeypatch.setattr(ag._op, "forward", lambda q, k, v, causal, return_lse: (q * 2, q.new_zeros(
        (q.size(0), q.size(2), q.size(1)), dtype=torch.float32)))
    monkeypatch.setattr(ag._op, "backward", lambda dout, q, k, v, out, lse, causal, deterministic: (
        dout * 2, torch.zeros_like(k), torch.zeros_like(v)))
    for name in ("_fwd", "_bwd"):
        def body(*args, _body=getattr(ag, name), _name=name):
            direct.append(_name)
            return _body(*args)
        monkeypatch.setattr(ag, name, body)
    return direct


def test_differentiating_a_gradient_is_refused(monkeypatch):
    direct = _stand_ins(monkeypatch)
    q, k, v = (torch.ones(1, 4, 2, 128, dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    out = ag.attention(q, k, v, True)
    out.sum().backward()
    assert direct == ["_fwd", "_bwd"]                   # an ordinary step passes the operators by
    assert torch.equal(q.grad, torch.full_like(q, 2))
    out = ag.attention(q, k, v, True)
    grad, = torch.autograd.grad(out.sum(), q, create_graph=True)
    with pytest.raises(RuntimeError, match="no autograd formula"):
        (out.sum() + grad.square().sum()).backward()


def test_lookers_on_still_see_the_operators(monkeypatch):
    # Meta and fake tensors, tracers, dispatch and function modes and profilers see the operators; only plain CUDA calls
    # pass them by.
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    meta = torch.empty(1, 128, 4, 128, dtype=torch.bfloat16, device="meta", requires_grad=True)
    out = ag.attention(meta, meta, meta, True)
    assert out.device.type == "meta" and out.shape == meta.shape
    assert torch.autograd.grad(out, meta, torch.empty_like(out))[0].shape == meta.shape
    with FakeTensorMode():
        q = torch.empty(1, 128, 4, 128, dtype=torch.bfloat16, device="meta")
        assert not ag._plain_call(q)
        graph = make_fx(lambda t: ag.attention(t, t, t, True))(q).graph
    assert any(n.target is torch.ops.b200attn.fwd.default for n in graph.nodes)

    direct = _stand_ins(monkeypatch)
    seen = []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    def step():
        q = torch.ones(1, 4, 2, 128, dtype=torch.bfloat16, requires_grad=True)
        ag.attention(q, q, q, True).sum().backward()
        assert torch.equal(q.grad, torch.full_like(q, 2))

    with Dispatch():
        step()
    assert torch.ops.b200attn.fwd.default in seen and torch.ops.b200attn.bwd.default in seen
    seen.clear()
    with Function():
        step()
    assert torch.ops.b200attn.fwd in seen
    assert direct in ([], ["_bwd"])                        # backward() runs inside the mode's handler, without the mode
    direct.clear()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        step()
    assert {"b200attn::fwd", "b200attn::bwd"} <= {e.key for e in prof.key_averages()}
    graph = make_fx(lambda t: ag.attention(t, t, t, True))(torch.ones(1, 4, 2, 128, dtype=torch.bfloat16)).graph
    assert any(n.target is torch.ops.b200attn.fwd.default for n in graph.nodes)
    monkeypatch.setattr(ag, "_LOOKER_CHECKS", None)       # a torch without the checks
    step()
    assert direct == []


@pytest.mark.parametrize("owner,name", [("torch.utils._python_dispatch", "_get_current_dispatch_mode"),
                                        ("torch._C._functorch", "peek_interpreter_stack"),
                                        ("torch._C", "_len_torch_function_stack"),
                                        ("torch._C._autograd", "_profiler_enabled")])
def test_a_torch_without_a_check_is_found_out(monkeypatch, owner, name):
    import importlib
    assert ag._looker_checks() is not None
    monkeypatch.delattr(importlib.import_module(owner), name)
    assert ag._looker_checks() is None
