"""Host-side behaviour of the min_fa3_op mirror that needs no GPU: launch-grid override
resolution and argument validation order/messages (reference: bindings.cpp:32-62, 240-331;
include/min_fa3_launch_override.h:16-52; csrc/backward/min_fa3_bwd_bindings.cu:156-190)."""
from __future__ import annotations

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import min_fa3_op
from min_fa3_demo_b200 import min_fa3_op as op, ring


def test_root_module_reexports_api():
    for name in ("forward", "forward_varlen", "backward", "backward_varlen"):
        assert getattr(min_fa3_op, name) is getattr(op, name)


def test_resolve_launch_grid_shape():
    assert op._debug_resolve_launch_grid_shape(132) == (132, 1, 1)
    assert op._debug_resolve_launch_grid_shape(132, manual_block_count=7) == (7, 1, 1)
    with pytest.raises(ValueError, match="only supports the current 1D persistent grid"):
        op._debug_resolve_launch_grid_shape(4, 2, 1, manual_block_count=7)
    with pytest.raises(ValueError, match="must be greater than 0"):
        op._debug_resolve_launch_grid_shape(4, manual_block_count=0)
    with pytest.raises(ValueError, match="32-bit grid.x"):
        op._debug_resolve_launch_grid_shape(4, manual_block_count=2**31)
    with pytest.raises(RuntimeError, match="auto_grid_x must be between 0"):
        op._debug_resolve_launch_grid_shape(-1)


def _bshd(b=1, s=8, h=2, d=128, dtype=torch.bfloat16):
    return torch.zeros(b, s, h, d, dtype=dtype)


def test_forward_rejects_bad_inputs_before_any_launch():
    q, k, v = _bshd(), _bshd(), _bshd()
    with pytest.raises(ValueError, match="manual_block_count must be greater than 0"):
        op.forward(q, k, v, True, manual_block_count=-3)
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        op.forward(q, k, v, True)


def test_backward_rejects_bad_inputs_before_any_launch():
    q = _bshd()
    lse = torch.zeros(1, 2, 8)
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        op.backward(q, q, q, q, q, lse, True)


@pytest.mark.parametrize("bad,msg", [
    (dict(dtype=torch.float16), "must have dtype torch.bfloat16"),
    (dict(d=64), "must have head_dim D=128"),
])
def test_check_helpers_messages(bad, msg):
    t = _bshd(**bad)
    # the device check comes first in the reference; emulate a CUDA tensor by checking the
    # remaining rules directly
    with pytest.raises(RuntimeError, match=msg):
        op._check(t.dtype == torch.bfloat16, "q must have dtype torch.bfloat16")
        op._check(t.size(3) == 128, "q must have head_dim D=128")


def test_varlen_host_checks():
    cu_dev_like = torch.tensor([0, 4, 8], dtype=torch.int32)
    with pytest.raises(RuntimeError, match="must have dtype torch.int32"):
        op._check_cu_seqlens_host(torch.tensor([0, 4, 8]), cu_dev_like, "cu_seqlens_q_host")
    with pytest.raises(RuntimeError, match="same length as its CUDA cu_seqlens tensor"):
        op._check_cu_seqlens_host(torch.tensor([0, 8], dtype=torch.int32), cu_dev_like,
                                  "cu_seqlens_q_host")
    op._check_cu_seqlens_host(cu_dev_like.clone(), cu_dev_like, "cu_seqlens_q_host")


# ---------------------------------------------------------------------------------------
# Refusals of calls that are in order but for one argument.  The tensors are fakes on "cuda:0": sizes, types and strides, no
# memory, so that nothing can be launched, here or on a GPU.
# ---------------------------------------------------------------------------------------
class Launched(Exception):
    pass


def on_cuda(*shape, dtype=torch.bfloat16, device="cuda:0"):
    with FakeTensorMode():
        return torch.empty(shape, dtype=dtype, device=device)


@pytest.fixture(params=["device known", "device new"])
def host_checks_only(request, monkeypatch):
    """Both ways through the checks: the one expression first, and, on a device not seen before, the list at once."""
    def launched(*args, **kwargs):
        raise Launched

    monkeypatch.setattr(op, "_SM100", {0} if request.param == "device known" else set())
    monkeypatch.setattr(torch.cuda, "get_device_capability", lambda device=None: (10, 0))
    for name in ("_call_fwd", "_call_bwd"):
        monkeypatch.setattr(op, name, launched)


def packed_arguments():
    cu = torch.tensor([0, 100, 256], dtype=torch.int32)
    return dict(q=on_cuda(256, 4, 128), k=on_cuda(256, 2, 128), v=on_cuda(256, 2, 128),
                cu_seqlens_q=on_cuda(3, dtype=torch.int32), cu_seqlens_k=on_cuda(3, dtype=torch.int32), max_seqlen_q=156,
                max_seqlen_k=156, is_causal=True, cu_seqlens_q_host=cu, cu_seqlens_k_host=cu)


def test_packed_forward_refuses_fewer_values_than_keys(host_checks_only):
    with pytest.raises(RuntimeError, match="v must not have fewer tokens than k. Got 255 vs 256"):
        op.forward_varlen(**dict(packed_arguments(), v=on_cuda(255, 2, 128)))


def test_context_parallel_forward_refuses_fewer_values_than_keys():
    a = packed_arguments()
    with pytest.raises(RuntimeError, match="v must not have fewer tokens than k. Got 255 vs 256"):
        ring._common_checks(a["q"], a["k"], on_cuda(255, 2, 128), a["cu_seqlens_q"], a["cu_seqlens_k"], a["cu_seqlens_q_host"],
                            a["cu_seqlens_k_host"], 156, 156, 1, 0)
