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
# Refusals of calls that are in order but for one thing.  The tensors are fakes on "cuda:0": sizes, types and strides, no
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


def dense_arguments(backward):
    a = dict(q=on_cuda(2, 128, 4, 128), k=on_cuda(2, 128, 2, 128), v=on_cuda(2, 128, 2, 128), is_causal=True)
    if backward:
        a.update(dout=on_cuda(2, 128, 4, 128), out=on_cuda(2, 128, 4, 128), softmax_lse=on_cuda(2, 4, 128, dtype=torch.float32))
    return a


def arguments(entry):
    if entry in ("forward", "backward"):
        return dense_arguments(entry == "backward")
    a = packed_arguments()
    if entry == "backward_varlen":
        del a["cu_seqlens_q_host"], a["cu_seqlens_k_host"]
        a.update(dout=on_cuda(256, 4, 128), out=on_cuda(256, 4, 128), softmax_lse=on_cuda(4, 256, dtype=torch.float32))
    return a


ENTRIES = ["forward", "backward", "forward_varlen", "backward_varlen"]
DENSE, PACKED = ("forward", "backward"), ("forward_varlen", "backward_varlen")
BACKWARD, FORWARD = ("backward", "backward_varlen"), ("forward", "forward_varlen")


@pytest.mark.parametrize("entry", ENTRIES)
def test_good_calls_are_accepted(entry, host_checks_only, monkeypatch):
    calls = [arguments(entry)]
    if entry == "forward_varlen":                                         # rows of v that k has no counterpart for
        calls.append(dict(calls[0], v=on_cuda(300, 2, 128)))
    monkeypatch.setattr(torch, "empty", lambda *args, **kwargs: None)     # lse, on a device that may not be there
    for a in calls:
        with pytest.raises(Launched):
            getattr(op, entry)(**a)


def _with_size(name, dim, size):
    def change(a):
        shape = list(a[name].shape)
        shape[dim] = size
        a[name] = on_cuda(*shape, dtype=a[name].dtype)
    return change


def _all(*changes):
    def change(a):
        for c in changes:
            c(a)
    return change


def _with_sizes(names, dim, size):
    return _all(*(_with_size(name, dim, size) for name in names))


def _with_dtype(name, dtype):
    def change(a):
        a[name] = on_cuda(*a[name].shape, dtype=dtype)
    return change


def _strided(name):
    def change(a):
        shape = a[name].shape
        with FakeTensorMode():
            a[name] = torch.empty((*shape[:-1], 2 * shape[-1]), dtype=a[name].dtype, device="cuda:0")[..., ::2]
        assert a[name].shape == shape and not a[name].is_contiguous()
    return change


def _on_device(name, device):
    def change(a):
        a[name] = on_cuda(*a[name].shape, dtype=a[name].dtype, device=device)
    return change


def _without_first_dim(name):
    def change(a):
        a[name] = on_cuda(*a[name].shape[1:], dtype=a[name].dtype)
    return change


def _set(**values):
    return lambda a: a.update(values)


def _host(name, *values, dtype=torch.int32):
    return _set(**{name: torch.tensor(values, dtype=dtype)})


def bad_calls():
    cases = []

    def add(label, entries, change, message):
        cases.extend(pytest.param(e, change, message, id=f"{e}-{label}") for e in entries)

    for name in ("q", "k", "v", "out", "dout"):
        entries = BACKWARD if name in ("out", "dout") else ENTRIES
        add(f"{name} fp16", entries, _with_dtype(name, torch.float16), f"{name} must have dtype torch.bfloat16")
        add(f"{name} rank", entries, _without_first_dim(name), f"{name} must have ")
        add(f"{name} width", entries, _with_size(name, -1, 64), f"{name} must have head_dim D=128")
        add(f"{name} strides", entries, _strided(name), f"{name} must be contiguous")
        add(f"{name} cpu", entries, _on_device(name, "cpu"), f"{name} must be a CUDA tensor")
        if name != "q":
            add(f"{name} device", entries, _on_device(name, "cuda:1"), "must be on the same CUDA device")
    for name in ("out", "dout"):
        for label, dim, size in (("rows", 0, 1), ("heads", -2, 2)):
            add(f"{name} {label}", BACKWARD, _with_size(name, dim, size), f"{name} must have the same shape as q")
        add(f"{name} length", ("backward",), _with_size(name, 1, 127), f"{name} must have the same shape as q")
    for name in ("k", "v"):
        add(f"{name} batch", DENSE, _with_size(name, 0, 1), "must have the same (batch size )?B")
        add(f"{name} tokens", DENSE, _with_size(name, 1, 127), "k and v must have the same (sequence length )?Sk")
        add(f"{name} heads", ENTRIES, _with_size(name, -2, 1), "k and v must have the same KV head count")
        add(f"{name} total", ("backward_varlen",), _with_size(name, 0, 255), "k and v must have the same total_k")
    add("group", FORWARD, _with_size("q", -2, 3), "qhead % kvhead == 0")
    add("lse fp64", BACKWARD, _with_dtype("softmax_lse", torch.float64), "softmax_lse must have dtype torch.float32")
    add("lse strides", BACKWARD, _strided("softmax_lse"), "softmax_lse must be contiguous")
    add("lse cpu", BACKWARD, _on_device("softmax_lse", "cpu"), "softmax_lse must be a CUDA tensor")
    add("lse device", BACKWARD, _on_device("softmax_lse", "cuda:1"), "softmax_lse must be on the same CUDA device")
    for dim in (0, 1):
        add(f"lse dim {dim}", BACKWARD, _with_size("softmax_lse", dim, 1), "softmax_lse must have shape")
    add("lse length", ("backward",), _with_size("softmax_lse", 2, 127), "softmax_lse must have shape")
    for name in ("cu_seqlens_q", "cu_seqlens_k"):
        add(f"{name} int64", PACKED, _with_dtype(name, torch.int64), f"{name} must have dtype torch.int32")
        add(f"{name} rank", PACKED, _set(**{name: on_cuda(1, 3, dtype=torch.int32)}), f"{name} must (be 1D|have shape)")
        add(f"{name} strides", PACKED, _strided(name), f"{name} must be contiguous")
        add(f"{name} cpu", PACKED, _on_device(name, "cpu"), f"{name} must be a CUDA tensor")
        add(f"{name} device", PACKED, _on_device(name, "cuda:1"), "must be on the same CUDA device")
        add(f"{name} length", ("backward_varlen",), _with_size(name, 0, 4), "must have the same B")
        add(f"{name} length", ("forward_varlen",), _with_size(name, 0, 4), "same length as its CUDA cu_seqlens")
        add(f"{name} one entry", PACKED, _with_size(name, 0, 1), f"{name} must have shape")
        host = f"{name}_host"
        add(f"{host} int64", ("forward_varlen",), _host(host, 0, 100, 256, dtype=torch.int64), f"{host} must have dtype torch.int32")
        add(f"{host} length", ("forward_varlen",), _host(host, 0, 256), f"{host} must have the same length")
        add(f"{host} rank", ("forward_varlen",), _set(**{host: torch.zeros(1, 3, dtype=torch.int32)}), f"{host} must be 1D")
        add(f"{host} strides", ("forward_varlen",), _set(**{host: torch.zeros(6, dtype=torch.int32)[::2]}),
            f"{host} must be contiguous")
        add(f"{host} cuda", ("forward_varlen",), _set(**{host: on_cuda(3, dtype=torch.int32)}), f"{host} must be a CPU tensor")
        add(f"{host} first", ("forward_varlen",), _host(host, 1, 100, 256), f"{host} must start with 0")
        add(f"{host} last", ("forward_varlen",), _host(host, 0, 100, 255), rf"{host}\[-1\] must equal")
    for name in ("max_seqlen_q", "max_seqlen_k"):
        add(f"{name} 0", PACKED, _set(**{name: 0}), "must be positive")
        add(f"{name} 2^31", PACKED, _set(**{name: 2**31}), "must fit (in )?int32")
    # Sizes that several arguments have in common.
    rows_q, rows_k = ("q", "out", "dout"), ("k", "v")
    empty = "B, Sq, and Sk must be positive"
    add("batch", ("forward",), _with_sizes(rows_k, 0, 3), "must have the same batch size B")
    add("batch", ("backward",), _with_sizes(rows_k, 0, 3), "must have the same B")
    add("no batch", ("backward",), _with_sizes((*rows_q, *rows_k, "softmax_lse"), 0, 0), empty)
    add("no rows", ("backward",), _all(_with_sizes(rows_q, 1, 0), _with_size("softmax_lse", 2, 0)), empty)
    add("no keys", ("backward",), _with_sizes(rows_k, 1, 0), empty)
    add("no rows", ("backward_varlen",), _all(_with_sizes(rows_q, 0, 0), _with_size("softmax_lse", 1, 0)),
        "total_q and total_k must be positive")
    add("no keys", ("backward_varlen",), _with_sizes(rows_k, 0, 0), "total_q and total_k must be positive")
    add("group", ("backward",), _all(_with_sizes(rows_q, 2, 3), _with_size("softmax_lse", 1, 3)), "qhead must be divisible by kvhead")
    add("group", ("backward_varlen",), _all(_with_sizes(rows_q, 1, 3), _with_size("softmax_lse", 0, 3)),
        "qhead must be divisible by kvhead")
    return cases


@pytest.mark.parametrize("entry,change,message", bad_calls())
def test_a_bad_call_is_refused_on_the_host(entry, change, message, host_checks_only):
    a = arguments(entry)
    change(a)
    with pytest.raises(RuntimeError, match=message):
        getattr(op, entry)(**a)


@pytest.mark.parametrize("entry", DENSE + PACKED)
def test_another_compute_capability_is_refused(entry, monkeypatch):
    monkeypatch.setattr(op, "_SM100", set())
    monkeypatch.setattr(torch.cuda, "get_device_capability", lambda device=None: (9, 0))
    for _ in range(2):                      # a refusal is not remembered as a pass
        with pytest.raises(RuntimeError, match="only supports Blackwell SM100. Current device capability is 9.0"):
            getattr(op, entry)(**arguments(entry))
