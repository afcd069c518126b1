"""The forward and backward launches can be captured into a CUDA graph and replayed: the
library allocates nothing, every launch and memset goes to the caller's stream, and the work
scheduler's counters are reset on every replay, by a captured memset node or by a kernel that
runs anyway (the planner, the backward's preprocess, the forward itself).  Replays must reproduce
the eager results (out, dk, dv bit for bit; dq too in deterministic mode).  The forward's kernels
and the planner start while the kernel before them ends, so what they wait for is tested here as
well: in a graph, and across streams."""
from __future__ import annotations

import pytest
import torch

import min_fa3_op
from gpu_util import assert_cut, make_bshd, make_varlen

pytestmark = pytest.mark.gpu


def test_forward_backward_capture_and_replay():
    q, k, v, dout = make_bshd(55, 2, 1024, 8, 2)
    qc, kc, vc, dc = q.cuda(), k.cuda(), v.cuda(), dout.cuda()
    # Eager run first: also performs the one-time per-device kernel configuration.
    out_e, lse_e = min_fa3_op.forward(qc, kc, vc, True, return_lse=True)
    dq_e, dk_e, dv_e = min_fa3_op.backward(dc, qc, kc, vc, out_e, lse_e, True, deterministic=True)
    torch.cuda.synchronize()

    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            out_g, lse_g = min_fa3_op.forward(qc, kc, vc, True, return_lse=True)
            dq_g, dk_g, dv_g = min_fa3_op.backward(dc, qc, kc, vc, out_g, lse_g, True, deterministic=True)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        for t in (out_g, dq_g, dk_g, dv_g):
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out_g, out_e) and torch.equal(lse_g, lse_e)
        assert torch.equal(dq_g, dq_e) and torch.equal(dk_g, dk_e) and torch.equal(dv_g, dv_e)

    # New inputs through the same graph: copy into the captured buffers and replay.
    q2, k2, v2, d2 = make_bshd(56, 2, 1024, 8, 2)
    qc.copy_(q2.cuda()); kc.copy_(k2.cuda()); vc.copy_(v2.cuda()); dc.copy_(d2.cuda())
    graph.replay()
    torch.cuda.synchronize()
    out_n, lse_n = min_fa3_op.forward(qc, kc, vc, True, return_lse=True)
    dq_n, dk_n, dv_n = min_fa3_op.backward(dc, qc, kc, vc, out_n, lse_n, True, deterministic=True)
    torch.cuda.synchronize()
    assert torch.equal(out_g, out_n) and torch.equal(dq_g, dq_n) and torch.equal(dk_g, dk_n) and torch.equal(dv_g, dv_n)


def test_cut_calls_capture_and_replay():
    # The forward is cut along its keys, the backward along its steps; their partial results lie in the graph's pool, in
    # buffers that are free again when each call has been captured.
    assert_cut(True, "fwd", 1, 700, 6000, 8, 2, True)
    assert_cut(True, "bwd", 1, 2000, 2000, 8, 2, True)
    q, k, v, _ = (t.cuda() for t in make_bshd(57, 1, 700, 8, 2, sk=6000))
    q2, k2, v2, dout = (t.cuda() for t in make_bshd(58, 1, 2000, 8, 2))

    def run():
        out, lse = min_fa3_op.forward(q, k, v, True, return_lse=True)
        out2, lse2 = min_fa3_op.forward(q2, k2, v2, True, return_lse=True)
        return (out, lse, out2, lse2, *min_fa3_op.backward(dout, q2, k2, v2, out2, lse2, True, deterministic=True))

    eager = run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run()
    for _ in range(3):
        for t in captured:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(captured, eager))


def _packed(q, k, v, cu, cu_host, longest):
    return min_fa3_op.forward_varlen(q, k, v, cu, cu, longest, longest, True, cu_seqlens_q_host=cu_host, cu_seqlens_k_host=cu_host,
                                     return_lse=True)


def test_packed_calls_capture_and_replay():
    # Planner -> forward -> planner -> forward of another's output -> backward with its planner; a dense call without a counter
    # between them.  Replays take the documents from the captured cu_seqlens, which a kernel of the graph writes right before.
    lengths, other = [300, 77, 512, 1, 134], [1, 640, 20, 300, 63]
    q, k, v, dout, cu_host = make_varlen(61, lengths, 8, 2)
    cu_other_host = make_varlen(61, other, 8, 2)[4]
    q, k, v, dout = (t.cuda() for t in (q, k, v, dout))
    source, cu = cu_host.cuda(), torch.zeros_like(cu_host, device="cuda")
    dense = [t.cuda() for t in make_bshd(62, 2, 200, 4, 4)[:3]]

    def run(host, longest):
        torch.add(source, 0, out=cu)
        out, lse = _packed(q, k, v, cu, host, longest)
        out_dense = min_fa3_op.forward(*dense, True)
        out2, lse2 = _packed(out, k, v, cu, host, longest)
        return (out, lse, out_dense, out2, lse2,
                *min_fa3_op.backward_varlen(dout, out, k, v, out2, lse2, cu, cu, longest, longest, True, deterministic=True))

    eager = run(cu_host, 640)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run(cu_host, 640)
    for _ in range(3):
        for t in captured:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(captured, eager))
    source.copy_(cu_other_host.cuda())
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(captured, run(cu_other_host, 640)))


@pytest.mark.parametrize("b,s", [(1, 128), (2, 640), (8, 1024)])
def test_inputs_that_another_stream_writes(b, s):
    # The consumer's stream always has a kernel of this library right before the event that it waits for, and the producer is
    # kept busy for about a millisecond before it writes.
    qh, kvh = 16, 4
    new = [torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16) for h in (qh, kvh, kvh)]
    host = torch.arange(0, (b + 1) * s, s, dtype=torch.int32)
    new_cu = host.cuda()
    expected = min_fa3_op.forward(*new, True, return_lse=True)
    expected_packed = _packed(*(t.flatten(0, 1) for t in new), new_cu, host, s)
    producer, consumer = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        inputs = [torch.zeros_like(t) for t in new]
        cu = torch.zeros_like(new_cu)
        torch.cuda.synchronize()
        with torch.cuda.stream(consumer):
            min_fa3_op.forward(*new, True)
        with torch.cuda.stream(producer):
            torch.cuda._sleep(2_000_000)
            for t, n in zip((*inputs, cu), (*new, new_cu)):
                t.copy_(n)
            written = torch.cuda.Event()
            written.record()
        with torch.cuda.stream(consumer):
            consumer.wait_event(written)
            got = min_fa3_op.forward(*inputs, True, return_lse=True)
            got_packed = _packed(*(t.flatten(0, 1) for t in inputs), cu, host, s)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip((*got, *got_packed), (*expected, *expected_packed)))
