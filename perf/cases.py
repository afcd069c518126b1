"""Performance cases: attention calls as programs make them, through the public entry points.

A case is one pass of one of five kinds:

    fwd      ``min_fa3_op.forward``: evaluation and prefill; with fewer query rows than keys it continues
             sequences whose K/V are already there (one token or a chunk at a time)
    train    ``min_fa3_op.forward`` + ``backward``, or the same through ``autograd.attention``
    vfwd     ``min_fa3_op.forward_varlen`` on packed documents
    vtrain   ``forward_varlen`` + ``backward_varlen``, or ``autograd.attention_varlen``
    ring     forward + backward through ``autograd.RingAttention`` (one rank: its own shard only)

Head dimension 128 and bf16 are all the library has.  ``listed()`` gives one case for each kind of use,
``draw()`` more of the same ranges, ``prepare()`` / ``run()`` execute one, ``work()`` counts the bytes and
operations it cannot do without, ``tolerance()`` says how far two correct results may be apart and ``exact()``
gives the same attention in 64 bits.
"""
from __future__ import annotations

import math
import random

import torch

import min_fa3_op
from min_fa3_demo_b200 import autograd

HEAD_DIM = 128

# (query heads, key/value heads) of the repository's benchmark configurations and tests: grouped, wide groups, one
# key/value head per query head, one for all.
HEADS = [(32, 8), (16, 4), (64, 8), (32, 32), (8, 2), (8, 1)]


def listed():
    return [
        # A single short sequence: what one call costs.
        dict(name="fwd_short", kind="fwd", batch=1, sq=128, sk=128, qh=32, kvh=32, causal=True),
        # One new token for each of 16 sequences that are 4,000 tokens long.
        dict(name="fwd_one_token", kind="fwd", batch=16, sq=1, sk=4001, qh=32, kvh=8, causal=True),
        # The next chunk of a long prompt against the part that was read before.
        dict(name="fwd_chunk", kind="fwd", batch=1, sq=512, sk=16384, qh=32, kvh=8, causal=True),
        # A batch of ordinary prompts.
        dict(name="fwd_prompts", kind="fwd", batch=4, sq=2048, sk=2048, qh=32, kvh=8, causal=True),
        # Packed short documents (reranking, classification) of ragged lengths.
        dict(name="vfwd_short_docs", kind="vfwd", total=16384, median=250, sigma=0.7, shortest=16, longest=2048, docs=1,
             qh=16, kvh=4, causal=True),
        # Benchmark configuration 1, as a model calls it: the differentiable front end on a small batch.
        dict(name="train_small", kind="train", batch=2, sq=1024, sk=1024, qh=16, kvh=4, causal=True, api="autograd",
             deterministic=False),
        # An encoder: no mask, one key/value head per query head, a length that is no multiple of anything.
        dict(name="train_encoder", kind="train", batch=2, sq=3001, sk=3001, qh=32, kvh=32, causal=False, api="op",
             deterministic=False),
        # Reproducible training: the backward with a fixed order of additions.
        dict(name="train_repeatable", kind="train", batch=2, sq=4096, sk=4096, qh=32, kvh=8, causal=True, api="op",
             deterministic=True),
        # Benchmark configuration 2, causal.
        dict(name="train_bench", kind="train", batch=4, sq=8192, sk=8192, qh=32, kvh=8, causal=True, api="op",
             deterministic=False),
        # One long sequence.
        dict(name="train_long", kind="train", batch=1, sq=32768, sk=32768, qh=32, kvh=8, causal=True, api="op",
             deterministic=False),
        # Benchmark configuration 3: a packed batch of documents of very different lengths.
        dict(name="vtrain_packed", kind="vtrain", total=65536, median=1500, sigma=1.2, shortest=128, longest=32768, docs=0,
             qh=32, kvh=8, causal=True, api="op"),
        # The head layout and length mixture of benchmark configuration 5 on one rank.
        dict(name="ring_one_rank", kind="ring", total=32768, median=2000, sigma=1.0, shortest=256, longest=16384, docs=0,
             qh=64, kvh=8, causal=True),
    ]


def _log_uniform(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["fwd", "fwd", "fwd", "train", "train", "train", "vfwd", "vtrain", "ring"])
        qh, kvh = rng.choice(HEADS)
        case = dict(kind=kind, qh=qh, kvh=kvh, causal=rng.random() < 0.8)
        if kind in ("fwd", "train"):
            sq = _log_uniform(rng, 64, 32768)
            if rng.random() < 0.3:                       # often a round number of tokens
                sq = max(128, sq // 128 * 128)
            case.update(sq=sq, sk=sq)
            if kind == "fwd" and rng.random() < 0.5:     # the sequences are there already: a token or a chunk more
                case.update(sq=_log_uniform(rng, 1, 1024), causal=True)
                case.update(sk=_log_uniform(rng, max(128, case["sq"]), 32768))
            case["batch"] = _log_uniform(rng, 1, max(1, min(32, 65536 // case["sk"])))
        else:
            median = _log_uniform(rng, 150, 3000)
            case.update(total=_log_uniform(rng, 4096, 65536), median=median, sigma=round(rng.uniform(0.4, 1.2), 2),
                        shortest=16, longest=16384, docs=rng.randrange(1000))
            if kind == "ring":                           # shards consist of whole 256-token pieces
                case.update(total=max(4096, case["total"] // 256 * 256), shortest=256)
        if kind in ("train", "vtrain"):
            case["api"] = rng.choice(["op", "autograd"])
        if kind == "train":
            case["deterministic"] = rng.random() < 0.2
        w = work(case)
        if w["flops"] <= most and w["bytes"] <= 4e9:
            return case


def lengths(case):
    """Document lengths of a packed case: log-normal, clipped, drawn until ``total`` is reached, the last one cut."""
    rng = random.Random(case["docs"])
    step = 256 if case["kind"] == "ring" else 1
    out, left = [], case["total"]
    while left > 0:
        n = round(rng.lognormvariate(math.log(case["median"]), case["sigma"]))
        n = min(max(n, case["shortest"]), case["longest"])
        n = min(max(step, n // step * step), left)
        out.append(n)
        left -= n
    return out


class _State:
    pass


def _tensors(s, gen, q_shape, kv_shape, train):
    def normal(shape):
        return torch.randn(shape, device="cuda", generator=gen, dtype=torch.float32).to(torch.bfloat16)
    s.q, s.k, s.v = normal(q_shape), normal(kv_shape), normal(kv_shape)
    s.dout = normal(q_shape) if train else None


def prepare(case, seed):
    s = _State()
    s.case, s.kind, s.causal = case, case["kind"], case["causal"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    train = s.kind in ("train", "vtrain", "ring")
    if s.kind in ("fwd", "train"):
        _tensors(s, gen, (case["batch"], case["sq"], case["qh"], HEAD_DIM),
                 (case["batch"], case["sk"], case["kvh"], HEAD_DIM), train)
    else:
        s.lens = lengths(case)
        _tensors(s, gen, (case["total"], case["qh"], HEAD_DIM), (case["total"], case["kvh"], HEAD_DIM), train)
    if s.kind in ("vfwd", "vtrain"):
        s.cu_host = torch.tensor([0] + s.lens, dtype=torch.int32).cumsum(0, dtype=torch.int32)
        s.cu = s.cu_host.cuda()
        s.longest = max(s.lens)
    if s.kind == "ring":
        s.ring = autograd.RingAttention(case["total"], case["kvh"], is_causal=s.causal, max_documents=len(s.lens),
                                        device=torch.device("cuda", torch.cuda.current_device()))
    if s.kind == "ring" or case.get("api") == "autograd":
        for t in (s.q, s.k, s.v):
            t.requires_grad_(True)
    return s


def run(s):
    if s.kind == "fwd":
        return min_fa3_op.forward(s.q, s.k, s.v, s.causal, return_lse=True)
    if s.kind == "vfwd":
        return min_fa3_op.forward_varlen(s.q, s.k, s.v, s.cu, s.cu, s.longest, s.longest, s.causal,
                                         cu_seqlens_q_host=s.cu_host, cu_seqlens_k_host=s.cu_host, return_lse=True)
    if s.kind == "train":
        if s.case["api"] == "autograd":
            out = autograd.attention(s.q, s.k, s.v, s.causal, deterministic=s.case["deterministic"])
            return (out, *torch.autograd.grad(out, (s.q, s.k, s.v), s.dout))
        out, lse = min_fa3_op.forward(s.q, s.k, s.v, s.causal, return_lse=True)
        return (out, lse, *min_fa3_op.backward(s.dout, s.q, s.k, s.v, out, lse, s.causal,
                                               deterministic=s.case["deterministic"]))
    if s.kind == "vtrain":
        if s.case["api"] == "autograd":
            out = autograd.attention_varlen(s.q, s.k, s.v, s.cu, s.cu, s.longest, s.longest, s.causal,
                                            cu_seqlens_q_host=s.cu_host, cu_seqlens_k_host=s.cu_host)
            return (out, *torch.autograd.grad(out, (s.q, s.k, s.v), s.dout))
        out, lse = min_fa3_op.forward_varlen(s.q, s.k, s.v, s.cu, s.cu, s.longest, s.longest, s.causal,
                                             cu_seqlens_q_host=s.cu_host, cu_seqlens_k_host=s.cu_host, return_lse=True)
        return (out, lse, *min_fa3_op.backward_varlen(s.dout, s.q, s.k, s.v, out, lse, s.cu, s.cu, s.longest, s.longest,
                                                      s.causal))
    ones, zeros = [1] * len(s.lens), [0] * len(s.lens)
    out = s.ring(s.q, s.k, s.v, s.lens, s.lens, ones, zeros)
    return (out, *torch.autograd.grad(out, (s.q, s.k, s.v), s.dout))


def _visible(sq: int, sk: int, causal: bool) -> int:
    """Number of (query row, key) pairs that a sequence computes; the mask is aligned to the last row and key."""
    if not causal:
        return sq * sk
    rows = min(sq, sk)                                   # rows that see a key: the last `rows` of them
    return rows * sk - rows * (rows - 1) // 2


def work(case):
    qh, kvh = case["qh"], case["kvh"]
    train = case["kind"] in ("train", "vtrain", "ring")
    if case["kind"] in ("fwd", "train"):
        rows_q, rows_k = case["batch"] * case["sq"], case["batch"] * case["sk"]
        visible = case["batch"] * _visible(case["sq"], case["sk"], case["causal"])
    else:
        rows_q = rows_k = case["total"]
        visible = sum(_visible(n, n, case["causal"]) for n in lengths(case))
    q_bytes, k_bytes, lse_bytes = rows_q * qh * HEAD_DIM * 2, rows_k * kvh * HEAD_DIM * 2, rows_q * qh * 4
    moved = 2 * q_bytes + 2 * k_bytes + lse_bytes        # q, k, v in; out, lse out
    if train:
        moved += 2 * q_bytes + 2 * k_bytes               # dout in; dq, dk, dv out
    return {"bytes": moved, "flops": (14 if train else 4) * HEAD_DIM * qh * visible}


def tolerance(case):
    # Against the same attention in 64 bits the outputs differ by 1.9e-3 ... 2.5e-3 in the 2-norm (bf16 probabilities and
    # bf16 results), and one value by at most 0.13 of the root mean square (dq of a causal sequence's first rows, whose
    # terms are many times the mean): four times that.
    return {"rel": 1e-2, "max": 0.5}


def _attend(q, k, v, dout, causal):
    """One sequence in 64 bits: q, dout [sq, QH, 128], k, v [sk, KVH, 128] -> out, lse [QH, sq], dq, dk, dv."""
    sq, sk, qh, group = q.size(0), k.size(0), q.size(1), q.size(1) // k.size(1)
    scale = 1.0 / math.sqrt(HEAD_DIM)
    out, lse = torch.empty_like(q), q.new_empty((qh, sq))
    dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for r0 in range(0, sq, 2048):
        r1 = min(r0 + 2048, sq)
        seen = min(sk, r1 + sk - sq) if causal else sk
        hidden = None
        if causal:
            hidden = (torch.arange(seen, device=q.device)[None, :]
                      > torch.arange(r0, r1, device=q.device)[:, None] + (sk - sq))
        for h in range(qh):
            kh, vh = k[:seen, h // group], v[:seen, h // group]
            s = (q[r0:r1, h] @ kh.T).mul_(scale)
            if hidden is not None:
                s.masked_fill_(hidden, -math.inf)
            lse[h, r0:r1] = torch.logsumexp(s, dim=1)
            p = s.sub_(lse[h, r0:r1, None]).exp_()
            out[r0:r1, h] = p @ vh
            if dout is not None:
                do = dout[r0:r1, h]
                dv[:seen, h // group] += p.T @ do
                ds = (do @ vh.T).sub_((do * out[r0:r1, h]).sum(1, keepdim=True)).mul_(p).mul_(scale)
                dq[r0:r1, h] = ds @ kh
                dk[:seen, h // group] += ds.T @ q[r0:r1, h]
    return out, lse, dq, dk, dv


def exact(case, seed):
    if work(case)["flops"] > 2e13:                       # more than about 20 seconds in 64 bits
        return None
    s = prepare(case, seed)
    q, k, v = (t.detach().double() for t in (s.q, s.k, s.v))
    dout = None if s.dout is None else s.dout.double()
    if s.kind in ("fwd", "train"):
        parts = [_attend(q[b], k[b], v[b], None if dout is None else dout[b], s.causal) for b in range(q.size(0))]
        out, lse, dq, dk, dv = (torch.stack(x) for x in zip(*parts))
    else:
        parts = [_attend(*x, s.causal) for x in zip(q.split(s.lens), k.split(s.lens), v.split(s.lens),
                                                    [None] * len(s.lens) if dout is None else dout.split(s.lens))]
        out, lse, dq, dk, dv = (torch.cat(x, dim=1 if n == 1 else 0) for n, x in enumerate(zip(*parts)))
    if s.dout is None:
        return out, lse
    if s.kind == "ring" or case.get("api") == "autograd":
        return out, dq, dk, dv
    return out, lse, dq, dk, dv
