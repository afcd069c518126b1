"""Forward parity on the GPU: the CUDA path (through min_fa3_op -> C ABI) against the CPU
oracle and the reference's golden fixtures.  Acceptance: O within 2x the max-abs error of a
bf16 PyTorch attention against the fp32 oracle, LSE within 1e-3 absolute."""
from __future__ import annotations

import pytest
import torch

import min_fa3_op
from min_fa3_demo_b200 import min_fa3_op as min_fa3_op_impl
from conftest import from_bf16_bits, load_golden
from gpu_util import (assert_cut, assert_lse, assert_within, bound, is_cut, make_bshd, make_varlen, plain_workspace_forward,
                      varlen_bf16_errors)
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


def run_bshd(q, k, v, causal, **kw):
    out, lse = min_fa3_op.forward(q.cuda(), k.cuda(), v.cuda(), causal, return_lse=True, **kw)
    torch.cuda.synchronize()
    return out, lse


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,s,qh,kvh", [
    (1, 128, 32, 32),      # reference test default shape
    (1, 129, 4, 2),        # one row past a tile
    (2, 1024, 16, 4),      # benchmark configuration 1
    (1, 333, 2, 1),        # ragged, MQA
    (3, 640, 8, 8),
    (1, 1, 2, 2),          # single token
])
def test_bshd_forward_vs_oracle(b, s, qh, kvh, causal):
    q, k, v, _ = make_bshd(1234 + s, b, s, qh, kvh)
    out, lse = run_bshd(q, k, v, causal)
    assert out.shape == q.shape and out.dtype == torch.bfloat16
    assert lse.shape == (b, qh, s) and lse.dtype == torch.float32
    ref_out, ref_lse = orc.bshd_forward(q, k, v, causal)
    e = orc.bf16_attention_error(q, k, v, causal)["o"]
    assert_within("O", out, ref_out, e)
    assert_lse(lse, ref_lse)


@pytest.mark.parametrize("sq,sk", [(256, 512), (128, 1000), (300, 200), (512, 128)])
def test_bshd_forward_rectangular_causal(sq, sk):
    # bottom-right aligned mask; with sq > sk the first rows see no key: O = 0, LSE = -inf
    q, k, v, _ = make_bshd(77, 1, sq, 4, 2, sk=sk)
    out, lse = run_bshd(q, k, v, True)
    ref_out, ref_lse = orc.bshd_forward(q, k, v, True)
    e = orc.bf16_attention_error(q, k, v, True)["o"]
    assert_within("O", out, ref_out, max(e, 4e-3))
    assert_lse(lse, ref_lse)
    if sq > sk:
        assert torch.all(out[0, : sq - sk] == 0)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,sq,sk,qh,kvh,cut", [
    (1, 1, 1024, 8, 1, False),      # one row of 8 heads: one tile, 8 of its rows used
    (1, 1, 4096, 8, 1, True),       # ... with the keys cut into eight pieces
    (2, 1, 4001, 8, 2, True),       # ... with a ragged last key block
    (5, 1, 4001, 32, 32, True),     # 160 items, of which the last 12 are cut
    (1, 31, 2049, 16, 4, True),     # 124 packed rows
    (1, 33, 3000, 16, 4, True),     # 132: four rows in the second tile
    (1, 300, 4096, 4, 4, True),     # nothing to pack; the second item has 44 rows
    (1, 200, 5000, 32, 1, True),    # 32 heads a row: four rows a tile
    (1, 1030, 2048, 8, 2, True),    # causal: items of different lengths, cut into different numbers of pieces
    (1, 2048, 2048, 4, 1, True),    # causal: items of one piece among them
    (1, 100, 3000, 12, 2, False),   # groups of 6 are not packed and not cut: two heads an item
    (1, 90, 1100, 6, 2, False),     # groups of 3
    (1, 700, 1024, 256, 1, False),  # more heads than a tile has rows
    (1, 9000, 70, 40, 40, False),   # causal: CTAs draw many items in a row that see no key
    (1, 4500, 70, 24, 4, False),    # ... of two heads each
])
def test_bshd_forward_packed_rows_and_key_pieces(b, sq, sk, qh, kvh, cut, causal):
    assert_cut(cut, "fwd", b, sq, sk, qh, kvh, causal)
    q, k, v, _ = make_bshd(31 + sq, b, sq, qh, kvh, sk=sk)
    out, lse = run_bshd(q, k, v, causal)
    min_fa3_op_impl.check_last_status("forward")
    ref_out, ref_lse = orc.bshd_forward(q, k, v, causal)
    e = orc.bf16_attention_error(q, k, v, causal)["o"]
    assert_within("O", out, ref_out, e)
    assert_lse(lse, ref_lse)
    # The plain workspace is enough for the same call, without cutting the keys.
    out2, lse2 = plain_workspace_forward(q.cuda(), k.cuda(), v.cuda(), causal)
    assert_within("O (plain workspace)", out2, ref_out, e)
    assert_lse(lse2, ref_lse)


@pytest.mark.parametrize("b,sq,sk,qh,kvh,causal", [
    (2, 1, 4001, 8, 2, True),         # eight pieces
    (1, 300, 4096, 4, 4, False),      # two tiles, the second with 44 rows
    (1, 8192, 8192, 2, 1, True),      # items of one piece and pieces without a block for the first tile
])
def test_key_pieces_keep_nan_and_infinities(b, sq, sk, qh, kvh, causal):
    # A NaN or an infinity shows in the same places whether the keys are cut or not: one in a query row, in a key (none of
    # those whose exponential is the polynomial, which clamps NaN in both kernels) or in a value.
    assert_cut(True, "fwd", b, sq, sk, qh, kvh, causal)
    q, k, v, _ = (t.cuda() for t in make_bshd(5 + sq, b, sq, qh, kvh, sk=sk))
    for name, row, value in (("q", sq // 2, float("nan")), ("k", 5, float("nan")), ("k", sk // 2 + 1, float("nan")),
                             ("k", sk - 1, float("nan")), ("v", 5, float("nan")), ("v", sk - 1, float("inf"))):
        bad = {"q": q, "k": k, "v": v}
        bad[name] = bad[name].clone()
        bad[name][0, row, 0, 77] = value
        out, lse = run_bshd(bad["q"], bad["k"], bad["v"], causal)
        plain_out, plain_lse = plain_workspace_forward(bad["q"], bad["k"], bad["v"], causal)
        where = f"{name}[{row}] = {value}"
        assert not torch.isfinite(plain_out).all(), where
        assert torch.equal(torch.isnan(out), torch.isnan(plain_out)), where
        assert torch.equal(torch.isposinf(out), torch.isposinf(plain_out)), where
        assert torch.equal(torch.isneginf(out), torch.isneginf(plain_out)), where
        assert torch.equal(torch.isnan(lse), torch.isnan(plain_lse)), where
        assert torch.equal(torch.isneginf(lse), torch.isneginf(plain_lse)), where


@pytest.mark.parametrize("cut,b,sq,sk,qh,kvh,causal", [
    (True, 1, 512, 16384, 32, 8, True),      # 194 us uncut, 114 cut
    (True, 2, 3001, 3001, 32, 32, False),    # 255 and 248: the last of six rounds
    (True, 1, 1, 4096, 8, 1, True),
    (False, 1, 1, 1024, 8, 1, True),         # eight blocks, and nothing gained
    (False, 1, 6829, 6829, 8, 2, True),      # 91 and 101: the shortest items come last anyway
    (False, 1, 6192, 6192, 8, 1, True),      # 84 and 91
    (False, 2, 1024, 1024, 16, 4, True),     # 21 and 35
    (False, 1, 512, 16384, 24, 8, True),     # groups that are no power of two are not cut
])
def test_which_calls_are_cut(cut, b, sq, sk, qh, kvh, causal):
    assert_cut(cut, "fwd", b, sq, sk, qh, kvh, causal)


@pytest.mark.parametrize("blocks", [1, 7, 300])
def test_a_cut_call_is_the_same_on_any_number_of_ctas(blocks):
    sizes = (1, 300, 4096, 4, 4)
    assert_cut(True, "fwd", *sizes, True)
    q, k, v, _ = make_bshd(6, 1, 300, 4, 4, sk=4096)
    out, lse = run_bshd(q, k, v, True)
    out2, lse2 = run_bshd(q, k, v, True, manual_block_count=blocks)
    assert torch.equal(out, out2) and torch.equal(lse, lse2)


def test_partial_results_do_not_outlive_the_call():
    # Kept for check_last_status is the workspace alone, not the 16 MiB and more of a cut call's partial results.
    sizes = (1, 512, 8192, 32, 8, True)
    assert_cut(True, "fwd", *sizes)
    assert_cut(True, "bwd", 1, 2048, 2048, 32, 8, True)
    q, k, v, _ = (t.cuda() for t in make_bshd(3, 1, 512, 32, 8, sk=8192))
    q2, k2, v2, dout = (t.cuda() for t in make_bshd(4, 1, 2048, 32, 8))
    out2, lse2 = min_fa3_op.forward(q2, k2, v2, True, return_lse=True)
    min_fa3_op.forward(q, k, v, True)
    min_fa3_op.backward(dout, q2, k2, v2, out2, lse2, True)
    kept = min_fa3_op_impl._LAST.workspaces
    lib = min_fa3_op_impl._cabi.load()
    assert kept["forward"].numel() == lib.b2a_fwd_workspace_bytes(1, 512, 0)
    assert kept["backward"].numel() == lib.b2a_bwd_workspace_bytes(1, 2048, 2048, 32, 8, 0)
    min_fa3_op_impl.check_last_status("forward")
    min_fa3_op_impl.check_last_status("backward")


@pytest.mark.parametrize("tag,causal", [("full", False), ("causal", True)])
def test_bshd_forward_golden(tag, causal):
    g = load_golden(f"bshd_{tag}")
    q, k, v = (from_bf16_bits(g[n]) for n in ("q", "k", "v"))
    out, _ = run_bshd(q, k, v, causal)
    golden = from_bf16_bits(g["out_bf16"]).float()
    e = orc.bf16_attention_error(q, k, v, causal)["o"]
    # the golden output is itself rounded to bf16: allow that rounding on top of the rule
    assert (out.float().cpu() - golden).abs().max().item() <= bound(e) + 2.0 ** -8 * golden.abs().max().item()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lengths,qh,kvh", [
    ([128, 129], 4, 2),                                  # reference varlen default
    ([128, 111, 94, 128, 111, 94], 8, 2),                # S - 17*(i%3), reference backward test
    ([1, 700, 255, 257, 1024, 3], 4, 4),
    ([2048], 2, 1),
    ([37] * 40, 2, 2),                                   # many short documents
    ([200, 0, 77, 0], 4, 2),                             # empty documents inside and at the end
    ([0, 128], 2, 2),                                    # ... and in front
])
def test_varlen_forward_vs_oracle(lengths, qh, kvh, causal):
    q, k, v, dout, cu = make_varlen(99 + len(lengths), lengths, qh, kvh)
    out, lse = min_fa3_op.forward_varlen(
        q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lengths), max(lengths), causal,
        cu_seqlens_q_host=cu, cu_seqlens_k_host=cu, return_lse=True)
    torch.cuda.synchronize()
    assert lse.shape == (qh, sum(lengths))
    ref_out, ref_lse = orc.varlen_forward(q, k, v, cu.tolist(), cu.tolist(), causal)
    e = varlen_bf16_errors(q, k, v, dout, cu, causal)["o"]
    assert_within("O", out, ref_out, e)
    assert_lse(lse, ref_lse)


@pytest.mark.parametrize("tag,causal", [("full", False), ("causal", True)])
def test_varlen_forward_golden(tag, causal):
    g = load_golden(f"varlen_{tag}")
    q, k, v = (from_bf16_bits(g[n]) for n in ("q", "k", "v"))
    cu = torch.from_numpy(g["cu_seqlens"])
    lengths = (cu[1:] - cu[:-1]).tolist()
    out = min_fa3_op.forward_varlen(
        q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lengths), max(lengths), causal,
        cu_seqlens_q_host=cu, cu_seqlens_k_host=cu)
    golden = from_bf16_bits(g["out_bf16"]).float()
    assert (out.float().cpu() - golden).abs().max().item() <= 2e-2


def test_varlen_different_q_and_k_lengths():
    gen = torch.Generator().manual_seed(5)
    q_lens, k_lens = [100, 260, 7], [300, 260, 90]
    cu_q = torch.tensor([0, 100, 360, 367], dtype=torch.int32)
    cu_k = torch.tensor([0, 300, 560, 650], dtype=torch.int32)
    q = torch.randn(367, 4, 128, generator=gen).to(torch.bfloat16)
    k = torch.randn(650, 2, 128, generator=gen).to(torch.bfloat16)
    v = torch.randn(650, 2, 128, generator=gen).to(torch.bfloat16)
    for causal in (False, True):
        out, lse = min_fa3_op.forward_varlen(
            q.cuda(), k.cuda(), v.cuda(), cu_q.cuda(), cu_k.cuda(), max(q_lens), max(k_lens), causal,
            cu_seqlens_q_host=cu_q, cu_seqlens_k_host=cu_k, return_lse=True)
        ref_out, ref_lse = orc.varlen_forward(q, k, v, cu_q.tolist(), cu_k.tolist(), causal)
        assert_within("O", out, ref_out, 4e-3)
        assert_lse(lse, ref_lse)


@pytest.mark.parametrize("blocks", [1, 7, 500])
def test_manual_block_count_gives_same_result(blocks):
    q, k, v, _ = make_bshd(11, 2, 1024, 8, 2)
    base, base_lse = run_bshd(q, k, v, True)
    out, lse = run_bshd(q, k, v, True, manual_block_count=blocks)
    assert torch.equal(out, base) and torch.equal(lse, base_lse)


def test_forward_error_behaviour_on_gpu():
    q, k, v, _ = make_bshd(3, 1, 128, 6, 4)
    with pytest.raises(RuntimeError, match="qhead % kvhead == 0"):
        min_fa3_op.forward(q.cuda(), k.cuda(), v.cuda(), True)
    q, k, v, _ = make_bshd(3, 1, 128, 4, 4)
    with pytest.raises(RuntimeError, match="must be contiguous BSHD"):
        min_fa3_op.forward(q.cuda().transpose(1, 2), k.cuda(), v.cuda(), True)
    cu = torch.tensor([0, 100, 128], dtype=torch.int32)
    qv, kv, vv = q[0].cuda(), k[0].cuda(), v[0].cuda()
    bad = torch.tensor([0, 100, 127], dtype=torch.int32)
    with pytest.raises(RuntimeError, match=r"cu_seqlens_q_host\[-1\] must equal q.size\(0\)"):
        min_fa3_op.forward_varlen(qv, kv, vv, cu.cuda(), cu.cuda(), 100, 100, True,
                                  cu_seqlens_q_host=bad, cu_seqlens_k_host=cu)


# ---------------------------------------------------------------------------------------
# Full benchmark sizes: size-independent properties
# ---------------------------------------------------------------------------------------
@pytest.mark.parametrize("causal", [False, True])
def test_full_size_rows_against_oracle_and_properties(causal):
    """Config 2 (B=4, S=8192, QH=32, KVH=8): sampled query rows against the CPU oracle, and
    the prefix property of causal attention."""
    torch.manual_seed(0)
    b, s, qh, kvh = 4, 8192, 32, 8
    q = torch.randn(b, s, qh, 128, device="cuda").to(torch.bfloat16)
    k = torch.randn(b, s, kvh, 128, device="cuda").to(torch.bfloat16)
    v = torch.randn(b, s, kvh, 128, device="cuda").to(torch.bfloat16)
    out, lse = min_fa3_op.forward(q, k, v, causal, return_lse=True)
    assert torch.isfinite(out.float()).all() and torch.isfinite(lse).all()

    # sampled rows of (batch 3, query heads 28..31 -> kv head 7) against the fp32 oracle
    rows = torch.tensor([0, 1, 127, 128, 255, 256, 4095, 4096, 8063, 8064, 8191])
    qs = q[3, rows][:, 28:32].cpu()
    ks, vs = k[3, :, 7:8].cpu(), v[3, :, 7:8].cpu()
    qpos = rows if causal else None
    kpos = torch.arange(s) if causal else None
    ref_out, ref_lse = orc.attention_positions(qs, ks, vs, qpos, kpos)
    assert (out[3, rows][:, 28:32].float().cpu() - ref_out).abs().max().item() <= 1.6e-2
    assert (lse[3, 28:32][:, rows].cpu() - ref_lse).abs().max().item() <= 1e-3

    if causal:
        # prefix property: the first n rows only depend on the first n keys
        n = 1536
        out_prefix = min_fa3_op.forward(q[:, :n].contiguous(), k[:, :n].contiguous(),
                                        v[:, :n].contiguous(), True)
        assert (out_prefix.float() - out[:, :n].float()).abs().max().item() <= 1.6e-2
    else:
        # permuting the keys (K and V together) does not change non-causal attention
        perm = torch.randperm(s, device="cuda")
        out_perm = min_fa3_op.forward(q, k[:, perm].contiguous(), v[:, perm].contiguous(), False)
        assert (out_perm.float() - out.float()).abs().max().item() <= 1.6e-2

    # rows of P sum to one: with V = 1 the output is exactly one
    ones = torch.ones_like(v)
    out_ones = min_fa3_op.forward(q, k, ones, causal)
    assert (out_ones.float() - 1.0).abs().max().item() <= 2.0 ** -7


@pytest.mark.parametrize("b,s,qh,kvh", [(1, 1, 8, 2), (1, 130, 3, 3), (1, 128, 32, 32), (2, 1184, 16, 4), (2, 1185, 16, 4)])
def test_calls_with_an_item_for_each_cta(b, s, qh, kvh):
    """The first three cases have at most as many items as CTAs: nothing is handed out, and the kernel itself clears the status
    words (the last two have 152 items).  Fewer CTAs take the items from the counter instead; the results are the same bits."""
    q, k, v = (torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16) for h in (qh, kvh, kvh))
    for causal in (False, True):
        dirty = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in (256, 256, 512)]
        del dirty                                        # the workspace is likely to be one of these
        out, lse = min_fa3_op.forward(q, k, v, causal, return_lse=True)
        min_fa3_op_impl.check_last_status("forward")
        out2, lse2 = min_fa3_op.forward(q, k, v, causal, return_lse=True, manual_block_count=1)
        min_fa3_op_impl.check_last_status("forward")
        assert torch.equal(out, out2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("b,s,qh,kvh", [(-1, 130, 1, 1), (0, 130, 1, 1), (1, 130, 1, 1), (3, 128, 6, 1), (1, 300, 6, 1)])
def test_as_many_items_as_sms(b, s, qh, kvh):
    """Exactly as many items as SMs, one less and one more (one key/value head: b counts from the number of SMs, a sequence is an
    item), and calls of 6 heads over 1, of which every second item of at most 128 rows is empty.  The ticket in the workspace
    says which way a call went; fewer CTAs, which take the items from the counter, give the same bits."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if qh == 1:
        b += sms
    items = b * ((s + 255) // 256) * qh                  # neither case packs heads into rows
    q, k, v = (torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16) for h in (qh, kvh, kvh))
    for causal in (False, True):
        assert not is_cut("fwd", b, s, s, qh, kvh, causal)
        dirty = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in (1024, 1024)]
        del dirty                                        # the workspace is likely to be one of these
        out, lse = min_fa3_op.forward(q, k, v, causal, return_lse=True)
        min_fa3_op_impl.check_last_status("forward")
        ticket = min_fa3_op_impl._LAST.workspaces["forward"][:4].view(torch.int32).item()
        assert ticket == -items if items <= sms else ticket > 0, "whether items were handed out"
        out2, lse2 = min_fa3_op.forward(q, k, v, causal, return_lse=True, manual_block_count=1)
        min_fa3_op_impl.check_last_status("forward")
        assert torch.equal(out, out2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("change", ["dtype", "rank", "width", "strides", "cpu", "batch", "keys", "kv_heads", "group"])
def test_refusals_after_a_good_call(change):
    """Once a device is known, the checks are one expression: it has to send every bad call to the one that says why."""
    q, k, v = (torch.randn(2, 128, h, 128, device="cuda", dtype=torch.bfloat16) for h in (4, 2, 2))
    out, lse = min_fa3_op.forward(q, k, v, True, return_lse=True)
    min_fa3_op.backward(out, q, k, v, out, lse, True)
    bad = {"dtype": lambda: k.half(), "rank": lambda: k[0], "width": lambda: k[..., :64].contiguous(),
           "strides": lambda: k.transpose(1, 2).contiguous().transpose(1, 2), "cpu": lambda: k.cpu(),
           "batch": lambda: k[:1].contiguous(), "keys": lambda: k[:, :64].contiguous(), "kv_heads": lambda: k[:, :, :1].contiguous(),
           "group": lambda: torch.cat([k, k[:, :, :1]], 2)}[change]()
    with pytest.raises(RuntimeError):
        min_fa3_op.forward(q, bad, torch.cat([v, v[:, :, :1]], 2) if change == "group" else v, True)
    with pytest.raises(RuntimeError):
        min_fa3_op.backward(out, q, bad, torch.cat([v, v[:, :, :1]], 2) if change == "group" else v, out, lse, True)
    cu = torch.tensor([0, 128, 256], dtype=torch.int32)
    qp, kp, vp = (t.flatten(0, 1) for t in (q, k, v))
    o, l = min_fa3_op.forward_varlen(qp, kp, vp, cu.cuda(), cu.cuda(), 128, 128, True, cu_seqlens_q_host=cu, cu_seqlens_k_host=cu,
                                     return_lse=True)
    if change in ("dtype", "width", "strides", "cpu", "kv_heads", "group", "rank"):
        bad = {"rank": kp[0], "strides": kp.transpose(0, 1).contiguous().transpose(0, 1)}.get(change, bad.flatten(0, 1))
        vg = torch.cat([vp, vp[:, :1]], 1) if change == "group" else vp
        with pytest.raises(RuntimeError):
            min_fa3_op.forward_varlen(qp, bad, vg, cu.cuda(), cu.cuda(), 128, 128, True, cu_seqlens_q_host=cu,
                                      cu_seqlens_k_host=cu)
        with pytest.raises(RuntimeError):
            min_fa3_op.backward_varlen(o, qp, bad, vg, o, l, cu.cuda(), cu.cuda(), 128, 128, True)
    for host in (cu.long(), cu[:2], torch.tensor([1, 128, 256], dtype=torch.int32), torch.tensor([0, 128, 255], dtype=torch.int32)):
        with pytest.raises(RuntimeError):
            min_fa3_op.forward_varlen(qp, kp, vp, cu.cuda(), cu.cuda(), 128, 128, True, cu_seqlens_q_host=host,
                                      cu_seqlens_k_host=cu)


@pytest.mark.parametrize("b,s,qh,kvh", [(1, 128, 8, 8), (2, 640, 16, 4), (8, 1024, 16, 4)])
def test_calls_that_feed_each_other(b, s, qh, kvh):
    """A forward's kernels come up while the one before them ends: each has to wait for what that one writes.  Ten calls whose
    queries are the last one's output give the same bits with and without a pause between them, dense and packed in turn."""
    q0, k, v = (torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16) for h in (qh, kvh, kvh))
    cu = torch.arange(0, (b + 1) * s, s, dtype=torch.int32)
    cu_dev = cu.cuda()

    def chain(pause):
        q = q0
        for i in range(10):
            if i % 2 == 0:
                q = min_fa3_op.forward(q, k, v, True)
            else:
                q = min_fa3_op.forward_varlen(q.flatten(0, 1), k.flatten(0, 1), v.flatten(0, 1), cu_dev, cu_dev, s, s, True,
                                              cu_seqlens_q_host=cu, cu_seqlens_k_host=cu).view(b, s, qh, 128)
            if pause:
                torch.cuda.synchronize()
        return q

    expected = chain(True)
    for _ in range(3):
        assert torch.equal(chain(False), expected)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("s", [384, 1024, 1500])
def test_bshd_forward_with_a_growing_maximum(s, causal):
    """Blocks are taken from the last key to the first, and here each has larger scores than the one before, so O is rescaled
    at nearly every block: each time the P V before it has to be done, and no S or P may be lost."""
    q, k, v, _ = make_bshd(5, 1, s, 4, 2)
    k = (k.float() * torch.linspace(24, 1, s).view(1, s, 1, 1)).to(torch.bfloat16)
    out, lse = run_bshd(q, k, v, causal)
    ref_out, ref_lse = orc.bshd_forward(q, k, v, causal)
    # LSE up to about 100: 1e-3 holds for values of a few units, so the same relative bound for these.
    assert_within("O", out, ref_out, orc.bf16_attention_error(q, k, v, causal)["o"])
    assert (lse.cpu() - ref_lse).abs().max() <= 1e-3 * max(1.0, ref_lse.abs().max().item() / 8)
