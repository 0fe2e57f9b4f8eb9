"""sm_100a attention kernels (one ring step) against the fp32 dense oracle, plus the public op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(B, Sq, Sk, H, D, cbs=0, q_off=0, k_off=0, seg=False, bias=False, pdrop=0.0, prev=False, seg_p=0.01):
    from ringattention_b200.ops import _lib, flash, reference as R

    torch.manual_seed(0)
    dev = "cuda"
    q = torch.randn(B, Sq, H, D, device=dev).bfloat16()
    k = torch.randn(B, Sk, H, D, device=dev).bfloat16()
    v = torch.randn(B, Sk, H, D, device=dev).bfloat16()
    do = torch.randn(B, Sq, H, D, device=dev).bfloat16()
    qp, kp = flash.Positions(q_off), flash.Positions(k_off)
    q_pos, k_pos = qp.tensor(Sq, dev), kp.tensor(Sk, dev)
    ms = flash.MaskSpec(causal_block_size=cbs, q_pos=qp, k_pos=kp)
    seg_q = seg_k = bs = None
    if seg:
        tot = max(q_off + Sq, k_off + Sk)
        ids = torch.cumsum((torch.rand(B, tot, device=dev) < seg_p).int(), dim=1).int()
        seg_q, seg_k = ids[:, q_pos].contiguous(), ids[:, k_pos].contiguous()
        ms.seg_q, ms.seg_k = seg_q, seg_k
        ms.seg_q_mm, ms.seg_k_mm = flash.seg_tile_minmax(seg_q), flash.seg_tile_minmax(seg_k)
    if bias:
        bs = torch.randn(B, 1, Sk, device=dev)
        ms.bias = bs
    if pdrop > 0:
        ms.seed, ms.pdrop = 1234567891234, pdrop
    o_prev = lse_prev = None
    if prev:
        o_prev = torch.randn(B, Sq, H, D, device=dev)
        lse_prev = torch.randn(B, H, Sq, device=dev)
    out, lse = flash.flash_fwd(q, k, v, ms, o_prev=o_prev, lse_prev=lse_prev, out_fp32=prev)
    qf, kf, vf = [t.float().requires_grad_(True) for t in (q, k, v)]
    ref, ref_lse = R.dense_attention(qf, kf, vf, q_pos, k_pos, causal_block_size=cbs or None,
                                     bias=None if bs is None else bs[:, :, None, :], seg_q=seg_q,
                                     seg_k=seg_k, seed=ms.seed, pdrop=pdrop, dtype=torch.float32,
                                     return_lse=True)
    if prev:
        mref, mlse = R.merge_partials(o_prev, lse_prev, ref.detach(), ref_lse.detach())
        assert (out.float() - mref).abs().max() < 0.02
        return
    assert (out.float() - ref.detach()).abs().max() < 0.02
    fin = torch.isfinite(ref_lse)
    if fin.any():
        assert (lse[fin] - ref_lse.detach()[fin]).abs().max() < 1e-2
    assert bool((lse[~fin] == float("-inf")).all())
    # backward
    lse2, delta = flash.flash_bwd_prep(out, do, lse)
    dq_acc = torch.zeros(B, Sq, H, D, device=dev)
    dk, dv = torch.zeros_like(k), torch.zeros_like(k)
    flash.flash_bwd(q, k, v, do, lse2, delta, ms, dq_acc, dk, dv)
    torch.cuda.synchronize()
    _lib.check_status()
    ref.backward(do.float())
    for got, want in ((dq_acc, qf.grad), (dk, kf.grad), (dv, vf.grad)):
        assert (got.float() - want).abs().max() <= 0.02 * want.abs().max() + 1e-3


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("cbs", [0, 1, 64])
def test_attention_causal_variants(D, cbs):
    _case(2, 512, 512, 2, D, cbs=cbs)


def test_attention_ragged_and_offsets():
    _case(1, 200, 333, 2, 128)
    _case(1, 200, 333, 2, 128, cbs=1, q_off=133)
    _case(1, 384, 640, 2, 128, cbs=1, q_off=256)
    _case(1, 300, 700, 3, 64, cbs=1, q_off=400, seg=True)


def test_attention_segments_bias_dropout():
    _case(1, 512, 512, 2, 128, cbs=1, seg=True)
    _case(1, 512, 512, 2, 128, bias=True)
    _case(1, 512, 512, 2, 128, cbs=1, pdrop=0.2)


def test_attention_long_documents_take_the_plain_path_inside_a_segment():
    """Documents several tiles long: tile pairs inside one segment skip the per-column masking, pairs of
    different segments are skipped through the visibility bitmask, boundary tiles take the masked path."""
    _case(2, 2048, 2048, 2, 128, cbs=1, seg=True, seg_p=0.002)
    _case(1, 1536, 2048, 2, 128, cbs=0, seg=True, seg_p=0.003)
    _case(1, 1024, 1024, 2, 64, cbs=1, seg=True, seg_p=0.004, pdrop=0.1)


def test_attention_fully_masked_block_and_carry():
    _case(1, 512, 512, 2, 128, cbs=1, k_off=512)           # block entirely in the causal future
    _case(1, 512, 512, 2, 128, cbs=1, q_off=512, prev=True)  # merge with an earlier ring step


def test_public_op_autograd_matches_reference():
    import ringattention_b200 as rab

    torch.manual_seed(3)
    q, k, v = [torch.randn(2, 384, 4, 128, device="cuda").bfloat16().requires_grad_(True) for _ in range(3)]
    ids = torch.cumsum((torch.rand(2, 384, device="cuda") < 0.02).int(), 1).int()
    kw = dict(causal_block_size=1, query_chunk_size=128, key_chunk_size=128)
    out = rab.ringattention(q, k, v, None, ids, None, None, True, kw)
    g = torch.randn_like(out)
    out.backward(g)
    q2, k2, v2 = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    ref = rab.ringattention_ref(q2, k2, v2, None, ids, None, None, True, kw)
    ref.backward(g.float())
    assert (out.float() - ref).abs().max() < 0.02
    for a, b in ((q.grad, q2.grad), (k.grad, k2.grad), (v.grad, v2.grad)):
        assert (a.float() - b).abs().max() <= 0.02 * b.abs().max() + 1e-3


def test_full_bias_is_served_by_the_torch_path():
    import ringattention_b200 as rab

    q, k, v = [torch.randn(1, 64, 2, 64, device="cuda").bfloat16() for _ in range(3)]
    bias = torch.randn(1, 1, 64, 64, device="cuda")
    out = rab.ringattention(q, k, v, bias, None, None, None, True, dict(query_chunk_size=32, key_chunk_size=32))
    assert out.shape == q.shape and out.dtype == v.dtype


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (2, 130, 2, 128), (1, 257, 3, 64), (2, 128, 7, 128), (1, 1000, 9, 128), (1, 129, 16, 64)])
@pytest.mark.parametrize("strided", [False, True])
def test_backward_preparation(B, S, H, D, strided):
    """delta, the scaled log-sum-exp and the zeroed accumulator at head counts around the eight of a CTA, at lengths around
    a padded tile, and on views into a wider buffer. Tolerance: an fp32 sum of D products, 1e-6 of their magnitudes."""
    from ringattention_b200.ops import flash

    torch.manual_seed(S)
    wide = torch.randn(2, B, S, H, 3, D, device="cuda").bfloat16()
    out, dout = (w[:, :, :, 1] if strided else w[:, :, :, 1].contiguous() for w in wide)
    lse = torch.randn(B, H, S, device="cuda")
    lse[:, :, S // 2] = -float("inf")
    acc = torch.full((B * S * H * D + 64,), 7.0, device="cuda")
    lse2, delta = flash.flash_bwd_prep(out, dout, lse, acc[:-64].view(B, S, H, D))
    terms = (out.double() * dout.double()).permute(0, 2, 1, 3)
    assert ((delta[:, :, :S].double() - terms.sum(-1)).abs() <= 1e-6 * terms.abs().sum(-1) + 1e-12).all()
    assert (delta[:, :, S:] == 0).all() and (lse2[:, :, S:] == -float("inf")).all()
    want = torch.where(torch.isinf(lse), lse, -lse * 1.4426950408889634)
    assert torch.allclose(lse2[:, :, :S], want, rtol=1e-6, atol=0)
    assert (acc[:-64] == 0).all() and (acc[-64:] == 7).all()


def _oracle(q, k, v, dout, hidden, bias=None):
    """Dense attention and its gradients in 64 bits; rows without a visible key give zeros."""
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    x = torch.einsum("bqhd,bkhd->bhqk", q, k) / q.shape[-1] ** 0.5
    if bias is not None:
        x = x + bias.double()
    x = x.masked_fill(hidden | (x < -1e30), -float("inf"))
    m = x.amax(-1, keepdim=True).clamp_min(-1e300)
    e = torch.exp(x - m)
    p = e / e.sum(-1, keepdim=True).clamp_min(1e-300)
    out = torch.einsum("bhqk,bkhd->bqhd", p, v)
    return (out.detach(), *torch.autograd.grad(out, (q, k, v), dout.double()))


def _check_call(B, Sq, Sk, H, D, *, cbs=None, seg=None, bias=None, cache_idx=None, grad=True):
    """``ringattention`` on one device against the oracle. bf16 keeps 8 bits: outputs within 1e-2 of the largest entry (P and
    the result are rounded once each, 2^-8 apiece at worst), gradients within 2e-2 (dS is rounded as well)."""
    import ringattention_b200 as rab

    g = torch.Generator(device="cuda").manual_seed(Sq * 7 + Sk)
    q, dout = (torch.randn(B, Sq, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Sk, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    hidden = torch.zeros(B, 1, Sq, Sk, dtype=torch.bool, device="cuda")
    if cbs:
        pos = torch.arange(Sq, device="cuda") + (cache_idx or 0)
        hidden |= (pos[:, None] // cbs < torch.arange(Sk, device="cuda")[None] // cbs)
    if seg is not None:
        hidden |= (seg[:, :, None] != seg[:, None, :])[:, None]
    want = _oracle(q, k, v, dout, hidden, bias)
    kw = dict(causal_block_size=cbs, query_chunk_size=Sq, key_chunk_size=Sk)
    q, k, v = (t.requires_grad_(grad) for t in (q, k, v))
    out = rab.ringattention(q, k, v, bias, seg, cache_idx, None, True, kw)
    got = [out.detach()] + (list(torch.autograd.grad(out, (q, k, v), dout)) if grad else [])
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.isfinite(a).all()
        assert (a.double() - b).abs().max() <= (0.01 if i == 0 else 0.02) * b.abs().max() + 1e-3, i


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S,pads", [(1371, (700, 1371, 256)), (513, (1, 128, 512)), (384, (129, 255, 383))])
def test_padding_bias_hides_whole_and_partial_tiles(S, pads, D):
    """The type's lowest value from a row's length on: tiles that are all padding are not visited, tiles without any are
    plain, the one between is masked; causal and not."""
    bias = torch.zeros(len(pads), 1, 1, S, device="cuda")
    for b, n in enumerate(pads):
        bias[b, 0, 0, n:] = torch.finfo(torch.float32).min
    _check_call(len(pads), S, S, 2, D, cbs=1, bias=bias)
    _check_call(len(pads), S, S, 2, D, bias=bias)


@pytest.mark.parametrize("D", [64, 128])
def test_finite_bias_in_some_tiles_and_per_head(D):
    """A finite bias in one tile only, padding with -inf elsewhere, a row whose keys are all hidden, a bias per head."""
    S, H = 640, 3
    bias = torch.zeros(2, H, 1, S, device="cuda")
    bias[0, 1, 0, 130:200] = torch.randn(70, device="cuda") * 3
    bias[0, 2, 0, 256:384] = -float("inf")
    bias[1, 0] = -float("inf")
    bias[1, 2, 0, ::2] = -float("inf")
    _check_call(2, S, S, H, D, bias=bias)
    _check_call(2, S, S, H, D, cbs=1, bias=bias)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("ids", ["per token", "runs", "one change", "alternating"])
def test_segment_ids_of_every_kind(ids, D):
    """Ids need not be sorted: every token its own, short runs that come back, one border inside a tile, two in turn."""
    B, S = 2, 700
    t = torch.arange(S, device="cuda")
    seg = {"per token": t, "runs": t // 5 % 7, "one change": (t >= 333).int(), "alternating": t % 2}[ids].int()[None].expand(B, S).contiguous()
    _check_call(B, S, S, 2, D, seg=seg)
    _check_call(B, S, S, 2, D, cbs=1, seg=seg, bias=torch.randn(B, 1, 1, S, device="cuda"))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,H,cbs,cache_idx", [
    (1, 1, 1, 1, 1, None), (1, 128, 128, 1, 1, None), (1, 129, 129, 2, 1, None), (2, 300, 300, 3, 64, None),   # one tile or two
    (1, 512, 512, 8, None, None), (1, 2048, 2048, 4, 1, None), (1, 1300, 1300, 2, None, None),                 # tiles shared by two groups
    (1, 16, 20000, 2, 1, 19984), (1, 200, 9000, 4, 1, 8000), (2, 100, 8200, 1, None, None), (1, 130, 4100, 2, 32, 3970),  # keys split
    (1, 128, 40000, 1, 1, 100),                                                                                # most keys in the future
    (1, 2048, 2048, 40, 1, None), (1, 700, 700, 64, None, None),                                               # many tiles: two query tiles a CTA
    (1, 2048, 2048, 67, 1, None),                                                                              # groups of unequal numbers of heads
])
def test_every_way_a_forward_is_cut_up(B, Sq, Sk, H, cbs, cache_idx, D):
    """Sizes on both sides of the rule that gives a CTA two query tiles or one, and splits the keys of a few query tiles."""
    _check_call(B, Sq, Sk, H, D, cbs=cbs, cache_idx=cache_idx, grad=Sq * Sk * B * H < 3e8)


@pytest.mark.parametrize("B,Sq,Sk,H,D,cbs,splits", [
    (1, 500, 16384, 16, 128, 0, 2), (1, 128, 4096, 32, 128, 0, 4), (1, 500, 16384, 32, 128, 0, 1), (1, 4096, 4096, 4, 128, 1, 1),
    (1, 12318, 12318, 2, 128, 1, 1), (1, 12269, 12269, 2, 64, 1, 1)])
def test_keys_are_split_as_was_fastest(B, Sq, Sk, H, D, cbs, splits, monkeypatch):
    """The rule's choice where every form was timed: two heads of 12318 causal rows take 106 us on whole rows, 120 with the keys over two CTAs."""
    from ringattention_b200.ops import _lib, flash

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("timed with 148 SMs")
    rule, chosen = _lib.lib().ra_attn_fwd_splits, []
    monkeypatch.setattr(_lib.lib(), "ra_attn_fwd_splits", lambda a: chosen.append(rule(a)) or chosen[-1])
    q, k = (torch.zeros(B, n, H, D, device="cuda", dtype=torch.bfloat16) for n in (Sq, Sk))
    flash.flash_fwd(q, k, k, flash.MaskSpec(causal_block_size=cbs, q_pos=flash.Positions(Sk - Sq), k_pos=flash.Positions(0)))
    assert chosen == [splits]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S,H,q_pos,k_pos", [
    (512, 8, (0,), (0,)),                     # four query tiles a head: two groups on one tile
    (2048, 4, (2048,), (0,)),                 # a block of earlier positions: every tile visible
    (1000, 8, (0, 7168, 512), (512, 6656, 512)),  # two runs of positions a shard, a ragged last tile
    (2048, 40, (0,), (0,)),                   # two query tiles a CTA
])
def test_carry_merged_in_place(S, H, q_pos, k_pos, D):
    """A ring step gives the accumulator and the log-sum-exp of the steps before and has them overwritten by the merged ones:
    the same bits as with tensors of their own, every time."""
    from ringattention_b200.ops import flash

    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v = (torch.randn(1, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    ms = flash.MaskSpec(causal_block_size=1, q_pos=flash.Positions(*q_pos), k_pos=flash.Positions(*k_pos))
    o_prev, lse_prev = torch.randn(1, S, H, D, device="cuda", generator=g), 6 + torch.randn(1, H, S, device="cuda", generator=g)
    lse_prev[0, 0, 3] = -float("inf")  # no key seen yet
    out, lse = flash.flash_fwd(q, k, v, ms, o_prev=o_prev, lse_prev=lse_prev, out_fp32=True)
    alone, lse_alone = flash.flash_fwd(q, k, v, ms, out_fp32=True)
    both = torch.logaddexp(lse_prev.double(), lse_alone.double())
    w = [torch.exp(x.double() - both).nan_to_num(0.0).permute(0, 2, 1)[..., None] for x in (lse_prev, lse_alone)]
    # the launch without a carry may be cut up otherwise: probabilities are rounded to bf16 (2^-9 of each) in both
    assert (out.double() - w[0] * o_prev.double() - w[1] * alone.double()).abs().max() < 2 ** -8 * v.abs().max()
    assert (lse.double() - both)[torch.isfinite(both)].abs().max() < 1e-5
    for _ in range(300):
        o, l = o_prev.clone(), lse_prev.clone()
        flash.flash_fwd(q, k, v, ms, o_prev=o, lse_prev=l, out=o, lse_out=l)
        assert torch.equal(o, out) and torch.equal(l, lse)


def _strange(where, q, k, v):
    """One entry or row that is no ordinary number; key and value 4000 lie in the middle of the cache."""
    if where == "query":
        q[0, 7, 0, 3] = float("nan")
    elif where == "key":
        k[0, 4000, :, 3] = float("nan")
    elif where == "infinite key":  # scores of +inf or -inf, by the query's sign
        k[0, 4000, :, 3] = float("inf")
    elif where == "value":
        v[0, 4000, :, 5] = float("nan")
    elif where == "infinite value":
        v[0, 4000, :, 5] = -float("inf")
    else:  # every key
        k[0, :, 0, 3] = float("nan")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("where", ["query", "key", "infinite key", "value", "infinite value", "every key"])
def test_what_is_no_number_passes_through_a_launch_split_over_the_keys(where, masked, D, monkeypatch):
    """A launch split over the keys gives NaN and infinities, and a log-sum-exp without a number, where one that is not split does, and the
    same numbers elsewhere (probabilities and results are rounded to bf16 on both sides, 2^-8 of the largest entry each). Without a mask also where dense
    attention in 64 bits does. The mask hides key 4000 from some rows, and all keys from one."""
    from ringattention_b200.ops import _lib, flash

    B, Sq, Sk, H = 1, 130, 8000, 2
    g = torch.Generator(device="cuda").manual_seed(D)
    q = torch.randn(B, Sq, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, Sk, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    _strange(where, q, k, v)
    ms = flash.MaskSpec(causal_block_size=0, q_pos=flash.Positions(0), k_pos=flash.Positions(0))
    if masked:
        m = torch.rand(B, 1, Sq, Sk, device="cuda", generator=g) < 0.5
        m[0, 0, 9] = False
        ms.keep_q, ms.keep_k, ms.keep_tiles = flash.mask_bitmaps(m)
    rule, chosen = _lib.lib().ra_attn_fwd_splits, []

    def spy(a):
        chosen.append(rule(a))
        return chosen[-1]

    monkeypatch.setattr(_lib.lib(), "ra_attn_fwd_splits", spy)
    out, lse = flash.flash_fwd(q, k, v, ms)
    assert chosen[0] > 1
    monkeypatch.setattr(_lib.lib(), "ra_attn_fwd_splits", lambda a: 1)
    want, want_lse = flash.flash_fwd(q, k, v, ms)
    out, want = out.float(), want.float()
    for a, b in ((out, want), (lse, want_lse)):
        fin = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fin) and torch.equal(a.isnan(), b.isnan()) and torch.equal(a == float("inf"), b == float("inf"))
        assert not fin.any() or bool(((a - b)[fin].abs() <= 2 ** -6 * b[fin].abs().max() + 1e-6).all())
    if not masked:
        x = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double())
        if where == "infinite key":  # the kernel's score is what fp32 gives
            x = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()).double()
        dense = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x / D ** 0.5, -1), v.double())
        assert torch.equal(out.isnan(), dense.isnan()) and torch.equal(out.isinf(), dense.isinf())
        assert not torch.isfinite(out).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,H", [(256, 1600, 2), (2048, 1600, 19), (130, 8000, 2)])  # one query tile a CTA, two, keys split
@pytest.mark.parametrize("first", ["seen", "hidden"])
def test_rows_that_outgrow_their_reference(first, Sq, Sk, H, D):
    """Scores of a tile are scaled by the reference of the tiles before it as long as no row's sum can hold an entry that outgrows it. Here the logits of a row
    step up by 2 to 800 from tile to tile, or down, or stay, by rows of all kinds side by side in a warp; `hidden`: many rows see no key
    of the first tiles. Against dense attention in 64 bits on the same bf16 numbers: 1e-2 of the largest entry (P and the result are rounded
    once each), the log-sum-exp within 2e-5 of the largest logit (fp32 sums of D products) plus 1e-3."""
    from ringattention_b200.ops import _lib, flash

    g = torch.Generator(device="cuda").manual_seed(Sq + D)
    q = torch.randn(1, Sq, H, D, device="cuda", generator=g)
    k, v = (torch.randn(1, Sk, H, D, device="cuda", generator=g) for _ in range(2))
    q[..., 0] = torch.tensor([1.0, -1.0, 0.0, 0.25, 2.0], device="cuda")[torch.randint(0, 5, (1, Sq, H), device="cuda", generator=g)]
    steps = torch.tensor([0.0, 2.0, 7.0, 7.0, 19.0, 60.0, 30.0, -80.0, 400.0, 390.0, 800.0], device="cuda")
    k[..., 0] = (steps[(torch.arange(Sk, device="cuda") // 128) % steps.numel()] * D ** 0.5)[None, :, None]
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    ms = flash.MaskSpec(causal_block_size=0, q_pos=flash.Positions(0), k_pos=flash.Positions(0))
    m = torch.ones(1, 1, Sq, Sk, dtype=torch.bool, device="cuda")
    if first == "hidden":
        m[0, 0, 1::3, :300] = False
        m[0, 0, 5::7, :1200] = False
        ms.keep_q, ms.keep_k, ms.keep_tiles = flash.mask_bitmaps(m)
    out, lse = flash.flash_fwd(q, k, v, ms)
    _lib.check_status()
    for h in range(H):
        x = (q[0, :, h].double() @ k[0, :, h].double().t() / D ** 0.5).masked_fill(~m[0, 0], -float("inf"))
        want = torch.softmax(x, -1) @ v[0, :, h].double()
        assert (out[0, :, h].double() - want).abs().max() <= 0.01 * want.abs().max()
        assert (lse[0, h].double() - torch.logsumexp(x, -1)).abs().max() <= 2e-5 * x[torch.isfinite(x)].abs().max() + 1e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("grows", [0.0, 7.5, 10.0, 14.0, 40.0])
def test_probabilities_are_rounded_at_the_scale_of_their_row(grows, D):
    """The rule of the reference, which fixes at what scale a probability is rounded to bf16: the first tile's maximum, then the maximum so far
    whenever one row of the 32 of a warp exceeds its own by 2^8. One key of the third tile stands `grows` powers of two above its row.
    Against the same rule in 64 bits: what is left are fp32 sums and roundings that fall the other way, some 3e-5; another scale for the
    rows' probabilities gives 1e-3."""
    from ringattention_b200.ops import _lib, flash

    Sq, Sk, H = 2048, 640, 19  # two query tiles a CTA
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(1, n, H, D, device="cuda", generator=g) for n in (Sq, Sk, Sk))
    q[..., 0], k[..., 0] = 1.0, 0.0
    k[:, 300, :, 0] = grows * math.log(2) * D ** 0.5
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    ms = flash.MaskSpec(causal_block_size=0, q_pos=flash.Positions(0), k_pos=flash.Positions(0))
    out, _ = flash.flash_fwd(q, k, v, ms, out_fp32=True)
    _lib.check_status()
    for h in (0, H - 1):
        x = q[0, :, h].double() @ k[0, :, h].double().t() * (D ** -0.5 / math.log(2))
        m, o, l = None, 0.0, 0.0
        for j in range(0, Sk, 128):
            new = x[:, j:j + 128].amax(1) if m is None else torch.maximum(m, x[:, j:j + 128].amax(1))
            if m is not None:
                new = torch.where((new > m + 8).view(-1, 32).any(1).repeat_interleave(32), new, m)
                o, l = o * torch.exp2(m - new)[:, None], l * torch.exp2(m - new)
            m = new
            p = torch.exp2(x[:, j:j + 128] - m[:, None])
            o, l = o + p.bfloat16().double() @ v[0, j:j + 128, h].double(), l + p.sum(1)
        want = o / l[:, None]
        assert (out[0, :, h].double() - want).norm() <= 2e-4 * want.norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (2, 130, 3), (1, 1000, 2)])
@pytest.mark.parametrize("views", [False, True])
def test_backward_in_one_call(B, S, H, D, views):
    """Preparation, backward and the cast of dQ behind one call against the three one by one (which a phase timer asks for), for gradients of
    their own and for views of one (B, S, 3, H, D) buffer: dK and dV the same bits, dQ (sums in any order) within 2^-7 of its largest entry."""
    from ringattention_b200.ops import _lib, attention as A
    from ringattention_b200.config import BlockwiseKwargs
    from ringattention_b200.utils import tracing

    g = torch.Generator(device="cuda").manual_seed(S)
    buf = torch.randn(B, S, 3, H, D, device="cuda", generator=g).bfloat16()
    q, k, v = buf.unbind(2) if views else (torch.empty(B, S, H, D, device="cuda", dtype=torch.bfloat16).copy_(t) for t in buf.unbind(2))
    dout = torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16()
    plan = A.make_plan(0, 1, B, S, S, H, BlockwiseKwargs(causal_block_size=1, query_chunk_size=S, key_chunk_size=S), device=q.device)
    out, lse = A.ring_forward(q, k, v, plan)
    got, n = [], []
    for timed in (False, True):
        to = torch.full_like(buf, 7.0).unbind(2) if views else (None, None, None)
        n0 = _lib.launches()
        tracing.set_phase_timer(tracing.PhaseTimer() if timed else None)
        try:
            got.append(A.ring_backward(q, k, v, out, lse, dout, plan, dq=to[0], dk=to[1], dv=to[2]))
        finally:
            tracing.set_phase_timer(None)
        n.append(_lib.launches() - n0)
    _lib.check_status()
    (dq, dk, dv), (dq2, dk2, dv2) = got
    assert n[0] == n[1] and torch.equal(dk, dk2) and torch.equal(dv, dv2)
    assert (dq.float() - dq2.float()).abs().max() <= 2 ** -7 * dq2.float().abs().max() + 1e-6
