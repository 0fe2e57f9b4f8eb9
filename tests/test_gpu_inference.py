"""Decode path: split-KV kernel + merge against the dense oracle, small-M linear, and the
inference engine (chunked prefill + greedy decode) against a full PyTorch forward."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 4, 128, 3000), (2, 4, 3, 64, 1111), (1, 8, 2, 128, 700), (1, 3, 2, 128, 500)])
def test_decode_attention_matches_dense(shape):
    import ringattention_b200 as rab
    from ringattention_b200.ops import _lib, decode as Dk, reference as R
    from ringattention_b200.parallel.mesh import resolve_axis

    B, QL, H, D, S = shape
    torch.manual_seed(0)
    q = torch.randn(B, QL, H, D, device="cuda").bfloat16()
    k = torch.randn(B, S, H, D, device="cuda").bfloat16()
    v = torch.randn_like(k)
    mask = torch.rand(B, 1, QL, S, device="cuda") < 0.7
    out = rab.ringattention_inference(q, k, v, mask, None)
    ref = R.dense_attention(q, k, v, extra_masked=~mask, dtype=torch.float32)
    assert (out.float() - ref).abs().max() < 0.02
    # position-driven variant used by the decoding loop: causal rule + partially filled cache
    out2 = Dk.ring_decode_attention(q, k, v, None, resolve_axis(None), n_valid=S - 100, q_pos0=S - 200, k_pos0=0)
    ref2 = R.dense_attention(q, k[:, :S - 100], v[:, :S - 100], torch.arange(S - 200, S - 200 + QL, device="cuda"),
                             torch.arange(S - 100, device="cuda"), causal_block_size=1, dtype=torch.float32)
    assert (out2.float() - ref2).abs().max() < 0.02
    torch.cuda.synchronize()
    _lib.check_status()


def test_decode_fully_masked_rows_are_zero():
    import ringattention_b200 as rab

    q = torch.randn(1, 2, 2, 128, device="cuda").bfloat16()
    k = torch.randn(1, 300, 2, 128, device="cuda").bfloat16()
    mask = torch.zeros(1, 1, 2, 300, dtype=torch.bool, device="cuda")
    mask[0, 0, 1, :17] = True
    out = rab.ringattention_inference(q, k, k, mask, None)
    assert bool((out[:, 0] == 0).all()) and bool(torch.isfinite(out.float()).all())


def test_small_m_linear():
    from ringattention_b200.ops import kernels as K

    torch.manual_seed(1)
    for M in (1, 3, 8):
        x = torch.randn(M, 512, device="cuda").bfloat16()
        w = torch.randn(1000, 512, device="cuda").bfloat16()
        r = torch.randn(M, 1000, device="cuda").bfloat16()
        y = K.small_m_linear(x, w, residual=r)
        ref = x.float() @ w.float().t() + r.float()
        assert (y.float() - ref).abs().max() <= 0.01 * ref.abs().max() + 0.05


def test_small_m_linear_prologues():
    """RMSNorm and SwiGLU applied while the kernel reads x, against plain fp32 PyTorch."""
    from ringattention_b200.ops import kernels as K

    torch.manual_seed(2)
    for M in (1, 4, 8):
        x = torch.randn(M, 1024, device="cuda").bfloat16()
        g = (1 + 0.1 * torch.randn(1024, device="cuda")).bfloat16()
        w = (torch.randn(776, 1024, device="cuda") / 32).bfloat16()
        y = K.norm_linear(x, g, 1e-5, w)
        xf = x.float()
        ref = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * g.float()) @ w.float().t()
        assert (y.float() - ref).abs().max() <= 0.01 * ref.abs().max() + 0.02

        gu = torch.randn(M, 2 * 1024, device="cuda").bfloat16()
        r = torch.randn(M, 776, device="cuda").bfloat16()
        y = K.swiglu_linear(gu, w, residual=r)
        h = (torch.nn.functional.silu(gu[:, :1024].float()) * gu[:, 1024:].float()).bfloat16().float()
        ref = h @ w.float().t() + r.float()
        assert (y.float() - ref).abs().max() <= 0.01 * ref.abs().max() + 0.02
        # the same numbers as the two-launch path: the activation is rounded to bf16 in both
        two = K.small_m_linear(K.swiglu_fwd(gu), w, residual=r)
        assert torch.equal(y, two)


@pytest.mark.parametrize("D,striped", [(128, False), (64, True)])
def test_rope_append_equals_rope_then_append(D, striped):
    from ringattention_b200.ops import kernels as K

    torch.manual_seed(3)
    B, H, S_max = 2, 8, 64
    qkv = torch.randn(B, 1, 3, H, D, device="cuda").bfloat16()
    state = torch.tensor([37, 0], device="cuda", dtype=torch.int64)
    stripe = (2, 1, 16, 32) if striped else None  # decoded token 5 -> rank 1, row 16 + 2
    caches = [torch.zeros(B, 2, H, S_max, D, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    views = [(c[:, 0].transpose(1, 2), c[:, 1].transpose(1, 2)) for c in caches]
    a = qkv.clone()
    K.rope_at_(a.view(B, 1, 3 * H, D)[:, :, :2 * H], state, 10000.0)
    K.kv_append(a, views[0][0], views[0][1], state, stripe=stripe)
    b = qkv.clone()
    K.rope_append(b, views[1][0], views[1][1], state, 10000.0, stripe=stripe)
    assert torch.equal(a, b) and torch.equal(caches[0], caches[1])
    row = 18 if striped else 37
    assert torch.equal(views[1][0][:, row], b[:, 0, 1]) and torch.equal(views[1][1][:, row], b[:, 0, 2])
    written = int(torch.count_nonzero(views[1][0][:, row])) + int(torch.count_nonzero(views[1][1][:, row]))
    assert int(torch.count_nonzero(caches[1])) == written  # no other cache row was touched


def test_merge_exchange_gives_up_on_a_silent_peer_and_still_merges_its_own_rows():
    """The one-launch cross-GPU merge with a second "rank" that never signals (its buffers are local and nobody
    writes them): every row's wait runs out, the status word gets the peer-timeout code, the kernel returns and
    the context keeps working. The silent rank's inbox slots hold lse = -inf, so the merged rows equal this
    rank's own."""
    import ctypes

    from ringattention_b200.ops import _lib
    from ringattention_b200.ops import decode as Dk

    torch.manual_seed(4)
    rows, parts, D, n = 16, 3, 128, 2
    o_part = torch.randn(rows, parts, D, device="cuda")
    lse_part = torch.randn(rows, parts, device="cuda")
    boxes_o = torch.zeros(n, 2, rows, n, D, device="cuda")
    boxes_l = torch.full((n, 2, rows, n), float("-inf"), device="cuda")
    flags = torch.zeros(n, rows, n, dtype=torch.int32, device="cuda")
    sync = torch.zeros(2, dtype=torch.int32, device="cuda")
    tab = lambda t: torch.tensor([t[i].data_ptr() for i in range(n)], dtype=torch.int64, device="cuda")
    to, tl, tf = tab(boxes_o), tab(boxes_l), tab(flags)
    out = torch.empty(rows, D, device="cuda")
    st = _lib.status_tensor()
    st.zero_()
    vp = ctypes.c_void_p
    _lib.call("ra_decode_merge_exchange", vp(o_part.data_ptr()), vp(lse_part.data_ptr()),
              ctypes.c_longlong(parts * D), ctypes.c_longlong(D), ctypes.c_longlong(parts), ctypes.c_longlong(1),
              rows, parts, D, 1, 0, vp(out.data_ptr()), 1, vp(to.data_ptr()), vp(tl.data_ptr()),
              vp(boxes_o[0].data_ptr()), vp(boxes_l[0].data_ptr()), rows, vp(tf.data_ptr()), vp(sync.data_ptr()), n, 0,
              ctypes.c_ulonglong(50_000_000), vp(st.data_ptr()), _lib.stream_ptr())
    torch.cuda.synchronize()
    with pytest.raises(_lib.KernelError, match="peer flag"):
        _lib.check_status()
    assert sync.tolist() == [1, 0]  # the launch counter advanced, the arrival counter is back at zero
    w = torch.softmax(lse_part, dim=1)
    ref = (w[:, :, None] * o_part).sum(1)
    assert (out - ref).abs().max() < 1e-4
    assert Dk.exchange_fits(rows) and not Dk.exchange_fits(10 ** 6)


def test_cuda_core_kernels_still_serve_several_rows(monkeypatch):
    """Calls with 2-8 rows go to the tensor-core kernels by default; with the thresholds raised the CUDA-core
    kernels (which serve one row by default) take them and give the same answers."""
    from ringattention_b200.ops import decode as Dk, kernels as K, reference as R
    from ringattention_b200.parallel.mesh import resolve_axis

    torch.manual_seed(5)
    B, QL, H, D, S = 1, 4, 2, 128, 900
    q = torch.randn(B, QL, H, D, device="cuda").bfloat16()
    k = torch.randn(B, S, H, D, device="cuda").bfloat16()
    v = torch.randn_like(k)
    x = torch.randn(4, 1024, device="cuda").bfloat16()
    g = (1 + 0.1 * torch.randn(1024, device="cuda")).bfloat16()
    w = (torch.randn(520, 1024, device="cuda") / 32).bfloat16()
    outs = []
    for rows in (2, 9):
        monkeypatch.setattr(Dk, "MMA_MIN_ROWS", rows)
        monkeypatch.setattr(K, "LINEAR_MMA_MIN_ROWS", rows)
        o = Dk.ring_decode_attention(q, k, v, None, resolve_axis(None), n_valid=S, q_pos0=S - QL, k_pos0=0)
        outs.append((o.float(), K.norm_linear(x, g, 1e-5, w).float(), K.small_m_linear(x, w).float()))
    ref = R.dense_attention(q, k, v, torch.arange(S - QL, S, device="cuda"), torch.arange(S, device="cuda"),
                            causal_block_size=1, dtype=torch.float32)
    for o, _, _ in outs:
        assert (o - ref).abs().max() < 0.02
    assert (outs[0][1] - outs[1][1]).abs().max() <= 0.02 * outs[1][1].abs().max() + 0.02
    assert (outs[0][2] - outs[1][2]).abs().max() <= 0.01 * outs[1][2].abs().max() + 0.02


def test_prefill_and_greedy_decode_match_full_forward():
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference
    from llama_torch import llama_forward_torch
    from ringattention_b200.ops import _lib

    cfg = LlamaConfig.named("llama-tiny")
    inf = LlamaInference(cfg, max_context=1024, batch=2, seed=5)
    T = 384
    torch.manual_seed(2)
    prompt = torch.randint(0, cfg.vocab_size, (2, T), device="cuda")
    gen, timing = inf.generate(prompt, 8, chunk=128)
    _lib.check_status()
    W = {n: inf.params.w(n) for n in inf.params.index}
    logits = llama_forward_torch(cfg, W, torch.cat([prompt, gen], dim=1).int())
    ref_next = logits[:, T - 1:-1].argmax(-1)
    assert (ref_next == gen).float().mean() >= 0.9
    assert len(timing["decode_ms"]) == 8 and inf.length == T + 8


def test_graph_replayed_decode_equals_eager_decode():
    """The CUDA-graph decode path (device-side position/step) must emit the same tokens as the eager path."""
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference
    from ringattention_b200.ops import _lib

    cfg = LlamaConfig.named("llama-tiny")
    torch.manual_seed(3)
    prompt = torch.randint(0, cfg.vocab_size, (2, 256), device="cuda")
    a = LlamaInference(cfg, max_context=512, batch=2, seed=7)
    b = LlamaInference(cfg, max_context=512, batch=2, seed=7)
    ga, _ = a.generate(prompt, 12, chunk=128, use_graph=True)
    gb, _ = b.generate(prompt, 12, chunk=128, use_graph=False)
    _lib.check_status()
    assert a._graph is not None and b._graph is None
    assert torch.equal(ga, gb)
    assert int(a.state[0].item()) == a.length == 256 + 12


def test_engine_reuse_after_reset_matches_a_fresh_engine():
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference

    cfg = LlamaConfig.named("llama-tiny")
    torch.manual_seed(4)
    p1 = torch.randint(0, cfg.vocab_size, (1, 256), device="cuda")
    p2 = torch.randint(0, cfg.vocab_size, (1, 384), device="cuda")
    eng = LlamaInference(cfg, max_context=1024, batch=1, seed=9)
    eng.generate(p1, 6, chunk=128)
    g2, _ = eng.generate(p2, 6, chunk=128)          # resets, re-records the decode graph
    fresh, _ = LlamaInference(cfg, max_context=1024, batch=1, seed=9).generate(p2, 6, chunk=128)
    assert torch.equal(g2, fresh) and eng.length == 384 + 6


@pytest.mark.parametrize("ql,S,H,D", [(1, 700, 2, 128), (8, 1111, 3, 64), (100, 900, 2, 128), (2048, 1536, 2, 128)])
def test_inference_op_any_query_length_with_gradients(ql, S, H, D):
    """ringattention_inference with a random boolean mask (ringattention_inference.py:8-35) and its VJP (:38-64)
    against dense fp32 attention, for query lengths on both sides of the 8-row decode kernel."""
    import ringattention_b200 as rab
    from ringattention_b200.ops import _lib, reference as R

    B = 2
    torch.manual_seed(ql)
    q, k, v = [torch.randn(B, n, H, D, device="cuda").bfloat16().requires_grad_(True) for n in (ql, S, S)]
    do = torch.randn(B, ql, H, D, device="cuda").bfloat16()
    mask = torch.rand(B, 1, ql, S, device="cuda") < 0.6
    mask[..., 0] = True  # no fully masked row: the dense oracle would average over nothing
    out = rab.ringattention_inference(q, k, v, mask, None)
    out.backward(do)
    qf, kf, vf = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    ref = R.dense_attention(qf, kf, vf, extra_masked=~mask, dtype=torch.float32)
    ref.backward(do.float())
    torch.cuda.synchronize()
    _lib.check_status()
    assert (out.float() - ref).abs().max() < 0.02
    for got, want in ((q.grad, qf.grad), (k.grad, kf.grad), (v.grad, vf.grad)):
        assert (got.float() - want).abs().max() <= 0.02 * want.abs().max() + 1e-3
    # without gradients the short queries take the split-KV decode kernel: same numbers
    with torch.no_grad():
        out2 = rab.ringattention_inference(q, k, v, mask, None)
    assert (out2.float() - ref).abs().max() < 0.02


def test_mask_bitmaps_round_trip():
    from ringattention_b200.ops import flash

    torch.manual_seed(3)
    B, Hm, Sq, Sk = 2, 3, 77, 301
    m = torch.rand(B, Hm, Sq, Sk, device="cuda") < 0.5
    by_q, by_k = flash.pack_mask(m)
    bits = torch.arange(32, device="cuda")
    got_q = ((by_q.unsqueeze(-1) >> bits) & 1).bool().flatten(3)[..., :Sk]        # (B, Hm, Sq, Sk)
    got_k = ((by_k.unsqueeze(-1) >> bits) & 1).bool().flatten(3)[..., :Sq]        # (B, Hm, Sk, Sq)
    assert torch.equal(got_q, m)
    assert torch.equal(got_k, m.transpose(2, 3))
    # padding bits are zero
    assert int(((by_q.unsqueeze(-1) >> bits) & 1).flatten(3)[..., Sk:].sum()) == 0


@pytest.mark.parametrize("ql,cache_idx", [(128, 384), (100, 411), (1, 639)])
def test_cache_idx_on_the_fused_path(ql, cache_idx):
    """``cache_idx``: replicated queries that start at global position ``cache_idx`` against the cache
    (ringattention_jax.py:31-35), causal, on the fused kernels including gradients."""
    import ringattention_b200 as rab
    from ringattention_b200.ops import _lib, reference as R

    B, H, D, Sk = 2, 2, 128, 640
    torch.manual_seed(cache_idx)
    q = torch.randn(B, ql, H, D, device="cuda").bfloat16().requires_grad_(True)
    k = torch.randn(B, Sk, H, D, device="cuda").bfloat16().requires_grad_(True)
    v = torch.randn(B, Sk, H, D, device="cuda").bfloat16().requires_grad_(True)
    do = torch.randn(B, ql, H, D, device="cuda").bfloat16()
    kw = dict(causal_block_size=1, query_chunk_size=128, key_chunk_size=128)
    out = rab.ringattention(q, k, v, None, None, cache_idx, None, True, kw)
    out.backward(do)
    qf, kf, vf = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    ref = R.dense_attention(qf, kf, vf, torch.arange(cache_idx, cache_idx + ql, device="cuda"),
                            torch.arange(Sk, device="cuda"), causal_block_size=1, dtype=torch.float32)
    ref.backward(do.float())
    torch.cuda.synchronize()
    _lib.check_status()
    assert (out.float() - ref).abs().max() < 0.02
    for got, want in ((q.grad, qf.grad), (k.grad, kf.grad), (v.grad, vf.grad)):
        assert (got.float() - want).abs().max() <= 0.02 * want.abs().max() + 1e-3


def test_fallback_to_pytorch_path_warns_once():
    import warnings

    import ringattention_b200 as rab
    from ringattention_b200 import api

    api._WARNED.clear()
    q = torch.randn(1, 64, 2, 64, device="cuda")  # fp32: not served by the kernels
    kw = dict(causal_block_size=1, query_chunk_size=64, key_chunk_size=64)
    with warnings.catch_warnings(record=True) as w:
        warnings.simplefilter("always")
        rab.ringattention(q, q, q, None, None, None, None, True, kw)
        rab.ringattention(q, q, q, None, None, None, None, True, kw)
    assert sum("PyTorch path" in str(x.message) for x in w) == 1


def test_streams_sharing_one_cached_context():
    """Three decode streams on one shared prefix (read once per step for all of them, private tails) against three
    single-stream engines that each cached the prefix themselves; teacher-forced, logits compared step by step."""
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference
    from ringattention_b200.ops import _lib

    cfg = LlamaConfig.named("llama-tiny")
    torch.manual_seed(4)
    prompt = torch.randint(0, cfg.vocab_size, (1, 384), device="cuda")
    shared = LlamaInference(cfg, max_context=1024, batch=1, seed=7, streams=3, max_new_tokens=16)
    logits = None
    for c0 in range(0, 384, 128):
        logits = shared.prefill_chunk(prompt[:, c0:c0 + 128])
    singles = []
    for _ in range(3):
        e = LlamaInference(cfg, max_context=1024, batch=1, seed=7)
        for c0 in range(0, 384, 128):
            e.prefill_chunk(prompt[:, c0:c0 + 128])
        singles.append(e)
    tok = logits[0].topk(3).indices                        # three different continuations
    worst = 0.0
    for _ in range(6):
        la = shared.decode_step(tok)                        # (3, vocab)
        lb = torch.cat([e.decode_step(tok[i:i + 1]) for i, e in enumerate(singles)], dim=0)
        worst = max(worst, ((la - lb).abs().max() / lb.abs().max()).item())
        tok = lb.argmax(dim=-1)
    torch.cuda.synchronize()
    _lib.check_status()
    assert worst < 0.03, worst
    # the graph-replayed path gives the same tokens as the eager one from here on
    shared._tok_buf.copy_(tok.to(torch.int32))
    eager = shared.decode_step(tok).argmax(dim=-1)
    assert eager.shape == (3,)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("nparts,B", [(1, 2), (3, 2), (15, 2), (16, 2), (33, 2), (512, 2), (1100, 2), (2, 170), (8, 170), (20, 170), (31, 170), (32, 170)])
def test_merge_of_few_and_many_partials(nparts, B, D):
    """All forms of the merge: a thread per column (fewer than four partials of 12 rows, fewer than 32 of 1020), 8 and 32 warps; with
    empty partials, a row without any and strided inputs. Tolerance: fp32 weights by exp of a difference below 40, 4e-6 relative, times sums of up to 1100 terms."""
    from ringattention_b200.ops import decode as Dk

    torch.manual_seed(nparts)
    H, QL = 3, 2
    rows = B * H * QL
    o = torch.randn(rows, nparts, D, device="cuda")
    lse = torch.randn(nparts, rows, device="cuda").t() * 5
    if nparts > 1:
        lse[:, nparts // 2] = -float("inf")
    lse[3] = -float("inf")
    out = torch.empty(B, QL, H, D, device="cuda")
    lse_out = torch.empty(rows, device="cuda")
    Dk.merge_partials(o, lse, H, QL, out=out, lse_out=lse_out)
    w = torch.softmax(lse.double(), 1).nan_to_num(0.0)
    want = (w[:, :, None] * o.double()).sum(1).view(B, H, QL, D).permute(0, 2, 1, 3)
    want_l = torch.logsumexp(lse.double(), 1).view(B, H, QL).permute(0, 2, 1).reshape(-1)
    assert (out.double() - want).abs().max() < 2e-5
    fin = torch.isfinite(want_l)
    assert torch.equal(torch.isfinite(lse_out), fin) and (lse_out.double() - want_l)[fin].abs().max() < 1e-5


def test_kinds_of_mask_tiles():
    from ringattention_b200.ops import flash

    m = torch.zeros(1, 2, 300, 333, dtype=torch.bool, device="cuda")
    m[0, 0] = True                       # full, the ragged tiles too
    m[0, 1, :128, 128:256] = True
    m[0, 1, 299, 332] = True
    m[0, 1, 130:200, 5:90] = True
    _, _, tiles = flash.mask_bitmaps(m, want_k=False)
    assert tiles[0, 0].unique().tolist() == [1]
    assert tiles[0, 1].tolist() == [[0, 1, 0], [2, 0, 0], [0, 0, 2]]
    every = torch.ones(1, 1, 300, 333, dtype=torch.bool, device="cuda")
    every[0, 0, 299, 332] = False
    assert flash.mask_bitmaps(every)[2][0, 0].tolist() == [[1, 1, 1], [1, 1, 1], [1, 1, 2]]


@pytest.mark.parametrize("need_grad", [False, True])
@pytest.mark.parametrize("B,ql,S,H,D,kind", [(1, 9, 3000, 2, 64, "causal"), (1, 500, 4096, 4, 128, "causal"), (2, 130, 2049, 3, 64, "holes"),
                                             (1, 300, 1000, 5, 128, "per head"), (2, 64, 5000, 2, 128, "padding"), (1, 16, 9000, 1, 64, "nothing")])
def test_masked_prompt_chunks(B, ql, S, H, D, kind, need_grad):
    """Chunks of a prompt against a longer cache, with masks whose tiles are full, empty and mixed, at sizes where the keys are
    split over several CTAs and where they are not. bf16 in and out: 1e-2 of the largest entry, gradients 2e-2."""
    import ringattention_b200 as rab

    g = torch.Generator(device="cuda").manual_seed(S)
    q, dout = (torch.randn(B, ql, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    at = torch.arange(S, device="cuda")
    if kind == "causal":
        mask = (at[None] <= torch.arange(S - ql, S, device="cuda")[:, None])[None, None]
    elif kind == "holes":
        mask = torch.rand(B, 1, ql, S, device="cuda", generator=g) < 0.5
        mask[:, :, :, 256:512] = False
    elif kind == "per head":
        mask = (torch.rand(1, H, ql, S, device="cuda", generator=g) < 0.9) & (at < 700)
        mask[0, 1] = True
        mask[0, 2, 5] = False
    elif kind == "padding":
        mask = (at[None] < torch.tensor([S, 1300], device="cuda")[:, None])[:, None, None]
    else:
        mask = torch.zeros(1, 1, ql, S, dtype=torch.bool, device="cuda")
        mask[..., 3, 8000] = True
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    x = (torch.einsum("bqhd,bkhd->bhqk", qd, kd) / D ** 0.5).masked_fill(~mask, -float("inf"))
    e = torch.exp(x - x.amax(-1, keepdim=True).clamp_min(-1e300))
    want = torch.einsum("bhqk,bkhd->bqhd", e / e.sum(-1, keepdim=True).clamp_min(1e-300), vd)
    q, k, v = (t.requires_grad_(need_grad) for t in (q, k, v))
    out = rab.ringattention_inference(q, k, v, mask)
    assert (out.double() - want).abs().max() <= 0.01 * want.abs().max() + 1e-3
    if need_grad:
        got = torch.autograd.grad(out, (q, k, v), dout)
        for a, b in zip(got, torch.autograd.grad(want, (qd, kd, vd), dout.double())):
            assert (a.double() - b).abs().max() <= 0.02 * b.abs().max() + 1e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("ql", [1, 2, 5, 8])
@pytest.mark.parametrize("S,kind", [(37, "valid"), (700, "valid"), (5000, "valid"), (9000, "holes"), (40000, "valid"), (513, "per row"), (1000, "nothing")])
def test_decode_skips_rows_nobody_sees(S, kind, ql, D):
    """Cached rows that the mask hides from all query rows hold infinities: they are not read. Masks by query row and head, a batch row that sees nothing. bf16 in and out: 1e-2 of the largest entry."""
    import ringattention_b200 as rab

    B, H = (2, 3) if S < 40000 else (16, 8)  # (ranges too long for the bits: the test below)
    if S >= 40000 and (D, ql) not in ((64, 1), (64, 2)):
        pytest.skip("the long cache once for each kernel")
    g = torch.Generator(device="cuda").manual_seed(S + ql)
    q = torch.randn(B, ql, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    at = torch.arange(S, device="cuda")
    if kind == "valid":
        mask = (at[None] < torch.randint(S // 2, S, (B, 1), device="cuda", generator=g))[:, None, None]
    elif kind == "holes":
        mask = (torch.rand(B, 1, 1, S, device="cuda", generator=g) < 0.3) & (at < 4000)
    elif kind == "per row":
        mask = torch.rand(1, H, ql, S, device="cuda", generator=g) < 0.05
    else:
        mask = torch.ones(B, 1, 1, S, dtype=torch.bool, device="cuda")
        mask[1] = False
    seen = mask.any(2).any(1)  # (B|1, S)
    x = (torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / D ** 0.5).masked_fill(~mask, -float("inf"))
    e = torch.exp(x - x.amax(-1, keepdim=True).clamp_min(-1e300))
    want = torch.einsum("bhqk,bkhd->bqhd", e / e.sum(-1, keepdim=True).clamp_min(1e-300), v.double())
    if kind != "per row":  # rows that some other head sees are read there
        hidden = (~seen).expand(B, S)
        k[hidden], v[hidden] = float("inf"), float("nan")
    with torch.no_grad():
        out = rab.ringattention_inference(q, k, v, mask)
    assert (out.double() - want).abs().max() <= 0.01 * want.abs().max() + 1e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("ql", [1, 2, 8])
@pytest.mark.parametrize("S,off", [(4096, 0), (4097, 0), (4500, 1), (130, 3), (31, 2)])
def test_decode_mask_bits_at_the_edges_of_a_range(S, off, ql, D):
    """One range for all rows: as many as a CTA keeps bits for, one more (the mask is read as it is then), and mask rows that do
    not start at multiples of four bytes. bf16 inputs, probabilities in bf16 at most: 1e-2 of the largest entry."""
    from ringattention_b200.ops import decode as Dk

    g = torch.Generator(device="cuda").manual_seed(S + ql + D)
    H = 2
    q = torch.randn(1, ql, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(1, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    m = (torch.rand(1, H, ql, S + 4, device="cuda", generator=g) < 0.3)[..., off:off + S]
    m[0, 0, 0, :] = False
    o, lse = Dk.decode_partial(q, k, v, mask=m.view(torch.uint8), splits=1)
    out = torch.empty(1, ql, H, D, device="cuda")
    Dk.merge_partials(o, lse, H, ql, out=out)
    x = (torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / D ** 0.5).masked_fill(~m, -float("inf"))
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1).nan_to_num(0.0), v.double())
    assert (out.double() - want).abs().max() <= 0.01 * want.abs().max() + 1e-3


@pytest.mark.parametrize("N,K", [(1, 8), (7, 2040), (8, 2048), (2371, 2056), (4740, 64), (4096, 4096), (130, 5504), (64, 12288), (64, 12296)])
def test_row_products_at_the_edges_of_their_tiles(N, K):
    """One row against few and many columns, K in one, two, four and six chunks, none of them full, and past the last. Sums are fp32
    and the output is rounded to bf16, 2^-8 of the value; f(x) is rounded to bf16 before the product: term i is off by at most
    a_i = 2^-9 |f_i w_i|, the sum by 7 sqrt(sum a_i^2) but once in 10^10 (Hoeffding)."""
    from ringattention_b200.ops import kernels as Kn

    g = torch.Generator(device="cuda").manual_seed(N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, r, gain, x2 = rnd(1, K), rnd(N, K), rnd(1, N), rnd(K), rnd(1, 2 * K)

    def close(got, f, w, r=0.0, rounded=7 * 2.0 ** -9):
        want = f @ w.double().t() + r
        off = rounded * (f.square() @ w.double().square().t()).sqrt() + 2 ** -8 * want.abs() + 1e-5 * K ** 0.5
        assert bool(((got.double() - want).abs() <= off).all())

    close(Kn.linear_auto(x, w, residual=r), x.double(), w, r.double(), rounded=0.0)
    n = x.double() * torch.rsqrt(x.double().square().mean() + 1e-5) * gain.double()
    close(Kn.norm_linear(x, gain, 1e-5, w), n, w)
    close(Kn.swiglu_linear(x2, w, residual=r), torch.nn.functional.silu(x2[:, :K].double()) * x2[:, K:].double(), w, r.double())
    # the gated pair: gate and up are rounded as the two-launch form rounds them; where a sum's order puts one across a rounding
    # border, h moves by 2^-8 of its value: twice the error of one rounding
    F = max(8, N // 8 * 8)
    wgu, wd, r = (rnd(2 * F, K).double() * K ** -0.5).bfloat16(), rnd(40, F), rnd(1, 40)
    gu = Kn.norm_linear(x, gain, 1e-5, wgu).double()
    h = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    close(Kn.norm_swiglu_linear(x, gain, 1e-5, wgu, wd, residual=r), h, wd, r.double(), rounded=7 * 3 * 2.0 ** -9)


def test_recorded_step_is_kept_over_prompts_and_dropped_with_the_weights():
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference

    cfg = LlamaConfig.named("llama-tiny")
    torch.manual_seed(6)
    prompts = [torch.randint(0, cfg.vocab_size, (2, n), device="cuda") for n in (256, 128, 384)]
    fresh = lambda seed, p: LlamaInference(cfg, max_context=1024, batch=2, seed=seed).generate(p, 7)[0]
    eng = LlamaInference(cfg, max_context=1024, batch=2, seed=9)
    assert torch.equal(eng.generate(prompts[0], 7)[0], fresh(9, prompts[0]))
    graph = eng._graph
    assert torch.equal(eng.generate(prompts[1], 7)[0], fresh(9, prompts[1])) and eng._graph is graph
    eng.decode_step(torch.zeros(2, dtype=torch.int64, device="cuda"))  # an eager step between replays
    eng.reset()
    other = LlamaInference(cfg, max_context=1024, batch=2, seed=5).params
    eng.params = other
    assert torch.equal(eng.generate(prompts[2], 7)[0], fresh(5, prompts[2])) and eng._graph is not graph
    graph = eng._graph
    eng.params.p16_rep.mul_(1.5)  # in place: the recorded step reads what is there
    want = LlamaInference(cfg, max_context=1024, batch=2, params=other).generate(prompts[0], 7)[0]
    assert torch.equal(eng.generate(prompts[0], 7)[0], want) and eng._graph is graph


@pytest.mark.parametrize("Sq,Sk", [(1, 16), (4, 144), (130, 272), (300, 4096), (33, 500), (2, 2040)])
def test_mask_rows_at_multiples_of_sixteen_bytes(Sq, Sk):
    """The bitmaps and kinds of tiles of a mask do not depend on where its rows start: rows at multiples of 16 bytes (whole and ragged
    ends), rows that are not, a row shared by all queries, and bytes of any value."""
    from ringattention_b200.ops import flash

    g = torch.Generator(device="cuda").manual_seed(Sq + Sk)
    B, H, ld = 2, 3, (Sk + 15) // 16 * 16 + 16
    m = torch.randint(0, 256, (B, H, Sq, Sk), device="cuda", generator=g, dtype=torch.uint8)
    m *= torch.rand(B, H, Sq, Sk, device="cuda", generator=g) < 0.4
    m[0, 0], m[0, 1] = 0, 128
    room = torch.full((B, H, Sq, ld + 1), 7, device="cuda", dtype=torch.uint8)
    at16 = torch.full((B, H, Sq, ld), 9, device="cuda", dtype=torch.uint8)
    odd = room[..., 1:1 + Sk]
    odd.copy_(m)
    at16[..., :Sk].copy_(m)
    for a, b in zip(flash.mask_bitmaps(at16[..., :Sk]), flash.mask_bitmaps(odd)):
        assert torch.equal(a, b)
    want = torch.zeros(B, H, Sq, 128 * ((Sk + 127) // 128), device="cuda", dtype=torch.int64)
    want[..., :Sk] = m != 0
    words = (want.view(B, H, Sq, -1, 32) << torch.arange(32, device="cuda")).sum(-1)
    assert torch.equal(flash.mask_bitmaps(at16[..., :Sk])[0].long() & 0xffffffff, words)
    one = at16[:, :, :1, :Sk].expand(B, H, Sq, Sk)
    for a, b in zip(flash.mask_bitmaps(one), flash.mask_bitmaps(odd[:, :, :1].expand(B, H, Sq, Sk))):
        assert torch.equal(a, b)


def test_recording_a_step_when_memory_is_short(monkeypatch):
    """With little free memory the allocator's cached blocks are given back before a step is recorded, with enough they stay; a
    recording that runs out of memory all the same is made again without them."""
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models import engine
    from ringattention_b200.models.llama_infer import LlamaInference

    cfg = LlamaConfig.named("llama-tiny")
    prompt = torch.randint(0, cfg.vocab_size, (2, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    want = LlamaInference(cfg, max_context=512, batch=2, seed=4).generate(prompt, 6, use_graph=False)[0]
    cached = 256 << 20
    for room, fails in ((1 << 60, 0), (0, 0), (0, 1)):
        monkeypatch.setattr(engine, "RECORD_ROOM", room)
        eng = LlamaInference(cfg, max_context=512, batch=2, seed=4)
        step, calls = eng._greedy_step, []

        def body():
            calls.append(torch.empty(8 << 20, dtype=torch.uint8, device="cuda").numel())  # out of the recording's pool
            if len(calls) <= fails:
                raise torch.OutOfMemoryError("no memory")
            step()

        eng._greedy_step = body
        eng.generate(prompt, 3, use_graph=False)  # buffers and kernels exist
        block = torch.empty(cached, dtype=torch.uint8, device="cuda")
        del block
        held = torch.cuda.memory_reserved()
        assert torch.equal(eng.generate(prompt, 6)[0], want) and len(calls) == 1 + fails
        given_back = torch.cuda.memory_reserved() < held - cached // 2
        assert given_back == (room > 0 or fails > 0)


@pytest.mark.parametrize("rows,n", [(1, 1), (1, 3), (2, 31), (3, 1023), (8, 32000), (1, 50257), (4, 4096)])
@pytest.mark.parametrize("kind", ["random", "ties", "nan", "hidden", "view"])
def test_greedy_tokens(rows, n, kind):
    """The same column as argmax: the first of equal ones (zeros of both signs among them), a NaN before any number, rows of -inf."""
    from ringattention_b200.ops import kernels as K

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, n + 5, device="cuda", generator=g)
    x = x[:, 1:n + 1] if kind == "view" else x[:, :n].contiguous()
    if kind == "ties":
        x = x.round().clamp(-1, 0) * torch.tensor([1.0, -0.0], device="cuda")[torch.randint(0, 2, x.shape, device="cuda", generator=g)]
    elif kind == "nan":
        x[:, n // 2:][torch.rand(rows, n - n // 2, device="cuda", generator=g) < 0.1] = float("nan")
    elif kind == "hidden":
        x[:] = -float("inf")
        x[0, n - 1] = -3e38
    out = torch.full((rows,), -7, device="cuda", dtype=torch.int32)
    assert torch.equal(K.greedy(x, out).long(), x.argmax(-1))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("QL", [1, 3, 8])
@pytest.mark.parametrize("kind", ["filled", "filled, by query", "starts late", "a hole"])
def test_masked_decode_of_filled_ranges(kind, QL, D):
    """Ranges of the cache that are seen up to a place are read without asking for their rows one by one: ends on both sides of words of bits
    and of ranges, other ends for other queries (not plain then), rows hidden at the start and in the middle. What nobody sees holds NaN.
    Within 2^-6 of the largest entry of dense attention in 64 bits (P and the result are rounded to bf16)."""
    import ringattention_b200 as rab

    ends = [1, 31, 32, 33, 127, 128, 129, 1000, 1599, 1600]
    B, S, H = len(ends), 1600, 3
    g = torch.Generator(device="cuda").manual_seed(QL)
    q = torch.randn(B, QL, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    at = torch.arange(S, device="cuda")
    m = (at[None] < torch.tensor(ends, device="cuda")[:, None])[:, None, None].expand(B, 1, QL, S).clone()
    if kind == "filled, by query":
        m[:, :, -1:] &= at < 700
    elif kind == "starts late":
        m &= (at >= 40) | (m.sum(-1, keepdim=True) <= 40)
    elif kind == "a hole":
        m[..., 45:47] = False
    else:
        m = m[:, :, :1]
    dead = ~m.any(2)[:, 0]
    k[dead], v[dead] = float("nan"), float("nan")
    got = rab.ringattention_inference(q, k, v, m).double()
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), torch.nan_to_num(k.double())) / D ** 0.5
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x.masked_fill(~m, -float("inf")), -1), torch.nan_to_num(v.double()))
    assert torch.isfinite(got).all() and (got - want).abs().max() <= 2 ** -6 * want.abs().max()


def test_nothing_is_launched_first_inside_a_capture(monkeypatch):
    """A kernel that is loaded while a step is recorded holds up a process's first prompt: the one that only recorded steps use runs before."""
    from ringattention_b200.config import LlamaConfig
    from ringattention_b200.models.llama_infer import LlamaInference
    from ringattention_b200.ops import kernels as K

    capturing, greedy = [], K.greedy
    monkeypatch.setattr(K, "greedy", lambda *a: capturing.append(torch.cuda.is_current_stream_capturing()) or greedy(*a))
    eng = LlamaInference(LlamaConfig.named("llama-tiny"), max_context=256, batch=2, device="cuda")
    eng.generate(torch.randint(0, 100, (2, 128), device="cuda"), 5)
    assert capturing == [False, True]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("QL", [1, 3, 8])
@pytest.mark.parametrize("odd", [False, True])
def test_masked_decode_of_caches_padded_on_either_side(odd, QL, D):
    """One interval of the cache is seen, the same by every query row: it is read without asking for its rows. Its ends lie on both sides of words of
    bits and of ranges; `odd`: rows of the mask at addresses of any alignment. What nobody sees holds NaN. Tolerance as above."""
    import ringattention_b200 as rab

    spans = [(0, 1600), (1, 1600), (31, 32), (32, 33), (33, 127), (127, 129), (128, 1000), (500, 1599), (1599, 1600), (700, 701)]
    B, S, H = len(spans), 1600, 3
    g = torch.Generator(device="cuda").manual_seed(QL)
    q = torch.randn(B, QL, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    wide = torch.zeros(B, 1, 1, S + 1, device="cuda", dtype=torch.bool)
    m = wide[..., 1:] if odd else wide[..., :S].contiguous()
    for b, (lo, hi) in enumerate(spans):
        m[b, ..., lo:hi] = True
    dead = ~m[:, 0, 0]
    k[dead], v[dead] = float("nan"), float("nan")
    got = rab.ringattention_inference(q, k, v, m).double()
    x = torch.einsum("bqhd,bkhd->bhqk", q.double(), torch.nan_to_num(k.double())) / D ** 0.5
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x.masked_fill(~m, -float("inf")), -1), torch.nan_to_num(v.double()))
    assert torch.isfinite(got).all() and (got - want).abs().max() <= 2 ** -6 * want.abs().max()
