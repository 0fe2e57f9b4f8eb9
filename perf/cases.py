"""The workloads whose speed this library is judged by, one dict of plain values each.

Five kinds of work, all through the public entry points:

``attention``   ``ringattention`` on one GPU: a training step's forward and backward, or the forward alone
                (evaluation), causal or not, with packed documents or a padding bias;
``inference``   ``ringattention_inference`` over a cache: one to eight new rows (decoding), or a chunk of a prompt;
``ffn``         ``blockwise_feedforward`` over ``FusedSwiGLU``: forward and backward, or the forward alone;
``train``       ``Trainer.train_step`` of a LLaMA decoder: host batch in, loss out, gradients and weights updated;
``generate``    ``LlamaInference``: prompt in, greedy tokens out, and the logits of one more given token.

``listed()`` are the cases that are always looked at, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes
what a program has in hand before the call, ``run`` is one pass, ``exact`` the same in 64 bits with plain torch.
"""
import math

import torch
import torch.nn.functional as F

DEV = "cuda"


def listed():
    return [
        # a short step, as in fine-tuning on short texts or in this library's own tests: launches and host work count
        dict(name="attention 512 tokens", kind="attention", B=2, S=512, H=8, D=64, causal=True, docs=0, pad=False, grad=True),
        # a batch of unequal lengths, padded on the right: a length that is no multiple of any tile, and a key bias
        dict(name="attention odd padded", kind="attention", B=3, S=1371, H=12, D=64, causal=True, docs=0, pad=True, grad=True),
        # the context of an ordinary LLaMA pre-training step
        dict(name="attention 4K", kind="attention", B=1, S=4096, H=32, D=128, causal=True, docs=0, pad=False, grad=True),
        # long context out of packed documents (segment ids), as the trainer makes it
        dict(name="attention packed 16K", kind="attention", B=1, S=16384, H=16, D=128, causal=True, docs=2048, pad=False, grad=True),
        # one GPU's share of a long-context step: the operator benchmark's size
        dict(name="attention 32K", kind="attention", B=1, S=32768, H=32, D=128, causal=True, docs=0, pad=False, grad=True),
        # decoding a batch of chats of unequal lengths
        dict(name="decode batch 8", kind="inference", B=8, Q=1, S=4000, H=32, D=128, mask="valid"),
        # decoding at the end of a long document: one GPU's shard of a million-token cache
        dict(name="decode 128K", kind="inference", B=1, Q=1, S=131072, H=32, D=128, mask="none"),
        # a chunk of a prompt against what is already cached, with its causal mask
        dict(name="prompt chunk", kind="inference", B=1, Q=500, S=16384, H=32, D=128, mask="causal"),
        # feed-forward of a small model over a short batch
        dict(name="ffn 1024", kind="ffn", B=1, S=512, d=1024, F=2816, chunk=512, grad=True),
        # feed-forward of the 7B model in chunks
        dict(name="ffn 4096", kind="ffn", B=1, S=8192, d=4096, F=11008, chunk=4096, grad=True),
        # a whole training step of a small decoder: embedding to optimizer
        dict(name="train step", kind="train", B=1, S=4096, d=1024, L=4, H=8, F=2816, V=8192, docs=0),
        # a chat turn on half of the 1B model's layers: prompt, greedy tokens, next logits
        dict(name="generate", kind="generate", B=1, S=2048, new=32, d=2048, L=8, H=16, F=5504, V=32000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention"] * 5 + ["inference"] * 3 + ["ffn"] * 2 + ["train", "generate"])
    if kind == "attention":
        D, H = rng.choice([64, 128]), rng.choice([4, 8, 12, 16, 32])
        B, S = rng.choice([1, 1, 2, 3]), _log_int(rng, 200, 32768)
        if rng.random() < 0.5:
            S = max(256, S // 256 * 256)
        while B * H * S * S * D > 32 * 32768 * 32768 * 128 // 3:
            S = S // 2
        kind2 = rng.choice(["causal", "causal", "docs", "pad", "full"])
        return dict(kind=kind, B=B, S=S, H=H, D=D, causal=kind2 != "full", docs=max(64, S // 8) if kind2 == "docs" else 0,
                    pad=kind2 == "pad", grad=rng.random() < 0.75)
    if kind == "inference":
        D, H = rng.choice([64, 128]), rng.choice([8, 16, 32])
        if rng.random() < 0.65:
            B, Q, S, mask = rng.choice([1, 1, 2, 4, 8, 16]), rng.choice([1, 1, 1, 2, 4, 5, 8]), _log_int(rng, 300, 131072), rng.choice(["none", "valid"])
        else:
            B, Q, S, mask = rng.choice([1, 1, 2]), _log_int(rng, 16, 2048), _log_int(rng, 2048, 65536), "causal"
        while B * H * S * D > 131072 * 32 * 128:
            S = S // 2 + 1
        return dict(kind=kind, B=B, Q=Q, S=max(S, Q), H=H, D=D, mask=mask)
    if kind == "ffn":
        d, ff = rng.choice([(512, 1536), (1024, 2816), (2048, 5504), (4096, 11008)])
        chunk = rng.choice([128, 256, 384, 512, 1000, 2048, 4096])
        n = max(1, _log_int(rng, 128, 8192) // chunk)
        return dict(kind=kind, B=rng.choice([1, 1, 2]), S=chunk * min(n, 8), d=d, F=ff, chunk=chunk, grad=rng.random() < 0.7)
    if kind == "train":
        d, H, ff = rng.choice([(512, 4, 1536), (512, 8, 1536), (1024, 8, 2816), (2048, 16, 5504)])
        S = rng.choice([512, 1024, 2048, 4096])
        return dict(kind=kind, B=rng.choice([1, 2]), S=S, d=d, L=rng.choice([2, 3, 4]), H=H, F=ff, V=rng.choice([4096, 8192, 32000]),
                    docs=rng.choice([0, 0, S // 4]))
    d, H, ff = rng.choice([(1024, 8, 2816), (2048, 16, 5504), (4096, 32, 11008)])
    return dict(kind=kind, B=rng.choice([1, 1, 2, 4, 8]), S=128 * _log_int(rng, 1, 32), new=rng.choice([8, 16, 32]), d=d, L=rng.choice([2, 4, 8]),
                H=H, F=ff, V=32000)


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, device=DEV, generator=g, dtype=torch.float32).to(torch.bfloat16)


def _segments(case, seed):
    """Packed documents with a mean length of ``docs`` tokens: ids that grow along the sequence."""
    if not case["docs"]:
        return None
    g = torch.Generator()
    g.manual_seed(int(seed) + 7)
    new = torch.rand(case["B"], case["S"], generator=g) < 1.0 / case["docs"]
    new[:, 0] = False
    return new.int().cumsum(1).int()


def prepare(case, seed):
    return {"attention": _prepare_attention, "inference": _prepare_inference, "ffn": _prepare_ffn, "train": _prepare_train,
            "generate": _prepare_generate}[case["kind"]](case, seed)


def _prepare_attention(case, seed):
    B, S, H, D = case["B"], case["S"], case["H"], case["D"]
    g = _gen(seed)
    q, k, v, dout = (_randn(g, B, S, H, D) for _ in range(4))
    bias = None
    if case["pad"]:  # rows of the batch end at lengths of their own
        n = torch.randint(S // 2, S + 1, (B,), device=DEV, generator=g)
        bias = torch.zeros(B, 1, 1, S, device=DEV).masked_fill_(torch.arange(S, device=DEV)[None, None, None] >= n[:, None, None, None],
                                                              torch.finfo(torch.float32).min)
    seg = _segments(case, seed)
    kw = dict(causal_block_size=1 if case["causal"] else None, query_chunk_size=S, key_chunk_size=S, deterministic=True, dropout_rng=None,
              attn_pdrop=0.0, dtype=torch.float32, policy="nothing_saveable", precision=None, prevent_cse=True)
    return dict(case=case, q=q.requires_grad_(case["grad"]), k=k.requires_grad_(case["grad"]), v=v.requires_grad_(case["grad"]), dout=dout,
                bias=bias, seg=None if seg is None else seg.to(DEV), kw=kw)


def _prepare_inference(case, seed):
    B, Q, S, H, D = case["B"], case["Q"], case["S"], case["H"], case["D"]
    g = _gen(seed)
    q, k, v = _randn(g, B, Q, H, D), _randn(g, B, S, H, D), _randn(g, B, S, H, D)
    mask = None
    if case["mask"] == "valid":  # each row of the batch has filled its cache up to a place of its own
        n = torch.randint(S // 2, S + 1, (B,), device=DEV, generator=g)
        mask = torch.arange(S, device=DEV)[None, None, None] < n[:, None, None, None]
    elif case["mask"] == "causal":  # the chunk's rows are the last Q of the S cached ones
        mask = (torch.arange(S, device=DEV)[None] <= torch.arange(S - Q, S, device=DEV)[:, None])[None, None]
    return dict(case=case, q=q, k=k, v=v, mask=mask)


def _prepare_ffn(case, seed):
    from ringattention_b200.ops.ffn import FusedSwiGLU

    g = _gen(seed)
    ffn = FusedSwiGLU(case["d"], case["F"], device=DEV, seed=int(seed) % (1 << 30))
    x, dy = _randn(g, case["B"], case["S"], case["d"]), _randn(g, case["B"], case["S"], case["d"])
    return dict(case=case, ffn=ffn, x=x.requires_grad_(case["grad"]), dy=dy)


def _config(case):
    from ringattention_b200 import LlamaConfig

    return LlamaConfig(vocab_size=case["V"], d_model=case["d"], n_layers=case["L"], n_heads=case["H"], d_ff=case["F"], ffn_chunk_size=2048,
                       loss_chunk_size=2048)


def _prepare_train(case, seed):
    from ringattention_b200 import TrainConfig
    from ringattention_b200.trainer import Trainer

    tc = TrainConfig(model="", seq_len=case["S"], global_batch=case["B"], seed=int(seed) % (1 << 20), packed_mean_doc_len=case["docs"])
    t = Trainer(_config(case), tc)
    g = torch.Generator()
    g.manual_seed(int(seed) + 3)
    tokens = torch.randint(0, case["V"], (case["B"], case["S"]), generator=g, dtype=torch.int32)
    targets = torch.full_like(tokens, -1)
    targets[:, :-1] = tokens[:, 1:]
    seg = _segments(case, seed)
    if seg is not None:  # no target across the end of a document
        targets[:, :-1][seg[:, 1:] != seg[:, :-1]] = -1
    return dict(case=case, trainer=t, tokens=tokens, targets=targets, seg=seg)


def _prepare_generate(case, seed):
    """A decoder that is sure of its next token, as a trained one is on easy text: its head knows, for each token, the one that
    follows. The greedy tokens then do not hang on roundings; the logits still depend on every layer."""
    from ringattention_b200.models.llama_infer import LlamaInference

    g = _gen(seed)
    B, S, V, d = case["B"], case["S"], case["V"], case["d"]
    room = (S + case["new"] + 8 + 127) // 128 * 128
    eng = LlamaInference(_config(case), max_context=room, batch=B, device=DEV, seed=int(seed) % (1 << 20))
    after = torch.randperm(V, device=DEV, generator=g)
    embed = _randn(g, V, d)
    eng.params.w("embed").copy_(embed)
    eng.params.w("lm_head")[after] = embed * 0.02
    prompt = torch.randint(0, V, (B, S), device=DEV, generator=g)
    return dict(case=case, engine=eng, prompt=prompt, following=torch.randint(0, V, (B,), device=DEV, generator=g))


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    import ringattention_b200 as rab

    case = s["case"]
    if case["kind"] == "attention":
        if not case["grad"]:
            with torch.no_grad():
                return rab.ringattention(s["q"], s["k"], s["v"], s["bias"], s["seg"], None, None, True, s["kw"])
        out = rab.ringattention(s["q"], s["k"], s["v"], s["bias"], s["seg"], None, None, True, s["kw"])
        return dict(out=out, grads=torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"]))
    if case["kind"] == "inference":
        with torch.no_grad():
            return rab.ringattention_inference(s["q"], s["k"], s["v"], s["mask"])
    if case["kind"] == "ffn":
        if not case["grad"]:
            with torch.no_grad():
                return rab.blockwise_feedforward(s["ffn"], s["x"], case["chunk"], pre_remat=False)
        y = rab.blockwise_feedforward(s["ffn"], s["x"], case["chunk"], pre_remat=False)
        return dict(y=y, grads=torch.autograd.grad(y, (s["x"], s["ffn"].weight_gate_up, s["ffn"].weight_down), s["dy"]))
    if case["kind"] == "train":
        loss = s["trainer"].train_step(s["tokens"], s["targets"], s["seg"])
        P = s["trainer"].model.params
        return dict(loss=loss, grads=P.g32, weights=P.p32_s, weights_rep=P.p32_r)
    tokens, _ = s["engine"].generate(s["prompt"], case["new"])
    return dict(tokens=tokens, logits=s["engine"].decode_step(s["following"]))


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(case):
    """Visible (query, key) pairs of one head, over the batch."""
    B, S = case["B"], case["S"]
    if case.get("docs"):
        n = min(S, case["docs"])  # documents of geometric length: mean n, mean square about 2 n^2
        return B * S * min(n, (S + 1) / 2)
    return B * S * (S + 1) / 2 if case.get("causal", True) else B * S * S


def work(case):
    if case["kind"] == "attention":
        B, S, H, D = case["B"], case["S"], case["H"], case["D"]
        rows = B * S * H * D * 2
        return dict(bytes=(8 if case["grad"] else 4) * rows, flops=(14 if case["grad"] else 4) * _pairs(case) * H * D)
    if case["kind"] == "inference":
        B, Q, S, H, D = case["B"], case["Q"], case["S"], case["H"], case["D"]
        pairs = {"none": B * Q * S, "valid": B * Q * S * 0.75, "causal": B * Q * (S - (Q - 1) / 2)}[case["mask"]]
        keys = B * S * (0.75 if case["mask"] == "valid" else 1.0)
        return dict(bytes=4 * keys * H * D + 4 * B * Q * H * D, flops=4 * pairs * H * D)
    if case["kind"] == "ffn":
        rows, n = case["B"] * case["S"], 3 * case["d"] * case["F"]
        return dict(bytes=(4 if case["grad"] else 2) * n + (8 if case["grad"] else 4) * rows * case["d"], flops=(6 if case["grad"] else 2) * rows * n)
    d, L, ff, V, B, S = case["d"], case["L"], case["F"], case["V"], case["B"], case["S"]
    layer = 4 * d * d + 3 * d * ff
    if case["kind"] == "train":
        n = L * layer + V * d
        # bf16 weights read and written; fp32 gradients written; fp32 master weights and two moments read and written
        return dict(bytes=(n + V * d) * (2 + 2 + 4 + 24), flops=6 * n * B * S + 12 * L * d * _pairs(case))
    steps, n = case["new"] + 1, L * layer
    kv = 4 * L * d * B
    return dict(bytes=2 * n + 2 * (steps + 1) * V * d + steps * (2 * n + kv * (S + steps / 2)) + kv * S,
                flops=2 * B * (S + steps) * n + 2 * B * (steps + 1) * V * d + 4 * L * d * B * (S * S / 2 + steps * S))


def tolerance(case):
    """bf16 inputs and outputs, 32-bit sums."""
    if case["kind"] in ("attention", "inference", "ffn"):
        return {"rel": 0.01, "max": 0.2}
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    s = prepare(case, seed)
    return {"attention": _exact_attention, "inference": _exact_inference, "ffn": _exact_ffn, "train": _exact_train,
            "generate": _exact_generate}[case["kind"]](case, s)


def _dense(q, k, v, hide, dout=None, rows=2048):
    """Attention of one head and batch row in 64 bits: ``q (Sq, D)``; ``hide(r0, r1)`` is the mask of the hidden pairs of these
    query rows. With ``dout`` the gradients too."""
    scale = 1.0 / math.sqrt(q.shape[1])
    out = torch.empty_like(q)
    dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for r0 in range(0, q.shape[0], rows):
        r1 = min(q.shape[0], r0 + rows)
        x = (q[r0:r1] @ k.t()) * scale
        m = hide(r0, r1)
        if m is not None:
            x.masked_fill_(m, -math.inf)
        p = torch.softmax(x, -1)
        out[r0:r1] = p @ v
        if dout is not None:
            g = dout[r0:r1]
            dv += p.t() @ g
            ds = p * (g @ v.t() - (g * out[r0:r1]).sum(-1, keepdim=True)) * scale
            dq[r0:r1] = ds @ k
            dk += ds.t() @ q[r0:r1]
    return (out,) if dout is None else (out, dq, dk, dv)


def _exact_attention(case, s):
    B, S, H, D = case["B"], case["S"], case["H"], case["D"]
    got = [torch.empty(B, S, H, D, device=DEV, dtype=torch.float64) for _ in range(4 if case["grad"] else 1)]
    at = torch.arange(S, device=DEV)
    for b in range(B):
        def hide(r0, r1):
            m = torch.zeros(r1 - r0, S, dtype=torch.bool, device=DEV)
            if case["causal"]:
                m |= at[None] > at[r0:r1, None]
            if s["seg"] is not None:
                m |= s["seg"][b, r0:r1, None] != s["seg"][b][None]
            if s["bias"] is not None:
                m |= s["bias"][b, 0, 0][None] < 0
            return m
        for h in range(H):
            r = _dense(*(t.detach()[b, :, h].double() for t in (s["q"], s["k"], s["v"])), hide, s["dout"][b, :, h].double() if case["grad"] else None)
            for t, x in zip(got, r):
                t[b, :, h] = x
    return dict(out=got[0], grads=tuple(got[1:])) if case["grad"] else got[0]


def _exact_inference(case, s):
    B, Q, H, D = case["B"], case["Q"], case["H"], case["D"]
    got = torch.empty(B, Q, H, D, device=DEV, dtype=torch.float64)
    for b in range(B):
        m = None if s["mask"] is None else s["mask"][b if s["mask"].shape[0] > 1 else 0, 0]
        for h in range(H):
            got[b, :, h] = _dense(*(t[b, :, h].double() for t in (s["q"], s["k"], s["v"])),
                                  lambda r0, r1: None if m is None else ~(m if m.shape[0] == 1 else m[r0:r1]))[0]
    return got


def _swiglu(x, wgu, wd):
    gu = x @ wgu.t()
    n = wgu.shape[0] // 2
    return (F.silu(gu[..., :n]) * gu[..., n:]) @ wd.t()


def _exact_ffn(case, s):
    x, wgu, wd = (t.detach().double().requires_grad_(case["grad"]) for t in (s["x"], s["ffn"].weight_gate_up, s["ffn"].weight_down))
    y = _swiglu(x, wgu, wd)
    if not case["grad"]:
        return y
    return dict(y=y.detach(), grads=torch.autograd.grad(y, (x, wgu, wd), s["dy"].double()))


def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, theta):
    """``x (S, H, D)``: pairs (i, i + D/2) turned by position * theta^(-2i/D)."""
    S, _, D = x.shape
    inv = theta ** (-2.0 * torch.arange(D // 2, device=x.device, dtype=torch.float64) / D)
    a = torch.arange(S, device=x.device, dtype=torch.float64)[:, None, None] * inv
    u, w = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin()], -1)


def _decoder(case, cfg, W, tokens, seg=None):
    """Final normalised rows ``(S, d)`` of one sequence; ``W`` names the weights as the library does."""
    S, H, d = tokens.numel(), case["H"], case["d"]
    x = W["embed"][tokens.long()]
    at = torch.arange(S, device=DEV)
    hide = at[None] > at[:, None]
    if seg is not None:
        hide = hide | (seg[:, None] != seg[None])
    for l in range(case["L"]):
        qkv = (_norm(x, W[f"l{l}.n1"], cfg.rms_eps) @ W[f"l{l}.wqkv"].t()).view(S, 3, H, d // H)
        q, k, v = _rotate(qkv[:, 0], cfg.rope_theta), _rotate(qkv[:, 1], cfg.rope_theta), qkv[:, 2]
        p = torch.softmax((torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(d // H)).masked_fill(hide, -math.inf), -1)
        x = x + torch.einsum("hqk,khd->qhd", p, v).reshape(S, d) @ W[f"l{l}.wo"].t()
        x = x + _swiglu(_norm(x, W[f"l{l}.n2"], cfg.rms_eps), W[f"l{l}.wgu"], W[f"l{l}.wd"])
    return _norm(x, W["nf"], cfg.rms_eps)


def _exact_train(case, s):
    t = s["trainer"]
    P, tc = t.model.params, t.tc
    W = {n: P.w(n).double().requires_grad_() for n in list(P.mat) + list(P.rep)}
    loss = 0.0
    for b in range(case["B"]):
        seg = None if s["seg"] is None else s["seg"][b].to(DEV)
        logits = _decoder(case, t.cfg, W, s["tokens"][b].to(DEV), seg) @ W["lm_head"].t()
        tgt = s["targets"][b].to(DEV).long()
        loss = loss + F.cross_entropy(logits[tgt >= 0], tgt[tgt >= 0], reduction="sum") / (case["B"] * case["S"])
    loss.backward()
    # the flat buffers, as the optimizer sees them
    g_s, g_r = torch.zeros(P.numel_shard, device=DEV, dtype=torch.float64), torch.zeros(P.numel_rep, device=DEV, dtype=torch.float64)
    for n, (off, *_) in P.mat.items():
        g_s[off:off + W[n].numel()] = W[n].grad.reshape(-1)
    for n, (off, _) in P.rep.items():
        g_r[off:off + W[n].numel()] = W[n].grad.reshape(-1)
    norm = math.sqrt(float(g_s.square().sum() + g_r.square().sum()))
    clip = min(1.0, tc.grad_clip / (norm + 1e-6))

    def adamw(p, g, decay_end):  # the first step: both moments start from zero
        p, g = p.double(), g * clip
        decay = torch.where(torch.arange(p.numel(), device=DEV) < decay_end, tc.weight_decay, 0.0)
        return p - tc.lr * (g / (g.abs() + tc.eps) + decay * p)

    return dict(loss=float(loss), grads=torch.cat([g_s, g_r]), weights=adamw(P.p32_s, g_s, P.numel_shard),
                weights_rep=adamw(P.p32_r, g_r, P.rep_decay_end))


def _exact_generate(case, s):
    P, cfg = s["engine"].params, s["engine"].cfg
    W = {n: P.w(n).double() for n in list(P.mat) + list(P.rep)}
    tokens, logits = [], []
    for b in range(case["B"]):
        # the chain of the most likely tokens: guess it from the head alone, then look whether the whole model agrees
        seq = s["prompt"][b]
        for _ in range(case["new"]):
            nxt = (W["lm_head"] @ W["embed"][seq[-1]]).argmax()
            seq = torch.cat([seq, nxt[None]])
        seq = torch.cat([seq, s["following"][b:b + 1]])
        last = _decoder(case, cfg, W, seq)[-case["new"] - 2:] @ W["lm_head"].t()
        if not torch.equal(last[:-2].argmax(-1), seq[-case["new"] - 1:-1]):
            return None
        tokens.append(seq[-case["new"] - 1:-1])
        logits.append(last[-1])
    return dict(tokens=torch.stack(tokens), logits=torch.stack(logits))
