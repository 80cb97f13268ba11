"""The work that a user of this framework has it do, as measurable cases: whole calls of the decode engine (a decoded token,
a prompt), one layer of a layer-stack model, and the single operators a program calls at the operator boundary — linears
from one row to a batch, the feed-forward of a token and of a prompt, attention of a prompt, of one decoded row and of the
engine's fused decode form, and the linear recurrence of the recurrent mixers.

A case is a dict of plain values whose "kind" says which path it takes.  Sizes are those of the model configurations in
tinygpt_b200.models (hidden, heads, feed-forward) and of tinygpt_b200.stack_bench, at row counts and context lengths from
a single row to a 2 048-token prompt; `draw` takes any model, odd row counts and odd lengths.
"""
from __future__ import annotations

import math

import torch

from tinygpt_b200 import engine, models, ops, stack_bench

DEV = "cuda"
BF16 = torch.bfloat16

# (hidden, query heads, kv heads, head size, feed-forward) of the four configurations
MODELS = {
    "Qwen2.5-0.5B": models.QWEN25_05B,
    "Qwen3-1.7B": models.QWEN3_17B,
    "Llama-3.2-3B": models.LLAMA32_3B,
    "Mistral-7B-v0.3": models.MISTRAL_7B,
}


def listed():
    return [
        # the headline: one greedy decode step of a small model in the middle of a 128-token answer, logits back
        dict(name="token", kind="token", model="Qwen2.5-0.5B", batch=1, at=80),
        # a long prompt of the mid-size model: time to the first token
        dict(name="prompt", kind="prompt", model="Qwen3-1.7B", rows=2048),
        # the smallest call: one row through one projection with its bias
        dict(name="linear_one", kind="linear", rows=1, n=1152, k=896, bias=True),
        # a decode batch of eight sequences through one projection
        dict(name="linear_rows", kind="linear", rows=8, n=4096, k=2048, bias=False),
        # the feed-forward of one decoded token: norm, gate | up, SiLU, down, residual
        dict(name="mlp_token", kind="mlp_token", model="Llama-3.2-3B"),
        # the feed-forward of a long prompt: norm, two products, SiLU, residual
        dict(name="mlp_prompt", kind="mlp_prompt", model="Llama-3.2-3B", rows=2048),
        # attention of one decoded token over a long in-place cache, positions and cache write fused
        dict(name="attn_token", kind="attn_token", model="Llama-3.2-3B", at=4000, ctx=4096),
        # causal attention of a long prompt
        dict(name="attn_prompt", kind="attn_prompt", model="Qwen3-1.7B", batch=1, rows=2048),
        # causal attention of a batch of ragged-length prompts, small heads, seven query heads per kv head
        dict(name="attn_prompt_batch", kind="attn_prompt", model="Qwen2.5-0.5B", batch=4, rows=333),
        # attention of one decoded row through the operator boundary: a new query against every cached row
        dict(name="attn_row", kind="attn_row", model="Qwen3-1.7B", batch=1, keys=2049),
        # a layer of a layer-stack model over a prompt: windowed attention with kept first tokens, gated feed-forward, logits
        dict(name="stack_layer", kind="stack_layer", width=2048, heads=16, kv_heads=8, ff=6144, window=1024, keep_first=4,
             vocab=2048, rows=2048),
        # the linear recurrence of the recurrent mixers over a prompt, with the delta rule's removal
        dict(name="scan", kind="scan", form="delta", heads=16, dk=128, dv=128, lengths="2048"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "prompt", "linear", "mlp_token", "mlp_prompt", "attn_token", "attn_prompt", "attn_row", "stack_layer",
                       "scan"])
    if kind == "token":
        return dict(kind=kind, model=rng.choice(["Qwen2.5-0.5B", "Qwen3-1.7B"]), batch=rng.choice([1, 1, rng.randint(2, 8)]),
                    at=_log(rng, 9, 1000))
    if kind == "prompt":
        return dict(kind=kind, model=rng.choice(["Qwen2.5-0.5B", "Qwen3-1.7B"]), rows=_log(rng, 9, 2048))
    if kind == "linear":
        s = MODELS[rng.choice(sorted(MODELS))]
        n, k = rng.choice([(s.q_dim + 2 * s.kv_dim, s.hidden), (s.hidden, s.q_dim), (2 * s.intermediate, s.hidden),
                           (s.hidden, s.intermediate)])
        return dict(kind=kind, rows=_log(rng, 1, 16), n=n, k=k, bias=rng.random() < 0.4)
    if kind == "mlp_token":
        return dict(kind=kind, model=rng.choice(sorted(MODELS)))
    if kind == "mlp_prompt":
        return dict(kind=kind, model=rng.choice(sorted(MODELS)[:3]), rows=_log(rng, 17, 2048))
    if kind == "attn_token":
        ctx = rng.choice([256, 1024, 2304, 4096])
        return dict(kind=kind, model=rng.choice(sorted(MODELS)), at=min(ctx - 1, _log(rng, 8, ctx)), ctx=ctx)
    if kind == "attn_prompt":
        batch = rng.choice([1, 1, 2, 4])
        return dict(kind=kind, model=rng.choice(sorted(MODELS)), batch=batch, rows=_log(rng, 16, 2048 // batch))
    if kind == "attn_row":
        return dict(kind=kind, model=rng.choice(sorted(MODELS)), batch=rng.choice([1, 1, 4]), keys=_log(rng, 16, 4096))
    if kind == "stack_layer":
        heads, width = rng.choice([(16, 2048), (24, 3072)])
        window = rng.choice([0, 257, 1024])
        return dict(kind=kind, width=width, heads=heads, kv_heads=8, ff=rng.choice([5464, 6144, 8192]), window=window,
                    keep_first=4 if window else 0, vocab=2048, rows=_log(rng, 16, 2048))
    n_seq = rng.choice([1, 1, 3])
    return dict(kind="scan", form=rng.choice(["delta", "gated"]), heads=rng.choice([8, 16]), dk=rng.choice([64, 128]),
                dv=rng.choice([64, 128]), lengths=",".join(str(_log(rng, 1, 2048 // n_seq)) for _ in range(n_seq)))


# ------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed + 1))


def _randn(g, *shape, std=1.0, mean=0.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std + mean).to(dtype)


def _ids(g, vocab, *shape):
    return torch.randint(0, vocab, shape, generator=g, device=DEV, dtype=torch.int64)


def _angles(hd, theta, positions):
    """cos, sin [positions, hd / 2] of the rotate-half positions, 64 bits."""
    inv = 1.0 / (theta ** (torch.arange(0, hd, 2, device=DEV, dtype=torch.float64) / hd))
    a = positions.to(torch.float64)[:, None] * inv[None, :]
    return a.cos(), a.sin()


def _rope_table(spec, ctx):
    """The fp32 table [ctx, head size, 2] (cos, sin; both halves alike) that a program builds once per model."""
    c, s = _angles(spec.head_dim, spec.rope_theta, torch.arange(ctx, device=DEV))
    half = torch.stack([c, s], -1)
    return torch.cat([half, half], 1).float().contiguous()


def _model(case, seed, ctx):
    spec = MODELS[case["model"]].with_ctx(ctx)
    return spec, models.synth_weights(spec, seed=seed, device=DEV, device_generator=True)


def _in_token(case, seed):
    spec, w = _model(case, seed, 1024)
    g = _gen(seed)
    return spec, w, _ids(g, spec.vocab, case["batch"], case["at"]), _ids(g, spec.vocab, case["batch"], 1)


def _in_prompt(case, seed):
    spec, w = _model(case, seed, 2304)
    return spec, w, _ids(_gen(seed), spec.vocab, 1, case["rows"])


def _in_linear(case, seed):
    g = _gen(seed)
    return (_randn(g, case["rows"], case["k"]), _randn(g, case["n"], case["k"], std=0.02),
            _randn(g, case["n"], std=0.1) if case["bias"] else None)


def _in_mlp(case, seed):
    s, g = MODELS[case["model"]], _gen(seed)
    return (s, _randn(g, case.get("rows", 1), s.hidden), _randn(g, s.hidden, std=0.05, mean=1.0),
            _randn(g, 2 * s.intermediate, s.hidden, std=0.02), _randn(g, s.hidden, s.intermediate, std=0.02))


def _in_attn_token(case, seed):
    s, g = MODELS[case["model"]], _gen(seed)
    qn, kn = (_randn(g, s.head_dim, std=0.05, mean=1.0), _randn(g, s.head_dim, std=0.05, mean=1.0)) if s.qk_norm else (None, None)
    return (s, _randn(g, s.q_dim + 2 * s.kv_dim, std=1.5), _randn(g, case["ctx"], s.kv_heads, s.head_dim),
            _randn(g, case["ctx"], s.kv_heads, s.head_dim), qn, kn)


def _in_attn(case, seed, rows, keys):
    s, g, B = MODELS[case["model"]], _gen(seed), case["batch"]
    return (_randn(g, B, rows, s.q_heads, s.head_dim, std=1.5), _randn(g, B, keys, s.kv_heads, s.head_dim),
            _randn(g, B, keys, s.kv_heads, s.head_dim))


def _in_stack(case, seed):
    attn = models.AttnSpec(case["heads"], case["kv_heads"], 128, 128, 128 ** -0.5, case["window"], case["keep_first"])
    spec = models.StackSpec(name="layer", architecture="Kozusun", width=case["width"], vocab=case["vocab"],
                            layers=(models.StackLayerSpec(attn, case["ff"]),), embed_scale=8.0, residual_mult=0.3, norm_eps=1e-5,
                            norm_offset=1.0, max_ctx=2048, max_slots=1)
    w = stack_bench.device_stack_weights(spec, torch.device(DEV), seed)
    return spec, w, _ids(_gen(seed), spec.vocab, 1, case["rows"])


def _lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def _in_scan(case, seed):
    """The recurrence's operands as column ranges of one matrix, as the mixers lay them out.  "delta": a decay per key
    channel and the removal along a unit key; "gated": a decay per key channel, no removal."""
    g, n, H, dk, dv = _gen(seed), sum(_lengths(case)), case["heads"], case["dk"], case["dv"]
    f32 = torch.float32
    k = _randn(g, n, H, dk, dtype=f32)
    unit = k / k.norm(dim=-1, keepdim=True)
    cols = dict(d=torch.exp(-0.2 * torch.rand(n, H * dk, generator=g, device=DEV)), b=unit.reshape(n, H * dk),
                r=_randn(g, n, H * dk, dtype=f32), v=_randn(g, n, H * dv, dtype=f32))
    if case["form"] == "delta":
        cols["p"] = torch.rand(n, H * dk, generator=g, device=DEV) * unit.reshape(n, H * dk)
        cols["q"] = unit.reshape(n, H * dk)
    return cols


def prepare(case, seed):
    kind = case["kind"]
    if kind == "token":
        spec, w, prompt, tok = _in_token(case, seed)
        eng = engine.DecodeEngine(spec, w)
        eng.forward(prompt)
        return dict(kind=kind, eng=eng, at=case["at"], ids=tok)
    if kind == "prompt":
        spec, w, ids = _in_prompt(case, seed)
        return dict(kind=kind, eng=engine.DecodeEngine(spec, w), ids=ids)
    if kind == "linear":
        x, w, b = _in_linear(case, seed)
        return dict(kind=kind, x=x, w=w, b=b)
    if kind in ("mlp_token", "mlp_prompt"):
        s, x, norm, gu, down = _in_mlp(case, seed)
        return dict(kind=kind, x=x[0].contiguous() if kind == "mlp_token" else x, norm=norm, gu=gu, down=down, eps=s.rms_eps)
    if kind == "attn_token":
        s, qkv, kc, vc, qn, kn = _in_attn_token(case, seed)
        return dict(kind=kind, qkv=qkv, k=kc, v=vc, k_row=kc[case["at"]], v_row=vc[case["at"]],
                    args=dict(q_heads=s.q_heads, kv_heads=s.kv_heads, head_dim=s.head_dim, q_norm=qn, k_norm=kn, eps=s.rms_eps,
                              pos=torch.tensor([case["at"]], dtype=torch.int32, device=DEV), rope_table=_rope_table(s, case["ctx"])))
    if kind in ("attn_prompt", "attn_row"):
        n = case.get("rows", case.get("keys"))
        q, k, v = _in_attn(case, seed, n if kind == "attn_prompt" else 1, n)
        return dict(kind=kind, q=q, k=k, v=v)
    if kind == "stack_layer":
        spec, w, ids = _in_stack(case, seed)
        return dict(kind=kind, eng=engine.DecodeEngine(spec, w), ids=ids)
    cols, lens = _in_scan(case, seed), _lengths(case)
    big, views, at = torch.cat(list(cols.values()), 1), {}, 0
    for name, t in cols.items():
        views[name] = big[:, at:at + t.shape[1]]
        at += t.shape[1]
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(kind=kind, cols=views, sizes=dict(heads=case["heads"], dk=case["dk"], dv=case["dv"]),
                state=torch.zeros(len(lens), case["heads"] * case["dk"] * case["dv"], device=DEV),
                row0=torch.tensor([sum(lens[:i]) for i in range(len(lens))], **i32), count=torch.tensor(lens, **i32),
                slot=torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], **i32),
                pos=torch.tensor([t for n in lens for t in range(n)], **i32))


def run(state):
    kind = state["kind"]
    if kind == "token":
        state["eng"].seek(state["at"])
        return state["eng"].forward(state["ids"])
    if kind == "prompt":
        state["eng"].reset_cache()
        return state["eng"].forward(state["ids"])
    if kind == "linear":
        return ops.linear(state["x"], state["w"], state["b"])
    if kind == "mlp_token":
        act = ops.gemv_fused(state["x"], state["gu"], norm_weight=state["norm"], eps=state["eps"], silu_mul=True)
        return ops.gemv_fused(act, state["down"], residual=state["x"])
    if kind == "mlp_prompt":
        act = ops.silu_mul(ops.gemm(ops.rms_norm(state["x"], state["norm"], state["eps"]), state["gu"]))
        return ops.add(state["x"], ops.gemm(act, state["down"]))
    if kind == "attn_token":
        out = ops.attn_decode(state["qkv"], state["k"], state["v"], **state["args"])
        return [out, state["k_row"], state["v_row"]]
    if kind in ("attn_prompt", "attn_row"):
        return ops.flash_attention(state["q"], state["k"], state["v"], is_causal=kind == "attn_prompt")
    if kind == "stack_layer":
        state["eng"].reset_cache()
        return state["eng"].forward(state["ids"], all_positions=True)
    c = state["cols"]
    out = ops.stack_lin_scan(c["d"], c["b"], c["r"], c["v"], state["state"], state["row0"], state["count"], state["slot"], state["pos"],
                             p=c.get("p"), q=c.get("q"), **state["sizes"])
    return [out, state["state"]]


# --------------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    kind = case["kind"]
    if kind == "token":
        s, B, ctx = MODELS[case["model"]], case["batch"], case["at"] + 1
        kv = 4 * s.layers * s.kv_dim * ctx
        return dict(bytes=2 * s.weight_params + B * (kv + 2 * s.vocab),
                    flops=B * (2 * s.weight_params + 4 * s.layers * s.q_dim * ctx))
    if kind == "prompt":
        s, n = MODELS[case["model"]], case["rows"]
        return dict(bytes=2 * s.weight_params + 4 * s.layers * s.kv_dim * n + 2 * n * s.hidden + 2 * s.vocab,
                    flops=2 * n * s.layers * s.per_layer_params + 2 * s.vocab * s.hidden + 2 * s.layers * s.q_dim * n * (n + 1))
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return dict(bytes=2 * (m * k + n * k + m * n + (n if case["bias"] else 0)), flops=2 * m * n * k)
    if kind in ("mlp_token", "mlp_prompt"):
        s, m = MODELS[case["model"]], case.get("rows", 1)
        return dict(bytes=2 * (3 * s.intermediate * s.hidden + 2 * m * s.hidden + s.hidden), flops=6 * m * s.intermediate * s.hidden)
    if kind == "attn_token":
        s, n = MODELS[case["model"]], case["at"] + 1
        return dict(bytes=4 * n * s.kv_dim + 4 * s.q_dim + 8 * s.kv_dim, flops=4 * n * s.q_dim)
    if kind == "attn_prompt":
        s, B, n = MODELS[case["model"]], case["batch"], case["rows"]
        return dict(bytes=4 * B * n * (s.q_dim + s.kv_dim), flops=2 * B * s.q_dim * n * (n + 1))
    if kind == "attn_row":
        s, B, n = MODELS[case["model"]], case["batch"], case["keys"]
        return dict(bytes=4 * B * (n * s.kv_dim + s.q_dim), flops=4 * B * s.q_dim * n)
    if kind == "stack_layer":
        W, n, V = case["width"], case["rows"], case["vocab"]
        H, G, ff = case["heads"] * 128, case["kv_heads"] * 128, case["ff"]
        params = W * (H + 2 * G + case["heads"] + 2 * ff) + W * (H + ff)
        win, keep = case["window"] or n, case["keep_first"]
        pairs = sum(min(i + 1, win + min(keep, max(0, i + 1 - win))) for i in range(n))
        return dict(bytes=2 * (params + V * W + n * W + n * V), flops=2 * n * (params + V * W) + 4 * H * pairs)
    n, H, dk, dv = sum(_lengths(case)), case["heads"], case["dk"], case["dv"]
    vecs, per = (5, 8) if case["form"] == "delta" else (3, 5)
    return dict(bytes=4 * H * (n * (vecs * dk + 2 * dv) + len(_lengths(case)) * dk * dv), flops=per * n * H * dk * dv)


def tolerance(case):
    """About four times the error that the path shows against 64 bits: bf16 results and the roundings on the way there."""
    kind = case["kind"]
    if kind in ("token", "prompt"):
        return dict(rel=0.12)    # 24 … 28 layers of bf16 roundings (0.02 … 0.04): each layer's travel through all that follow
    if kind == "attn_token":
        return dict(rel=0.025)   # queries and keys are rounded again behind norm and rotation
    if kind in ("mlp_token", "mlp_prompt", "stack_layer"):
        return dict(rel=0.016)
    if kind == "scan":
        return dict(rel=1e-5)    # fp32 throughout
    return dict(rel=0.008)


# ------------------------------------------------------------------------------------------ the same, plain, in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, c, s):
    """x [..., rows, heads, hd]; c, s [rows, hd / 2]."""
    a, b = x.chunk(2, -1)
    c, s = c[:, None, :], s[:, None, :]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, mask):
    """q [B, n, Hq, hd], k, v [B, m, Hkv, hd], mask [n, m] or None → [B, n, Hq, hd]."""
    group = q.shape[2] // k.shape[2]
    out = torch.empty_like(q)
    for b in range(q.shape[0]):
        for h in range(q.shape[2]):
            s = q[b, :, h] @ k[b, :, h // group].t() * q.shape[-1] ** -0.5
            if mask is not None:
                s = s.masked_fill(~mask, -math.inf)
            out[b, :, h] = torch.softmax(s, -1) @ v[b, :, h // group]
    return out


def _causal(n):
    return torch.ones(n, n, dtype=torch.bool, device=DEV).tril()


def _whole_model(spec, w, ids):
    """Last-row logits [B, 1, V] of the token ids [B, n]."""
    B, n = ids.shape
    x = w["model.embed_tokens.weight"][ids].double()
    c, s = _angles(spec.head_dim, spec.rope_theta, torch.arange(n, device=DEV))
    mask = _causal(n)
    for l in range(spec.layers):
        p = "model.layers.%d." % l
        g = lambda name: w[p + name].double()  # noqa: E731
        qkv = _rms(x, g("input_layernorm.weight"), spec.rms_eps) @ g("self_attn.qkv_proj.weight").t()
        if spec.qkv_bias:
            qkv = qkv + g("self_attn.qkv_proj.bias")
        q, k, v = qkv.split([spec.q_dim, spec.kv_dim, spec.kv_dim], -1)
        q, k, v = (t.reshape(B, n, -1, spec.head_dim) for t in (q, k, v))
        if spec.qk_norm:
            q, k = _rms(q, g("self_attn.q_norm.weight"), spec.rms_eps), _rms(k, g("self_attn.k_norm.weight"), spec.rms_eps)
        o = _attend(_rotate(q, c, s), _rotate(k, c, s), v, mask).reshape(B, n, -1)
        x = x + o @ g("self_attn.o_proj.weight").t()
        gate, up = (_rms(x, g("post_attention_layernorm.weight"), spec.rms_eps) @ g("mlp.gate_up_proj.weight").t()).chunk(2, -1)
        x = x + (_silu(gate) * up) @ g("mlp.down_proj.weight").t()
    head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
    return _rms(x[:, -1:], w["model.norm.weight"].double(), spec.rms_eps) @ head.double().t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "token":
        spec, w, prompt, tok = _in_token(case, seed)
        return _whole_model(spec, w, torch.cat([prompt, tok], 1))
    if kind == "prompt":
        return _whole_model(*_in_prompt(case, seed))
    if kind == "linear":
        x, w, b = _in_linear(case, seed)
        y = x.double() @ w.double().t()
        return y if b is None else y + b.double()
    if kind in ("mlp_token", "mlp_prompt"):
        s, x, norm, gu, down = (t if not torch.is_tensor(t) else t.double() for t in _in_mlp(case, seed))
        gate, up = (_rms(x, norm, s.rms_eps) @ gu.t()).chunk(2, -1)
        y = x + (_silu(gate) * up) @ down.t()
        return y[0] if kind == "mlp_token" else y
    if kind == "attn_token":
        s, qkv, kc, vc, qn, kn = (t if not torch.is_tensor(t) else t.double() for t in _in_attn_token(case, seed))
        at, hd = case["at"], s.head_dim
        q, k, v = (t.reshape(1, -1, hd) for t in qkv.split([s.q_dim, s.kv_dim, s.kv_dim]))
        if qn is not None:
            q, k = _rms(q, qn, s.rms_eps), _rms(k, kn, s.rms_eps)
        c, sn = _angles(hd, s.rope_theta, torch.tensor([at], device=DEV))
        q, k = _rotate(q, c, sn), _rotate(k, c, sn)
        keys, vals = torch.cat([kc[:at], k]), torch.cat([vc[:at], v])
        return [_attend(q[None], keys[None], vals[None], None).reshape(-1), k[0], v[0]]
    if kind in ("attn_prompt", "attn_row"):
        n = case.get("rows", case.get("keys"))
        q, k, v = (t.double() for t in _in_attn(case, seed, n if kind == "attn_prompt" else 1, n))
        return _attend(q, k, v, _causal(n) if kind == "attn_prompt" else None)
    if kind == "stack_layer":
        spec, w, ids = _in_stack(case, seed)
        w = {k: t.double() for k, t in w.items()}
        lay, n, H = spec.layout(0), case["rows"], case["heads"]
        x = w["embed"][ids[0]] * spec.embed_scale
        z = _rms(x, 1.0 + w["l0.norm"], spec.norm_eps) @ w["l0.w_in"].t() + w["l0.b_in"]
        q, k, v = (z[:, o:o + h * 128].reshape(1, n, h, 128) for o, h in ((lay.off_q, H), (lay.off_k, case["kv_heads"]), (lay.off_v, case["kv_heads"])))
        i = torch.arange(n, device=DEV)
        mask = _causal(n)
        if case["window"]:
            mask = mask & ((i[:, None] - i[None, :] < case["window"]) | (i[None, :] < case["keep_first"]))
        o = _attend(q, k, v, mask)[0] * torch.sigmoid(z[:, lay.off_g:lay.off_g + H])[:, :, None]
        gate, up = z[:, lay.off_gate:lay.off_gate + case["ff"]], z[:, lay.off_up:lay.off_up + case["ff"]]
        act = torch.nn.functional.gelu(gate, approximate="tanh") * up
        W = w["l0.w_out"]
        x = x + spec.residual_mult * (o.reshape(n, -1) @ W[:, :H * 128].t() + act @ W[:, lay.off_act:lay.off_act + case["ff"]].t())
        return (_rms(x, 1.0 + w["final_norm"], spec.norm_eps) @ w["head"].t())[None]
    cols = {k: t.double() for k, t in _in_scan(case, seed).items()}
    H, dk, dv, lens = case["heads"], case["dk"], case["dv"], _lengths(case)
    out = torch.empty(sum(lens), H, dv, dtype=torch.float64, device=DEV)
    states, at = [], 0
    for n in lens:
        S = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV)
        for t in range(at, at + n):
            d, b, r = (cols[c][t].view(H, dk) for c in "dbr")
            new = d[:, :, None] * S + b[:, :, None] * cols["v"][t].view(H, 1, dv)
            if "p" in cols:
                new -= cols["p"][t].view(H, dk, 1) * (cols["q"][t].view(H, 1, dk) @ S)
            S = new
            out[t] = (r[:, None, :] @ S)[:, 0]
        states.append(S.reshape(-1))
        at += n
    return [out.reshape(sum(lens), -1), torch.stack(states)]
