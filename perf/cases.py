"""The framework's everyday work as timed cases, with a float64 restatement of each.

Two groups, each through the entry points a program calls:

* PaliGemma-3B-pt-224 through the drop-in model class (`modeling_gemma.PaliGemmaForConditionalGeneration`): image and
  prompt, prompts in a batch, one cached step for 1 to 32 sequences; and its vision tower through
  `PaliGemmaEngine.encode_images`.  Two cases run the whole model; the others run some of its layers at the model's own
  widths (a small vocabulary keeps the head from hiding the layers).
* The mixers and experts that the ragged-batch models are made of, through the C ABI of include/pg_b200.h: windowed
  attention over a paged cache, a routed mixture of experts, gated and plain linear attention; sizes as in
  `pg_b200/arch_bench.py`.

Ranges (`draw`): 1 to 64 images; prompts of 16 to 600 tokens, up to 1400 in a batch; cached steps for 1 to 32 sequences
behind 17 to 1400 tokens; ragged prompts of 16 to 2048 tokens for 1 to 4 sequences and single tokens of 1 to 16 sequences
behind 64 to 4000; 1 to 8192 tokens through the experts; 16-bit types (bf16, and fp16 where the model class takes it).
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "multimodal-financial-analysis-tool-using-paligemma_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from modeling_gemma import KVCache, PaliGemmaConfig, PaliGemmaForConditionalGeneration  # noqa: E402
from pg_b200 import _cabi as cabi  # noqa: E402
from pg_b200 import synth  # noqa: E402
from pg_b200.engine import PaliGemmaEngine  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
FULL = synth.PALIGEMMA_3B_224
BLOCK_VOCAB = synth.SMALL["vocab_size"]
PAGE = 64
F64 = torch.float64


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a first call: one image and a short prompt, all logits, as `forward` answers the reference's drivers, in the
        # type the reference publishes its numbers for
        {"name": "image_and_prompt", "kind": "prompt", "dtype": "fp16", "batch": 1, "tokens": 260, "layers": 18,
         "vision_layers": 27, "vocab": FULL["vocab_size"], "image": True},
        # the step every generated token costs: the whole decoder, one sequence, all logits
        {"name": "cached_step", "kind": "step", "dtype": "bf16", "batch": 1, "context": 261, "layers": 18,
         "vocab": FULL["vocab_size"]},
        # one request's image through the tower and the projector
        {"name": "one_image", "kind": "vision", "dtype": "bf16", "batch": 1, "vision_layers": 9},
        # a batch of images (feature extraction over a data set)
        {"name": "many_images", "kind": "vision", "dtype": "bf16", "batch": 64, "vision_layers": 9},
        # equal-length prompts admitted together
        {"name": "prompt_batch", "kind": "prompt", "dtype": "bf16", "batch": 4, "tokens": 323, "layers": 6,
         "vision_layers": 1, "vocab": BLOCK_VOCAB, "image": False},
        # a few long generations side by side
        {"name": "step_of_8", "kind": "step", "dtype": "bf16", "batch": 8, "context": 1344, "layers": 6,
         "vocab": BLOCK_VOCAB},
        # a full batch of generations
        {"name": "step_of_32", "kind": "step", "dtype": "bf16", "batch": 32, "context": 388, "layers": 6,
         "vocab": BLOCK_VOCAB},
        # windowed attention of four prompts of the ragged models
        {"name": "ragged_prompts", "kind": "attention", "seqs": 4, "tokens": 2048, "past": 0, "heads": 16, "kv_heads": 4,
         "dim": 128, "window": 1024},
        # the same attention in a decode step of a few sequences
        {"name": "ragged_step", "kind": "attention", "seqs": 8, "tokens": 1, "past": 1500, "heads": 16, "kv_heads": 4,
         "dim": 128, "window": 1024},
        # routed experts over the tokens of four prompts
        {"name": "experts_prompts", "kind": "experts", "tokens": 8192, "width": 2048, "experts": 16, "top": 2, "ff": 2048},
        # routed experts in a decode step of a few sequences
        {"name": "experts_step", "kind": "experts", "tokens": 8, "width": 2048, "experts": 16, "top": 2, "ff": 2048},
        # linear attention with a constant decay per head over four prompts
        {"name": "linear_attention", "kind": "scan", "decay": "head", "seqs": 4, "tokens": 2048, "heads": 16, "dim": 128},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vision", "prompt", "step", "step", "attention", "attention", "experts", "scan"])
    wide = rng.random() < 0.5
    if kind == "vision":
        return {"kind": kind, "dtype": rng.choice(["bf16", "fp16"]), "batch": _spread(rng, 1, 64),
                "vision_layers": rng.choice([3, 9])}
    if kind == "prompt":
        tokens = _spread(rng, 16, 600)
        return {"kind": kind, "dtype": rng.choice(["bf16", "fp16"]), "tokens": tokens,
                "batch": rng.randint(1, max(1, min(8, 1400 // tokens))), "layers": rng.choice([2, 6]), "vision_layers": 1,
                "vocab": BLOCK_VOCAB, "image": False}
    if kind == "step":
        return {"kind": kind, "dtype": rng.choice(["bf16", "fp16"]), "batch": _spread(rng, 1, 32),
                "context": _spread(rng, 17, 1400), "layers": rng.choice([4, 6]), "vocab": BLOCK_VOCAB}
    if kind == "attention":
        one = rng.random() < 0.4
        return {"kind": kind, "seqs": _spread(rng, 1, 16) if one else rng.randint(1, 4),
                "tokens": 1 if one else _spread(rng, 16, 2048),
                "past": _spread(rng, 64, 4000) if one else rng.choice([0, 0, rng.randint(1, 1500)]),
                "heads": 16 if wide else 8, "kv_heads": 4 if wide else 2, "dim": rng.choice([64, 128, 128]),
                "window": rng.choice([0, 512, 1024])}
    if kind == "experts":
        return {"kind": kind, "tokens": _spread(rng, 1, 8192), "width": 2048 if wide else 1024,
                "experts": 16 if wide else 8, "top": 2, "ff": 2048 if wide else 1024}
    return {"kind": kind, "decay": rng.choice(["head", "channel"]), "seqs": rng.randint(1, 4),
            "tokens": _spread(rng, 1, 2048), "heads": 16 if wide else 8, "dim": rng.choice([64, 128])}


# ------------------------------------------------------------------------------------------------ PaliGemma: inputs
def _config(case):
    cfg = {k: v for k, v in FULL.items()}
    vocab = case.get("vocab", BLOCK_VOCAB)
    image = FULL["image_token_index"] if vocab == FULL["vocab_size"] else synth.SMALL["image_token_index"]
    cfg.update(vocab_size=vocab, image_token_index=image,
               vision_config=dict(FULL["vision_config"], num_hidden_layers=case.get("vision_layers", 1)),
               text_config=dict(FULL["text_config"], vocab_size=vocab, num_hidden_layers=case.get("layers", 1)))
    return cfg


_STD = {"w": 0.02, "b": 0.02, "emb": 0.02, "pos": 0.02}
_INTO_STREAM = ("o_proj.weight", "down_proj.weight", "out_proj.weight", "fc2.weight")


def _weights(case, seed):
    """Random weights at the scale models are trained from: projections and embeddings N(0, 0.02), the projections into
    the residual stream divided by sqrt(2 x the model's layers), layer norms around 1, RMS norms (stored around zero)
    around 0."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    for key, shape, kind in synth.state_dict_spec(_config(case)):
        t = torch.empty(shape, dtype=DTYPES[case["dtype"]], device="cuda")
        std = _STD.get(kind, 0.1)
        if key.endswith(_INTO_STREAM):
            part = FULL["vision_config" if "vision_model" in key else "text_config"]
            std /= math.sqrt(2.0 * part["num_hidden_layers"])
        t.normal_(1.0 if kind == "ln_w" else 0.0, std, generator=gen)
        out[key] = t
    return out, gen


def _model(case, sd, kv_tokens):
    model = PaliGemmaForConditionalGeneration(PaliGemmaConfig(**_config(case)), init_weights=False, kv_pool_tokens=kv_tokens)
    model.load_state_dict(sd, strict=False, assign=True)
    model.tie_weights()
    return model.eval()


def _prompt_inputs(case, gen):
    cfg = _config(case)
    B, q = case["batch"], case["tokens"]
    ids = torch.randint(3, 7000, (B, q), device="cuda", generator=gen)
    pixels = None
    if case["image"]:
        n = cfg["vision_config"]["num_image_tokens"]
        ids[:, :n] = cfg["image_token_index"]
        pixels = torch.randn((B, 3, 224, 224), device="cuda", generator=gen).clamp_(-1, 1).to(DTYPES[case["dtype"]])
    return ids, pixels


def _step_inputs(case, gen):
    t = FULL["text_config"]
    B, T = case["batch"], case["context"]
    ids = torch.randint(3, 7000, (B, 1), device="cuda", generator=gen)
    shape = (B, t["num_key_value_heads"], T, t["head_dim"])
    kv = []
    for _ in range(case["layers"]):
        kv.append(tuple(torch.empty(shape, dtype=DTYPES[case["dtype"]], device="cuda").normal_(0.0, 0.9, generator=gen)
                        for _ in range(2)))
    return ids, kv


def _prepare_prompt(case, seed):
    sd, gen = _weights(case, seed)
    ids, pixels = _prompt_inputs(case, gen)
    model = _model(case, sd, 2 * case["batch"] * (case["tokens"] + 2 * PAGE))
    return {"model": model, "ids": ids, "pixels": pixels, "mask": torch.ones_like(ids)}


def _run_prompt(s):
    with torch.no_grad():
        return s["model"](input_ids=s["ids"], pixel_values=s["pixels"], attention_mask=s["mask"],
                          kv_cache=KVCache())["logits"]


def _prepare_step(case, seed):
    sd, gen = _weights(case, seed)
    ids, kv = _step_inputs(case, gen)
    B, T = case["batch"], case["context"]
    model = _model(case, sd, B * (T + 24 * PAGE))
    cache = KVCache()
    for li, (k, v) in enumerate(kv):
        cache.update(k, v, li)
    s = {"model": model, "cache": cache, "ids": ids, "context": T,
         "mask": torch.ones((B, T + 1), dtype=torch.int64, device="cuda")}
    _run_step(s)      # a program that decodes has stepped before: the cache lies in pages, the step is captured
    return s


def _run_step(s):
    paged = s["cache"]._paged
    if paged is not None:      # every pass decodes the token after the same context
        paged.length = s["context"]
        paged.kv_len.fill_(s["context"])
    with torch.no_grad():
        return s["model"](input_ids=s["ids"], attention_mask=s["mask"], kv_cache=s["cache"])["logits"]


def _prepare_vision(case, seed):
    sd, gen = _weights(case, seed)
    pixels = torch.randn((case["batch"], 3, 224, 224), device="cuda", generator=gen).clamp_(-1, 1)
    return {"engine": PaliGemmaEngine(_config(case), sd, kv_pool_tokens=8 * PAGE),
            "pixels": pixels.to(DTYPES[case["dtype"]])}


def _run_vision(s):
    return s["engine"].encode_images(s["pixels"])


# ------------------------------------------------------------------------------------------------ PaliGemma: float64
def _layer_norm(x, w, b):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w.to(F64), b.to(F64), 1e-6)


def _rms_norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * (1.0 + w.to(F64))


def _attend(q, k, v):
    """q [B, h, q, d], k and v [B, 1 or h, n, d]: softmax(q k^T / sqrt(d)) v, nothing masked."""
    s = torch.softmax((q @ k.transpose(-1, -2)) / math.sqrt(q.shape[-1]), -1)
    return s @ v


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _exact_vision(sd, case, pixels):
    v = FULL["vision_config"]
    heads, p = v["num_attention_heads"], v["patch_size"]
    vm = "vision_tower.vision_model."
    W = lambda k: sd[k].to(F64)  # noqa: E731
    out = []
    for px in pixels.split(8):
        x = torch.nn.functional.unfold(px.to(F64), p, stride=p).transpose(1, 2)
        x = x @ W(vm + "embeddings.patch_embedding.weight").flatten(1).T + W(vm + "embeddings.patch_embedding.bias")
        x = x + W(vm + "embeddings.position_embedding.weight")
        B, P, D = x.shape
        for i in range(case["vision_layers"]):
            L = f"{vm}encoder.layers.{i}."
            n = _layer_norm(x, sd[L + "layer_norm1.weight"], sd[L + "layer_norm1.bias"])
            q, k, u = ((n @ W(L + f"self_attn.{m}.weight").T + W(L + f"self_attn.{m}.bias"))
                       .view(B, P, heads, D // heads).transpose(1, 2) for m in ("q_proj", "k_proj", "v_proj"))
            a = _attend(q, k, u).transpose(1, 2).reshape(B, P, D)
            x = x + a @ W(L + "self_attn.out_proj.weight").T + W(L + "self_attn.out_proj.bias")
            n = _layer_norm(x, sd[L + "layer_norm2.weight"], sd[L + "layer_norm2.bias"])
            h = _gelu(n @ W(L + "mlp.fc1.weight").T + W(L + "mlp.fc1.bias"))
            x = x + h @ W(L + "mlp.fc2.weight").T + W(L + "mlp.fc2.bias")
        x = _layer_norm(x, sd[vm + "post_layernorm.weight"], sd[vm + "post_layernorm.bias"])
        out.append(x @ W("multi_modal_projector.linear.weight").T + W("multi_modal_projector.linear.bias"))
    return torch.cat(out)


def _rotate(x, pos, dtype):
    """Rotary positions of the decoder: pairs (i, i + d / 2); the frequencies are a buffer of the model's type."""
    d = x.shape[-1]
    f = (1.0 / (10000.0 ** (torch.arange(0, d, 2).float() / d))).to(dtype).to(F64).to(x.device)
    a = pos.to(F64)[:, None] * f
    c, s = torch.cos(a), torch.sin(a)
    x1, x2 = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)


def _exact_text(sd, case, ids, feats, pos, past):
    """Logits of the decoder over new tokens at positions `pos`, behind the cached keys and values `past`."""
    t, dtype = FULL["text_config"], DTYPES[case["dtype"]]
    D, heads, hd = t["hidden_size"], t["num_attention_heads"], t["head_dim"]
    lm = "language_model.model."
    W = lambda k: sd[k].to(F64)  # noqa: E731
    x = sd[lm + "embed_tokens.weight"][ids].to(F64)
    if feats is not None:
        n = feats.shape[1]
        x[:, :n] = feats / math.sqrt(D)
    x = x * float(torch.tensor(math.sqrt(D), dtype=dtype))
    B, q, _ = x.shape
    for i in range(case["layers"]):
        L = f"{lm}layers.{i}."
        n = _rms_norm(x, sd[L + "input_layernorm.weight"])
        Q = _rotate((n @ W(L + "self_attn.q_proj.weight").T).view(B, q, heads, hd).transpose(1, 2), pos, dtype)
        K = _rotate((n @ W(L + "self_attn.k_proj.weight").T).view(B, q, 1, hd).transpose(1, 2), pos, dtype)
        V = (n @ W(L + "self_attn.v_proj.weight").T).view(B, q, 1, hd).transpose(1, 2)
        if past is not None:
            K, V = torch.cat([past[i][0].to(F64), K], 2), torch.cat([past[i][1].to(F64), V], 2)
        a = _attend(Q, K, V).transpose(1, 2).reshape(B, q, heads * hd)
        x = x + a @ W(L + "self_attn.o_proj.weight").T
        n = _rms_norm(x, sd[L + "post_attention_layernorm.weight"])
        g = _gelu(n @ W(L + "mlp.gate_proj.weight").T) * (n @ W(L + "mlp.up_proj.weight").T)
        x = x + g @ W(L + "mlp.down_proj.weight").T
    n = _rms_norm(x, sd[lm + "norm.weight"])
    e = sd[lm + "embed_tokens.weight"]
    return torch.cat([n @ c.to(F64).T for c in e.split(32768)], -1)


def _exact_paligemma(case, seed):
    sd, gen = _weights(case, seed)
    if case["kind"] == "vision":
        pixels = torch.randn((case["batch"], 3, 224, 224), device="cuda", generator=gen).clamp_(-1, 1)
        return _exact_vision(sd, case, pixels.to(DTYPES[case["dtype"]]))
    if case["kind"] == "prompt":
        ids, pixels = _prompt_inputs(case, gen)
        feats = None if pixels is None else _exact_vision(sd, case, pixels)
        return _exact_text(sd, case, ids, feats, torch.arange(case["tokens"], device="cuda"), None)
    ids, kv = _step_inputs(case, gen)
    # the position of a cached token is the length of its attention mask
    return _exact_text(sd, case, ids, None, torch.full((1,), case["context"] + 1, device="cuda"), kv)


# ------------------------------------------------------------------------------------------------ ragged attention
def _slopes(heads):
    return torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)], dtype=torch.float32, device="cuda")


def _prepare_attention(case, seed):
    """Queries (normed: unit variance), gates and a paged cache whose pages lie scattered over the pool."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    S, T, H, G, d = case["seqs"], case["tokens"], case["heads"], case["kv_heads"], case["dim"]
    n, total = S * T, case["past"] + T
    cols = -(-total // PAGE)
    pages = S * cols + 3
    new = lambda *s: torch.empty(s, dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=gen)  # noqa: E731
    i32 = dict(dtype=torch.int32, device="cuda")
    s = dict(case, n=n, q=new(n, H * d), gate=new(n, H * d), k=new(pages, PAGE, G * d), v=new(pages, PAGE, G * d),
             pages=pages, table=torch.randperm(pages, device="cuda", generator=gen)[:S * cols].to(torch.int32).view(S, cols),
             slot=torch.arange(S, **i32).repeat_interleave(T), pos=(torch.arange(T, **i32) + case["past"]).repeat(S),
             slopes=_slopes(H), out=torch.empty((n, H * d), dtype=torch.bfloat16, device="cuda"),
             ws=torch.empty(5 << 19, dtype=torch.float32, device="cuda"))
    tiles = [(b * T + t, min(128, T - t), b, case["past"] + t) for b in range(S) for t in range(0, T, 128)]
    s["tiles"] = torch.tensor(tiles, **i32)
    return s


def _run_attention(s):
    L, p, H, G, d = cabi.lib(), cabi.ptr, s["heads"], s["kv_heads"], s["dim"]
    scale, cols = 1.0 / math.sqrt(d), s["table"].shape[1]
    if s["n"] >= 48:      # the engines' line between prompt portions and decode steps
        cabi.check(L.pg_attention_ragged_tc(p(s["out"]), H * d, p(s["q"]), H * d, p(s["gate"]), H * d, p(s["k"]), p(s["v"]),
                                            s["pages"] * PAGE, p(s["table"]), cols, PAGE, p(s["tiles"]), s["tiles"].shape[0],
                                            s["n"], H, G, d, d, scale, s["window"], p(s["slopes"]), None, cabi.PG_BF16,
                                            cabi.stream()), "attention_ragged_tc")
    else:
        cabi.check(L.pg_attention_ragged(p(s["out"]), H * d, p(s["q"]), H * d, p(s["gate"]), H * d, p(s["k"]), p(s["v"]),
                                         p(s["table"]), cols, PAGE, p(s["slot"]), p(s["pos"]), s["n"], H, G, d, d, scale,
                                         s["window"], p(s["slopes"]), p(s["ws"]), s["ws"].numel(), cabi.PG_BF16,
                                         cabi.stream()), "attention_ragged")
    return s["out"]


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    S, T, H, G, d = case["seqs"], case["tokens"], case["heads"], case["kv_heads"], case["dim"]
    total, out = case["past"] + T, []
    i = torch.arange(T, device="cuda")[:, None] + case["past"]
    j = torch.arange(total, device="cuda")[None, :]
    seen = (j <= i) if case["window"] <= 0 else (j <= i) & (i - j < case["window"])
    for b in range(S):
        rows = s["table"][b].long()
        k, v = (s[m][rows].reshape(-1, G, d)[:total].to(F64) for m in ("k", "v"))
        q = s["q"][b * T:(b + 1) * T].to(F64).view(T, H, d)
        head = []
        for h in range(H):
            g = h // (H // G)
            sc = q[:, h] @ k[:, g].T / math.sqrt(d) - s["slopes"][h].to(F64) * (i - j)
            head.append(torch.softmax(sc.masked_fill(~seen, -math.inf), -1) @ v[:, g])
        out.append(torch.stack(head, 1).reshape(T, H * d))
    return torch.cat(out) * torch.sigmoid(s["gate"].to(F64))


# ------------------------------------------------------------------------------------------------ routed experts
def _prepare_experts(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    T, D, E, F, top = (case[k] for k in ("tokens", "width", "experts", "ff", "top"))
    P = T * top
    new = lambda std, *s: torch.empty(s, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)  # noqa: E731
    i32 = dict(dtype=torch.int32, device="cuda")
    return dict(case, P=P, h=new(1.0, T, D), router=new(D ** -0.5, E, D), correction=new(0.01, E),
                gu=new(D ** -0.5, E, 2 * F, D), dn=new(F ** -0.5, E, D, F),
                idx=torch.empty(P, **i32), wts=torch.empty(P, dtype=torch.float32, device="cuda"),
                offsets=torch.empty(E + 1, **i32), rows=torch.empty(P, **i32), pair=torch.empty(P, **i32),
                a=new(1.0, P, D), act=new(1.0, P, F), y=new(1.0, P, D), out=new(1.0, T, D))


def _run_experts(s):
    L, p, st = cabi.lib(), cabi.ptr, cabi.stream()
    T, D, E, F, top, P, dt = s["tokens"], s["width"], s["experts"], s["ff"], s["top"], s["P"], cabi.PG_BF16
    cabi.check(L.pg_moe_route(p(s["idx"]), p(s["wts"]), None, p(s["h"]), D, p(s["router"]), p(s["correction"]), None, T, D, E,
                              top, 1.0, dt, st), "moe_route")
    cabi.check(L.pg_moe_sort(p(s["offsets"]), p(s["rows"]), p(s["pair"]), p(s["idx"]), P, top, E, st), "moe_sort")
    cabi.check(L.pg_gather_rows(p(s["a"]), p(s["h"]), D, p(s["rows"]), p(s["offsets"][E:]), P, D, dt, st), "gather_rows")
    cabi.check(L.pg_moe_gemm_act(p(s["act"]), F, p(s["a"]), D, None, p(s["gu"]), p(s["offsets"]), P, E, F, D, cabi.GLU_SILU, 0.0,
                                 2, None, dt, st), "experts up")
    cabi.check(L.pg_moe_gemm_act(p(s["y"]), D, p(s["act"]), F, None, p(s["dn"]), p(s["offsets"]), P, E, D, F, cabi.GLU_NONE, 0.0,
                                 2, None, dt, st), "experts down")
    cabi.check(L.pg_moe_combine_out(p(s["out"]), D, p(s["y"]), D, p(s["pair"]), p(s["wts"]), None, 0, T, D, top, dt, st),
               "moe_combine_out")
    return {"out": s["out"], "weights": s["wts"]}


def _exact_experts(case, seed):
    s = _prepare_experts(case, seed)
    E, F, top = case["experts"], case["ff"], case["top"]
    h = s["h"].to(F64)
    p = torch.softmax(h @ s["router"].to(F64).T, -1)
    _, idx = torch.sort(p + s["correction"].to(F64), dim=-1, descending=True, stable=True)
    idx = idx[:, :top]
    w = torch.gather(p, 1, idx)
    out = torch.zeros_like(h)
    for e in range(E):
        at, k = torch.nonzero(idx == e, as_tuple=True)
        if at.numel():
            g = h[at] @ s["gu"][e, :F].to(F64).T
            a = g * torch.sigmoid(g) * (h[at] @ s["gu"][e, F:].to(F64).T)
            out.index_add_(0, at, w[at, k][:, None] * (a @ s["dn"][e].to(F64).T))
    return {"out": out, "weights": w.reshape(-1)}


# ------------------------------------------------------------------------------------------------ linear attention
RANK, TAU = 16, 16.0


def _prepare_scan(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    S, T, H, d = case["seqs"], case["tokens"], case["heads"], case["dim"]
    n, L = S * T, cabi.lib()
    ld = 3 * H * d + (RANK if case["decay"] == "channel" else 0)
    new = lambda *s: torch.empty(s, dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=gen)  # noqa: E731
    f32 = dict(dtype=torch.float32, device="cuda")
    floats = L.pg_gla_record_floats(n, H, d, d) if case["decay"] == "channel" else L.pg_lightning_record_floats(n, H, d, d)
    return dict(case, n=n, ld=ld, proj=new(n, ld), w2=new(H * d, RANK), b2=new(H * d),
                decay_per_head=torch.exp(-_slopes(H)), rec=torch.empty(int(floats), **f32),
                state=torch.zeros((S, H, d, d), **f32), out=torch.empty((n, H * d), **f32),
                segs=torch.tensor([(b, b * T, T) for b in range(S)], dtype=torch.int32, device="cuda"))


def _run_scan(s):
    L, p, st = cabi.lib(), cabi.ptr, cabi.stream()
    n, H, d, S = s["n"], s["heads"], s["dim"], s["seqs"]
    s["state"].zero_()      # new sequences
    if s["decay"] == "head":
        cabi.check(L.pg_lightning_prep(p(s["rec"]), p(s["proj"]), s["ld"], 0, H * d, 2 * H * d, n, H, d, d, cabi.PG_BF16, st),
                   "lightning_prep")
        cabi.check(L.pg_lightning_attention(p(s["out"]), p(s["state"]), p(s["rec"]), p(s["decay_per_head"]), p(s["segs"]), S, H,
                                            d, d, st), "lightning_attention")
    else:
        cabi.check(L.pg_gla_prep(p(s["rec"]), p(s["proj"]), s["ld"], 0, H * d, 2 * H * d, 3 * H * d, RANK, p(s["w2"]), p(s["b2"]),
                                 d ** -0.5, 1.0 / TAU, n, H, d, d, cabi.PG_BF16, st), "gla_prep")
        cabi.check(L.pg_gla_attention(p(s["out"]), p(s["state"]), p(s["rec"]), p(s["segs"]), S, H, d, d, st), "gla_attention")
    return {"out": s["out"], "state": s["state"]}


def _exact_scan(case, seed):
    s = _prepare_scan(case, seed)
    S, T, H, d = case["seqs"], case["tokens"], case["heads"], case["dim"]
    x = s["proj"].to(F64)
    q, k, v = (x[:, i * H * d:(i + 1) * H * d].view(S, T, H, d) for i in range(3))
    if case["decay"] == "head":
        q, k, v = (z * torch.sigmoid(z) for z in (q, k, v))
        a = s["decay_per_head"].to(F64).view(1, 1, H, 1).expand(S, T, H, d)
    else:
        z = x[:, 3 * H * d:] @ s["w2"].to(F64).T + s["b2"].to(F64)
        a, q = torch.pow(torch.sigmoid(z), 1.0 / TAU).view(S, T, H, d), q * d ** -0.5
    state, out = torch.zeros((S, H, d, d), dtype=F64, device="cuda"), torch.empty((S, T, H, d), dtype=F64, device="cuda")
    for t in range(T):
        state = state * a[:, t, :, :, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = (state * q[:, t, :, :, None]).sum(2)
    return {"out": out.view(S * T, H * d), "state": state}


# ------------------------------------------------------------------------------------------------ the interface
_PREPARE = {"prompt": _prepare_prompt, "step": _prepare_step, "vision": _prepare_vision, "attention": _prepare_attention,
            "experts": _prepare_experts, "scan": _prepare_scan}
_RUN = {"prompt": _run_prompt, "step": _run_step, "vision": _run_vision, "attention": _run_attention, "experts": _run_experts,
        "scan": _run_scan}
_EXACT = {"prompt": _exact_paligemma, "step": _exact_paligemma, "vision": _exact_paligemma, "attention": _exact_attention,
          "experts": _exact_experts, "scan": _exact_scan}


def prepare(case, seed):
    return {"kind": case["kind"], "state": _PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["kind"]](state["state"])


def exact(case, seed):
    with torch.no_grad():
        return _EXACT[case["kind"]](case, seed)


def _vision_work(case, B):
    v = FULL["vision_config"]
    D, I, P, L = v["hidden_size"], v["intermediate_size"], v["num_image_tokens"], case["vision_layers"]
    kc = 3 * v["patch_size"] ** 2
    weights = kc * D + L * (4 * D * D + 2 * D * I) + D * FULL["projection_dim"]
    return {"bytes": 2.0 * (weights + P * D + B * (3 * v["image_size"] ** 2 + P * FULL["projection_dim"])),
            "flops": 2.0 * B * P * weights + 4.0 * B * L * P * P * D}


def _text_work(case, B, q, past):
    t = FULL["text_config"]
    D, F, hd, heads, V, L = t["hidden_size"], t["intermediate_size"], t["head_dim"], t["num_attention_heads"], case["vocab"], \
        case["layers"]
    layer = (heads + 2) * hd * D + heads * hd * D + 3 * D * F
    head = V * D
    return {"bytes": 2.0 * (L * layer + head + 2 * L * B * hd * (past + q)) + 4.0 * B * q * V,
            "flops": 2.0 * B * q * (L * layer + head) + 4.0 * L * B * q * (past + q) * heads * hd}


def work(case):
    kind = case["kind"]
    if kind == "vision":
        return _vision_work(case, case["batch"])
    if kind == "prompt":
        w = _text_work(case, case["batch"], case["tokens"], 0)
        if case["image"]:
            v = _vision_work(case, case["batch"])
            w = {k: w[k] + v[k] for k in w}
        return w
    if kind == "step":
        return _text_work(case, case["batch"], 1, case["context"])
    if kind == "attention":
        S, T, H, G, d, past = (case[k] for k in ("seqs", "tokens", "heads", "kv_heads", "dim", "past"))
        W = case["window"] if case["window"] > 0 else past + T
        pairs = sum(min(past + t + 1, W) for t in range(T))
        keys = min(past + T, W + T - 1)
        return {"bytes": 2.0 * (3 * S * T * H * d + 2 * S * keys * G * d), "flops": 4.0 * S * pairs * H * d}
    if kind == "experts":
        T, D, E, F, top = (case[k] for k in ("tokens", "width", "experts", "ff", "top"))
        met = E * (1.0 - (1.0 - top / E) ** T)      # experts that some token chooses
        return {"bytes": 2.0 * (met * 3 * F * D + E * D + 2 * T * D), "flops": 2.0 * T * (top * 3 * F * D + E * D)}
    S, T, H, d = case["seqs"], case["tokens"], case["heads"], case["dim"]
    return {"bytes": S * T * H * d * (3 * 2.0 + 4.0) + 2 * 4.0 * S * H * d * d, "flops": 4.0 * S * T * H * d * d}


def tolerance(case):
    """About four times the distance from the float64 restatement that the path shows on this hardware: 7e-3 to 1.5e-2 for
    the bf16 model (18 layers of 16-bit roundings), 1e-3 to 3e-3 in fp16, 1.9e-3 for an attention, 4.3e-3 for the experts,
    3.5e-7 for a scan's fp32 state and 1e-7 for its outputs (summed in another order: a few times that)."""
    kind = case["kind"]
    if kind == "scan":
        return {"rel": 4e-6}
    if kind == "attention":
        return {"rel": 8e-3}
    if kind == "experts":
        return {"rel": 1.7e-2}
    return {"rel": 3e-2 if case["dtype"] == "bf16" else 1.2e-2}
