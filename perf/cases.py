"""The work that programs have this framework do, as cases that can be timed and checked.

Four kinds, all through the public entry points:
  op        one quantized linear or one gate/up + down pair on ready activations (what a host framework calls layer by layer)
  prefill   a runner's forward over a batch of prompts into a new cache: first-token latency, prompt throughput
  step      one decode step of a Llama runner on a long cached context, driven by the caller (own sampling, verification of
            drafted tokens): forward of one token per sequence, then the cache is rolled back
  generate  greedy generation from short prompts (a recorded step is replayed), then one forward over the whole text for the
            logits of the continuation's tokens, as best-of-n reranking and evaluation score it

Weights are random matrices of the named decoder shapes. The head is the embedding moved by one id, so that the greedy choice
has a margin as a trained model's has: the continuation of id t is t + 1 unless the layers' outputs drown the embedding.
"exact" restates every path in 64 bits."""
import math
import os

import torch

from tpp_pytorch_extension_b200._C import _fused_llm_infer as F
from tpp_pytorch_extension_b200._C import _qtype
from tpp_pytorch_extension_b200.llm import fused_dofivik_infer as FD
from tpp_pytorch_extension_b200.llm import fused_llama_infer as FL
from tpp_pytorch_extension_b200.llm import fused_vedizen_infer as FV
from tpp_pytorch_extension_b200.llm.llm_common import TppCache, quantize_weight

VOCAB = 32000
INT8_BLOCK = 64
MAX_POS = 8192
# decoder shapes: the benchmark's two sizes, and the Llama shapes of its model legs cut to the same depth
MODELS = {
    "llama3": dict(layers=8, width=4096, heads=32, kv_heads=8, ff=14336, theta=5e5),
    "llama2": dict(layers=8, width=4096, heads=32, kv_heads=32, ff=11008, theta=1e4),
    "wide": dict(layers=8, width=4096, heads=32, kv_heads=32, ff=14336, theta=1e4),
    "deep": dict(layers=16, width=2048, heads=16, kv_heads=16, ff=8192, theta=1e4),
}
# (out, in) features of the linears of these shapes
LINEARS = ((4096, 4096), (6144, 4096), (11008, 4096), (14336, 4096), (4096, 11008), (4096, 14336), (2048, 8192), (8192, 2048))
EMBED_STD = {"llama": 2.0, "dofivik": 1.0, "vedizen": 0.25}
WEIGHT_STD = {"llama": 0.02, "dofivik": 0.01, "vedizen": 0.01}


def _op(name, weights, form, m, n, k):
    return dict(name=name, kind="op", weights=weights, form=form, m=m, n=n, k=k)


def _model(name, kind, family, model, weights, batch, tokens, new=0, ragged=False):
    return dict(name=name, kind=kind, family=family, model=model, weights=weights, batch=batch, tokens=tokens, new=new, ragged=ragged)


def listed():
    return [
        # one int8 linear with bias and SiLU for a batch of 32 decoding sequences
        _op("int8 linear 32", "qint8", "linear", 32, 11008, 4096),
        # the feed-forward of a decode step in MXFP4: gate/up with SiLU, then down
        _op("mxfp4 mlp 8", "mxfp4", "mlp", 8, 14336, 4096),
        # a serving engine's decode step: 16 sequences with 2048 cached tokens each
        _model("llama3 mxfp4 step 16x2048", "step", "llama", "llama3", "mxfp4", 16, 2048),
        # a batch of prompts of unequal lengths, padded on the left
        _model("llama3 mxfp4 prefill 4x1999 ragged", "prefill", "llama", "llama3", "mxfp4", 4, 1999, ragged=True),
        # interactive chat: one short prompt
        _model("llama3 mxfp4 generate 1x37", "generate", "llama", "llama3", "mxfp4", 1, 37, 40),
        # one sequence with a long prompt on an int8 model
        _model("llama2 int8 generate 1x1024", "generate", "llama", "llama2", "qint8", 1, 1024, 48),
        # prompt throughput of an unquantized model
        _model("llama bf16 prefill 16x2048", "prefill", "llama", "wide", "bf16", 16, 2048),
        # one long prompt on the latent-attention / delta-rule hybrid
        _model("dofivik bf16 prefill 1x4096", "prefill", "dofivik", "wide", "bf16", 1, 4096),
        # batched generation on it
        _model("dofivik bf16 generate 16x256", "generate", "dofivik", "wide", "bf16", 16, 256, 40),
        # batched prompts on the gated-linear / differential-attention decoder, narrow and deep
        _model("vedizen bf16 prefill 16x1024", "prefill", "vedizen", "deep", "bf16", 16, 1024),
        # a handful of chat sequences of unequal lengths on it
        _model("vedizen bf16 generate 5x131 ragged", "generate", "vedizen", "wide", "bf16", 5, 131, 40, ragged=True),
        # the same decoder family in true 32-bit, as used to check a converted model
        _model("vedizen f32 prefill 2x513", "prefill", "vedizen", "deep", "f32", 2, 513),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("op", "op", "prefill", "prefill", "prefill", "generate", "generate", "generate", "step"))
    if kind == "op":
        m, (n, k) = _log(rng, 1, 4096), rng.choice(LINEARS)
        weights = rng.choice(("mxfp4", "mxfp4", "qint8", "bf16"))
        form = rng.choice(("linear", "mlp")) if weights == "mxfp4" else "linear"
        c = _op("", weights, form, m, n, k)
    elif kind == "step":
        batch = _log(rng, 1, 32)
        model = rng.choice(("llama3", "llama2"))
        tokens = _log(rng, 100, min(6000, (65536 if model == "llama3" else 32768) // batch))
        c = _model("", kind, "llama", model, "mxfp4", batch, tokens)
    else:
        family, model, weights = rng.choice((("llama", "llama3", "mxfp4"), ("llama", "llama3", "mxfp4"), ("llama", "llama2", "qint8"),
                                             ("llama", "wide", "bf16"), ("dofivik", "wide", "bf16"), ("dofivik", "deep", "bf16"),
                                             ("dofivik", "deep", "f32"), ("vedizen", "wide", "bf16"), ("vedizen", "deep", "bf16"),
                                             ("vedizen", "deep", "f32")))
        if kind == "prefill":
            batch = _log(rng, 1, 16)
            most = 1500 if weights == "f32" else 8192
            c = _model("", kind, family, model, weights, batch, _log(rng, 17, min(4096, most // batch)), ragged=batch > 1 and rng.random() < 0.4)
        else:
            batch = _log(rng, 1, 8 if weights == "f32" else 48)
            most = 800 if weights == "f32" else 4096
            c = _model("", kind, family, model, weights, batch, _log(rng, 8, min(1024, most // batch)), rng.randint(12, 40), batch > 1 and rng.random() < 0.4)
    del c["name"]
    return c


# ---------------------------------------------------------------- what a program has in hand
def _shape(case):
    m = MODELS[case["model"]]
    if case["family"] == "llama":
        return FL.LlamaShape(m["layers"], m["width"], m["heads"], m["kv_heads"], m["ff"], VOCAB, rope_theta=m["theta"], max_position_embeddings=MAX_POS)
    if case["family"] == "dofivik":
        return FD.hybrid_shape(m["layers"], m["width"], m["heads"], m["ff"], VOCAB)
    return FV.vedizen_stack(m["layers"], m["width"], m["heads"], m["ff"], VOCAB)


def _dtype(case):
    return torch.float32 if case["weights"] == "f32" else torch.bfloat16


def _embedding(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    e = torch.randn(VOCAB, MODELS[case["model"]]["width"], generator=g, device="cuda")
    return (e * EMBED_STD[case["family"]]).to(torch.bfloat16), (e.roll(1, 0) * 0.02).to(torch.bfloat16)


def _prompt(case, seed):
    """Token ids and keep-mask (None without padding), [batch, tokens]; ragged prompts are padded on the left."""
    g = torch.Generator().manual_seed(seed + 2)
    B, S = case["batch"], case["tokens"]
    ids = torch.randint(0, VOCAB, (B, S), generator=g)
    if not case["ragged"]:
        return ids.cuda(), None
    length = torch.randint((S + 1) // 2, S + 1, (B, 1), generator=g)
    length[0] = S
    return ids.cuda(), (torch.arange(S).unsqueeze(0) >= S - length).to(torch.int64).cuda()


def _cached(case, seed):
    """Keys and values of the cached context, [layers] of [batch, kv_heads, tokens, 128]."""
    m, g = MODELS[case["model"]], torch.Generator(device="cuda").manual_seed(seed + 3)
    s = (case["batch"], m["kv_heads"], case["tokens"], m["width"] // m["heads"])
    return [tuple(torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16) for _ in "kv") for _ in range(m["layers"])]


def _op_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(torch.bfloat16)
    x = rnd(case["m"], case["k"])
    if case["form"] == "mlp":
        return x, [rnd(case["n"], case["k"], std=0.02), rnd(case["n"], case["k"], std=0.02), rnd(case["k"], case["n"], std=0.02)], None
    return x, [rnd(case["n"], case["k"], std=0.02)], rnd(case["n"], std=0.01)


def prepare(case, seed):
    os.environ["QINT8_BLOCK_SIZE"] = str(INT8_BLOCK)
    if case["kind"] == "op":
        x, ws, bias = _op_inputs(case, seed)
        ws = [quantize_weight(w, case["weights"]) for w in ws]
        if case["form"] == "mlp":
            ws[0].prepare(pair_with=ws[1])
            ws[2].prepare()
        elif case["weights"] != "bf16":
            ws[0].prepare()
        return dict(case, x=x, ws=ws, bias=bias)
    shape, std = _shape(case), WEIGHT_STD[case["family"]]
    if case["family"] == "llama":
        runner = FL.build_random_llama(shape, case["weights"], "cuda", seed, std, MAX_POS)
    elif case["family"] == "dofivik":
        runner = FD.build_random_dofivik(shape, _dtype(case), "cuda", seed, std)
    else:
        runner = FV.build_random_vedizen(shape, _dtype(case), "cuda", seed, std)
    runner.embed, runner.lm_head_w = (t.to(_dtype(case)) for t in _embedding(case, seed))
    state = dict(case, runner=runner)
    if case["kind"] == "step":
        state["cache"] = TppCache()
        for i, (k, v) in enumerate(_cached(case, seed)):
            state["cache"].update(k, v, i)
        B, ctx = case["batch"], case["tokens"]
        g = torch.Generator().manual_seed(seed + 2)
        state["ids"] = torch.randint(0, VOCAB, (B, 1), generator=g).cuda()
        state["mask"] = torch.ones(B, ctx + 1, device="cuda", dtype=torch.bfloat16)
        state["pos"] = torch.full((B, 1), ctx, device="cuda")
    else:
        state["ids"], state["mask"] = _prompt(case, seed)
        row = torch.arange(case["tokens"] - 1, case["tokens"] + case["new"] - 1, device="cuda")  # they predict the continuation
        state["rows"] = (torch.arange(case["batch"], device="cuda").unsqueeze(1) * (case["tokens"] + case["new"]) + row).flatten()
    return state


def _positions(mask):
    return None if mask is None else (mask.cumsum(-1) - 1).clamp(min=0)


def run(state):
    if state["kind"] == "op":
        if state["form"] == "mlp":
            h = F.fc_gate_up(state["x"], state["ws"][0], state["ws"][1])
            return {"hidden": h, "out": F.fc_plain(h, state["ws"][2])}
        return {"out": F.fc_plain_act(state["x"], state["ws"][0], state["bias"], "silu")}
    runner, ids, mask = state["runner"], state["ids"], state["mask"]
    if state["kind"] == "step":
        cache = state["cache"]
        logits, _ = runner.forward(ids, mask, state["pos"], cache)
        cache.crop(state["tokens"])
        return {"logits": logits, "cache": [cache.get_cpp().get(i) for i in range(len(cache))]}
    if state["kind"] == "prefill":
        logits, cache = runner.forward(ids, mask, _positions(mask))
        if state["family"] == "llama":
            return {"logits": logits, "cache": [cache.get_cpp().get(i) for i in range(len(cache))]}
        return {"logits": logits, "states": [lc.states for lc in cache.get_cpp().layers]}
    text = runner.generate(ids, state["new"], mask)
    if mask is not None:
        mask = torch.cat([mask, mask.new_ones(mask.shape[0], state["new"])], 1)
    runner.logit_rows = state["rows"]
    logits, _ = runner.forward(text, mask, _positions(mask))
    runner.logit_rows = None
    return {"text": text, "logits": logits}


# ---------------------------------------------------------------- what a pass cannot do without
WEIGHT_BYTES = {"mxfp4": 17 / 32, "qint8": 1 + 4 / INT8_BLOCK, "bf16": 2, "f32": 4}


def _layer_costs(case):
    """Per layer: (weights, FLOPs per token beside them and per pair of tokens that meet, bytes per token cached, bytes of
    recurrent state per sequence, tokens that an attention layer looks back at most)."""
    m = MODELS[case["model"]]
    D, H, ff, size = m["width"], m["heads"], m["ff"], 4 if case["weights"] == "f32" else 2
    if case["family"] == "llama":
        hd = D // H
        return [((2 * D + 2 * hd * m["kv_heads"]) * D + 3 * D * ff, 0, 4 * D, 2 * hd * m["kv_heads"] * 2, 0, 1 << 30)] * m["layers"]
    out = []
    for i in range(m["layers"]):
        attention = i % 4 == 3
        if case["family"] == "dofivik":
            own = i % 8 == 3
            if attention:
                w = 1536 * D + H * 192 * 1536 + 2 * H * 128 * 512 + H * D + H * 128 * D + (576 * D if own else 0) + 2 * D * ff
                out.append((w, 0, 2 * H * (192 + 128), 576 * size if own else 0, 6 * D * 4, 2048))
            else:
                out.append((6 * D * D + 128 * D + 2 * D * ff, 8 * D * 64, 0, 0, (6 * D + D * 64) * 4, 0))
        elif attention:
            g = max(1, H // 4)
            out.append((H * 128 * D + g * 256 * D + H * 128 * D + 3 * D * ff, 0, 4 * H * (64 + 128), g * 256 * size, 0, 2048))
        else:
            out.append((H * (2 * 64 + 2 * 128) * D + 16 * D + H * 64 * 16 + H * 128 * D + 3 * D * ff, 4 * H * 64 * 128, 0, 0, H * 64 * 128 * 4, 0))
    return out


def _pass_cost(case, batch, new, past, rows=1):
    """(bytes, FLOPs) of one forward of `new` tokens per sequence behind `past` cached ones, with the logits of `rows` of them."""
    m = MODELS[case["model"]]
    D, size = m["width"], 4 if case["weights"] == "f32" else 2
    by = VOCAB * D * size + batch * new * (D * size + 8) + batch * rows * VOCAB * (2 if case["family"] == "llama" else 4)
    fl = 2 * batch * rows * VOCAB * D
    for w, per_token, per_pair, cached, state, window in _layer_costs(case):
        pairs = sum(min(past + i + 1, window) for i in range(new)) if per_pair else 0
        seen = min(past, window)
        by += w * WEIGHT_BYTES[case["weights"]] + batch * ((new + seen) * cached + state * (2 if past else 1))
        fl += batch * (new * (2 * w + per_token) + pairs * per_pair)
    return by, fl


def work(case):
    if case["kind"] == "op":
        m, n, k = case["m"], case["n"], case["k"]
        if case["form"] == "mlp":
            return {"bytes": 3 * n * k * WEIGHT_BYTES["mxfp4"] + 2 * m * (2 * k + n), "flops": 6 * m * n * k}
        return {"bytes": n * k * WEIGHT_BYTES[case["weights"]] + 2 * (m * (n + k) + n), "flops": 2 * m * n * k}
    B, S = case["batch"], case["tokens"]
    if case["kind"] == "step":
        passes = [(1, S)]
    elif case["kind"] == "prefill":
        passes = [(S, 0)]
    else:
        passes = [(S, 0)] + [(1, S + i) for i in range(case["new"] - 1)] + [(S + case["new"], 0, case["new"])]
    costs = [_pass_cost(case, B, *p) for p in passes]
    return {"bytes": sum(c[0] for c in costs), "flops": sum(c[1] for c in costs)}


def tolerance(case):
    """Sums in 32 bits, and matrix operands rounded to bf16 once per layer and use: a right result is up to 2e-3 (MXFP4) or 6e-3
    (int8, which rounds activations to 8 bits) off for one linear and up to 1.6e-2 for a whole model, 5e-6 in float32."""
    if case["weights"] == "f32":
        return {"rel": 2e-5, "max": 2e-4}
    if case["kind"] == "op":
        return {"rel": 1e-2, "max": 4e-2}
    return {"rel": 2.5e-2, "max": 2e-1}


# ---------------------------------------------------------------- the same in 64 bits
def _mxfp4(w):
    """Values of w after quantization to E2M1 with a power-of-two scale per 32 inputs (round to nearest even, saturating)."""
    b = w.double().view(w.shape[0], -1, 32)
    top = b.abs().amax(-1, keepdim=True)
    scale = torch.where(top > 0, torch.exp2(torch.floor(torch.log2(top.clamp(min=1e-30))) - 2), torch.ones_like(top))
    a = (b / scale).abs()
    step = torch.where(a < 2, 0.5, torch.where(a < 4, 1.0, 2.0))
    return (torch.sign(b) * (torch.round(a / step) * step).clamp(max=6) * scale).view(w.shape)


def _int8(w):
    b = w.double().view(w.shape[0], -1, INT8_BLOCK)
    scale = (b.abs().amax(-1, keepdim=True) / 127.0).float()
    q = torch.round(b.float() * torch.where(scale > 0, 1 / scale, torch.zeros_like(scale))).clamp(-127, 127)
    return (q.double() * scale.double()).view(w.shape)


def _values(w, weights):
    return {"mxfp4": _mxfp4, "qint8": _int8}.get(weights, lambda t: t.double())(w)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _softmax_rows(score, value):
    """score [B, H, S, L] -> softmax over L times value [B, H, L, e], as [B, S, H * e]."""
    o = torch.softmax(score, -1) @ value
    return o.transpose(1, 2).flatten(2)


def _llama_exact(case, seed, ids, keep, cached=None):
    """(final normed hidden states [B, S, D], keys and values [layers] of [B, kv_heads, L, H])."""
    m = MODELS[case["model"]]
    D, Hq, Hk, ff, hd = m["width"], m["heads"], m["kv_heads"], m["ff"], m["width"] // m["heads"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda n, k: (torch.randn(n, k, generator=g, device="cuda") * WEIGHT_STD["llama"]).to(torch.bfloat16)
    rnd(VOCAB, D)  # the embedding that _embedding's replaces
    B, S = ids.shape
    past = 0 if cached is None else case["tokens"]
    keep = torch.ones(B, past + S, device="cuda", dtype=torch.int64) if keep is None else keep
    pos = (keep.cumsum(-1) - 1).clamp(min=0)[:, past:]
    inv = 1.0 / (m["theta"] ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd))
    angle = torch.outer(torch.arange(MAX_POS, dtype=torch.float32), inv)
    cos, sin = (f(angle).cuda().double()[pos].unsqueeze(1) for f in (torch.cos, torch.sin))
    lowest = torch.finfo(torch.bfloat16).min
    hidden = torch.ones(S, past + S, device="cuda", dtype=torch.bool).triu(past + 1)
    x = _embedding(case, seed)[0][ids].double()
    kv = []

    def rotate(t):
        a, b = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(m["layers"]):
        w = {n: rnd(*s) for n, s in (("q", (Hq * hd, D)), ("k", (Hk * hd, D)), ("v", (Hk * hd, D)), ("o", (D, Hq * hd)), ("gate", (ff, D)), ("up", (ff, D)),
                                     ("down", (D, ff)))}
        lin = lambda t, n: t @ _values(w[n], case["weights"]).T
        h = _rms(x, 1e-5)
        q, k, v = (lin(h, n).view(B, S, -1, hd).transpose(1, 2) for n in "qkv")
        q, k = rotate(q), rotate(k)
        if cached is not None:
            k, v = (torch.cat([c.double(), t], 2) for c, t in zip(cached[i], (k, v)))
        kv.append((k, v))
        ctx = []
        for b in range(B):  # one sequence at a time: the scores in 64 bits are large
            s = q[b].view(Hk, Hq // Hk, S, hd) @ k[b].unsqueeze(1).transpose(-1, -2) / math.sqrt(hd)
            s += torch.where(keep[b] > 0, 0.0, lowest)
            s = s.masked_fill_(hidden, -math.inf).view(1, Hq, S, -1)
            ctx.append(_softmax_rows(s, v[b].repeat_interleave(Hq // Hk, 0).unsqueeze(0)))
        x = x + lin(torch.cat(ctx), "o")
        h = _rms(x, 1e-5)
        x = x + lin(torch.nn.functional.silu(lin(h, "gate")) * lin(h, "up"), "down")
    return _rms(x, 1e-5), kv


def _drawn(shapes, order, seed, std):
    """Matrices of a hybrid decoder in the order in which they are drawn: name -> fp64 tensor, layer by layer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    for prefix in order:
        yield {n[len(prefix):]: (torch.randn(*s, generator=g, device="cuda") * std).to(torch.bfloat16).double()
               for n, s in shapes.items() if n.startswith(prefix) and len(s) == 2}


def _heads(t, n):
    return t.view(t.shape[0], t.shape[1], n, -1)


def _seen(pos, keep, same):
    """[B, 1, S, S]: which key positions a query meets."""
    i, j = pos.unsqueeze(-1), pos.unsqueeze(-2)
    return ((j <= i) & same(i, j) & keep.unsqueeze(-2)).unsqueeze(1)


def _attend(q, k, v, seen, score):
    """q, k [B, S, H, d], v [B, S, H, e]; rows of padding come out as zero."""
    out = []
    for b in range(q.shape[0]):
        s = score(q[b].transpose(0, 1) @ k[b].permute(1, 2, 0)).masked_fill_(~seen[b], -math.inf).unsqueeze(0)
        out.append(_softmax_rows(s, v[b].transpose(0, 1).unsqueeze(0)).nan_to_num_(0.0))
    return torch.cat(out)


def _dofivik_exact(case, seed, ids, keep):
    """(final normed hidden states, states per layer)."""
    shape = _shape(case)
    eps, alpha, D, std, taps = shape.norm_eps, shape.postln_alpha, shape.hidden_size, WEIGHT_STD["dofivik"], shape.taps
    B, S = ids.shape
    live = (torch.ones_like(ids) if keep is None else keep).bool()
    pos = (live.long().cumsum(-1) - 1).clamp(min=0)
    x = _embedding(case, seed)[0][ids].double() * live.unsqueeze(-1)
    latents, states = {}, []

    def conv(t, w):
        padded = torch.nn.functional.pad(t, (0, 0, taps - 1, 0))
        return t + sum(padded[:, j:j + S] * w[:, j] for j in range(taps)), padded[:, S:]

    def rotate(t, base):
        dims = t.shape[-1]
        ang = pos.double()[..., None, None] * base ** (-torch.arange(0, dims, 2, device="cuda").double() / dims)
        c, s, u, v = torch.cos(ang), torch.sin(ang), t[..., 0::2], t[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    weights = _drawn(FD.tensor_shapes(shape), [f"l{i}." for i in range(len(shape.layers))], seed, std)
    for i, (entry, w) in enumerate(zip(shape.layers, weights)):
        m, kept = entry["mixer"], {}
        H, d = m["heads"], m["dim"]
        h, kept["conv1"] = conv(x, w["canon1"])
        if entry["type"] == "latent_attention":
            j = m.get("kv_from", i)
            if j == i:
                both = h @ w["mix.dkv"].T
                latents[i] = _rms(both[..., :m["kv_rank"]], eps), rotate(both[..., None, m["kv_rank"]:], m["rot"]["base"])
            c, k_rot = latents[j]
            q = _heads(_rms(h @ w["mix.dq"].T, eps) @ w["mix.uq"].T, H)
            q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"]["base"])], -1)
            k = torch.cat([_heads(c @ w["mix.uk"].T, H), k_rot.expand(-1, -1, H, -1)], -1)
            seen = _seen(pos, live, lambda a, b: a - b < m["mask"]["size"])
            o = _attend(q, k, _heads(c @ w["mix.uv"].T, H), seen, lambda s: s * m["scale"])
            y = (_heads(o, H) * torch.sigmoid(h @ w["mix.g"].T).unsqueeze(-1)).flatten(2) @ w["mix.o"].T
        else:
            r, k, v = (_heads(h @ w["mix." + n].T, H) for n in "rkv")
            decay = _heads(torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w["mix.w1"].T) @ w["mix.w2"].T)), H)
            u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            ru = _heads(torch.sigmoid(h @ w["mix.a"].T), H) * u
            state, o = torch.zeros(B, H, d, d, device="cuda", dtype=torch.float64), torch.empty_like(v)
            for t in range(S):
                state = (decay[:, t].unsqueeze(-1) * state - ru[:, t].unsqueeze(-1) * (u[:, t].unsqueeze(-2) @ state)
                         + k[:, t].unsqueeze(-1) * v[:, t].unsqueeze(-2))
                o[:, t] = (r[:, t].unsqueeze(-2) @ state).squeeze(-2)
            kept["delta"] = state
            y = (_rms(o, eps).flatten(2) * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
        x = _rms(alpha * x + y, eps) * live.unsqueeze(-1)
        h, kept["conv2"] = conv(x, w["canon2"])
        z = h @ w["mlp.up"].T
        p = math.log(2.0)  # softplus(0), both parameters of the activation being zero
        z = torch.where(z > 0, p * z * z, (0.5 + p) * (torch.expm1(z.clamp(max=0)) - z)) + 0.5 * z
        x = _rms(alpha * x + z @ w["mlp.down"].T, eps) * live.unsqueeze(-1)
        states.append(kept)
    return _rms(x, eps), states


def _vedizen_exact(case, seed, ids, keep):
    """(final normed hidden states, states per layer)."""
    shape = _shape(case)
    B, S = ids.shape
    live = (torch.ones_like(ids) if keep is None else keep).bool()
    pos = (live.long().cumsum(-1) - 1).clamp(min=0)
    on = live.unsqueeze(-1)
    x = _embedding(case, seed)[0][ids].double() * shape.embed_scale * on
    states = []
    weights = _drawn(FV.tensor_shapes(shape), [f"l{i}." for i in range(len(shape.layers))], seed, WEIGHT_STD["vedizen"])
    for entry, w in zip(shape.layers, weights):
        m, kept = entry["mixer"], {}
        H, d, e = m["heads"], m["dim"], m["vdim"]
        h = torch.tanh(0.5 * x) * on
        if entry["type"] == "gla":
            q, k, v = (_heads(h @ w["mix." + n].T, H) for n in "qkv")
            decay = _heads(torch.sigmoid(h @ w["mix.a1"].T @ w["mix.a2"].T + 2.0) ** (1 / m["tau"]), H)
            state, o = torch.zeros(B, H, d, e, device="cuda", dtype=torch.float64), torch.empty_like(v)
            for t in range(S):
                state = torch.addcmul(decay[:, t].unsqueeze(-1) * state, k[:, t].unsqueeze(-1), v[:, t].unsqueeze(-2))
                o[:, t] = (q[:, t].unsqueeze(-2) @ state).squeeze(-2)
            kept["gla"] = state
            y = (_rms(o * d ** -0.5, shape.norm_eps).flatten(2) * torch.nn.functional.silu(h @ w["mix.g"].T)) @ w["mix.o"].T
        else:
            g = m["kv_heads"]
            q, k, v = _heads(h @ w["mix.q"].T, 2 * H), _heads(h @ w["mix.k"].T, 2 * g), _heads(h @ w["mix.v"].T, g)
            seen = _seen(pos, live, lambda a, b: a // m["mask"]["size"] == b // m["mask"]["size"])
            cap = lambda s: m["softcap"] * torch.tanh(s * (m["scale"] / m["softcap"]))
            one, two = (_attend(q[:, :, z::2], k[:, :, z::2].repeat_interleave(H // g, 2), v.repeat_interleave(H // g, 2), seen, cap) for z in (0, 1))
            o = _rms(_heads(one - m["diff"] * two, H), shape.norm_eps) * (1 - m["diff"])  # lambda is its constant part: lq1 lk1 = lq2 lk2
            y = o.flatten(2) @ w["mix.o"].T
        lim = entry["mlp"]["limit"]
        gate, up = (h @ w["mlp.gate"].T).clamp(max=lim), (h @ w["mlp.up"].T).clamp(-lim, lim)
        x = x + (y + (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w["mlp.down"].T) * on
        states.append(kept)
    return torch.tanh(0.5 * x), states


def _paged(k, pages):
    """[B, heads, L, H] -> the cache's [pages, B, heads, 32, H], zero behind the last token."""
    B, G, L, H = k.shape
    return torch.nn.functional.pad(k, (0, 0, 0, pages * 32 - L)).view(B, G, pages, 32, H).permute(2, 0, 1, 3, 4)


def exact(case, seed):
    if case["kind"] == "op":
        x, ws, bias = _op_inputs(case, seed)
        x, ws = x.double(), [_values(w, case["weights"]) for w in ws]
        if case["form"] == "mlp":
            h = torch.nn.functional.silu(x @ ws[0].T) * (x @ ws[1].T)
            return {"hidden": h, "out": h @ ws[2].T}
        return {"out": torch.nn.functional.silu(x @ ws[0].T + bias.double())}
    head = _embedding(case, seed)[1].double()
    model = {"llama": _llama_exact, "dofivik": _dofivik_exact, "vedizen": _vedizen_exact}[case["family"]]
    if case["kind"] == "step":
        ids = torch.randint(0, VOCAB, (case["batch"], 1), generator=torch.Generator().manual_seed(seed + 2)).cuda()
        h, kv = model(case, seed, ids, None, _cached(case, seed))
        pages = (case["tokens"] + 128 + 31) // 32
        return {"logits": h @ head.T, "cache": [[_paged(t, pages) for t in both] for both in kv]}
    ids, keep = _prompt(case, seed)
    if case["kind"] == "prefill":
        h, kept = model(case, seed, ids, keep)
        if case["family"] != "llama":
            return {"logits": h[:, -1:] @ head.T, "states": kept}
        pages = (case["tokens"] + 128 + 31) // 32
        return {"logits": h[:, -1:] @ head.T, "cache": [[_paged(t, pages) for t in both] for both in kept]}
    # the greedy continuation: a guess is the answer once every token of it is the choice behind those before it
    new, S = case["new"], case["tokens"]
    text = torch.cat([ids] + [(ids[:, -1:] + 1 + i) % VOCAB for i in range(new)], 1)
    keep = None if keep is None else torch.cat([keep, keep.new_ones(keep.shape[0], new)], 1)
    for _ in range(new):
        h, _ = model(case, seed, text, keep)
        best = (h[:, S - 1:-1] @ head.T).argmax(-1)
        if torch.equal(best, text[:, S:]):
            break
        text = torch.cat([ids, best], 1)
    return {"text": text, "logits": (h[:, S - 1:-1] @ head.T).flatten(0, 1)}
