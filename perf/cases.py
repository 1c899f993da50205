"""The calls whose speed this library answers for, at the sizes of its own configurations (LLaMA-7B, Baichuan-13B and
LLaMA-65B widths), each through a public entry point: single projections, the FFN and attention ops in prefill and
decode, a replayed decode step of a model, and the quantizer.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program holds before the call,
run() is the call, work() the bytes and operations that it cannot do without, exact() the same result in 64 bits."""
import math
import types

import torch

from eet_b200 import EET, modeling

EPS = 1e-6
ROPE_BASE = 10000.0
D = 128
VOCAB = 32000
# hidden size -> (heads, FFN size)
WIDTHS = {4096: (32, 11008), 5120: (40, 13696), 8192: (64, 22016)}
# (reduction, output) sizes of the projections: fused QKV, attention output, gate / up, down
PROJECTIONS = tuple(kn for h, (_, f) in WIDTHS.items() for kn in ((h, 3 * h), (h, h), (h, f), (f, h)))


def listed():
    return [
        # one user's decode step, the attention output projection with its residual: the smallest call there is
        {"name": "linear_m1", "op": "linear", "M": 1, "K": 4096, "N": 4096, "residual": True},
        # a dozen users' decode step, the fused QKV projection of the 13B width
        {"name": "linear_m12", "op": "linear", "M": 12, "K": 5120, "N": 15360, "residual": False},
        # a short prompt or a chunk of one, gate / up projection: a row count that fits no tile
        {"name": "linear_m100", "op": "linear", "M": 100, "K": 4096, "N": 11008, "residual": False},
        # 8 prompts of 512 tokens, down projection with its residual
        {"name": "linear_m4096", "op": "linear", "M": 4096, "K": 11008, "N": 4096, "residual": True},
        # a long batch of prompts at the 65B width, gate / up projection: the largest call
        {"name": "linear_m8192", "op": "linear", "M": 8192, "K": 8192, "N": 22016, "residual": False},
        # the FFN op as the model calls it in a decode step of 8 sequences
        {"name": "ffn_decode_b8", "op": "ffn", "B": 8, "S": 1, "hidden": 4096},
        # the FFN op over three ragged prompts at the 13B width
        {"name": "ffn_prefill_3x333", "op": "ffn", "B": 3, "S": 333, "hidden": 5120},
        # the attention op in a decode step, a thousand tokens of history
        {"name": "attention_decode_b8", "op": "attention", "B": 8, "S": 999, "hidden": 4096, "alibi": False,
         "decode": True, "padded": False},
        # the attention op over two long, left-padded prompts
        {"name": "attention_prefill_2x2048", "op": "attention", "B": 2, "S": 2048, "hidden": 4096, "alibi": False,
         "decode": False, "padded": True},
        # the same with ALiBi instead of rotary embedding, odd length
        {"name": "attention_prefill_alibi", "op": "attention", "B": 2, "S": 701, "hidden": 5120, "alibi": True,
         "decode": False, "padded": False},
        # a decode step of a model as it is served: captured once, replayed; 8 sequences of 512 tokens
        {"name": "decode_step_b8", "op": "model", "B": 8, "S": 512, "hidden": 4096, "alibi": False, "layers": 4},
        # quantizing and packing one FFN matrix, as loading and updating a model do for each
        {"name": "quantize_4096x11008", "op": "quantize", "K": 4096, "N": 11008, "fp32": False},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(("linear", "linear", "linear", "ffn", "ffn", "attention", "attention", "attention", "model", "quantize"))
    hidden = rng.choice((4096, 5120))
    if op == "linear":
        K, N = rng.choice(PROJECTIONS)
        return {"op": op, "M": _log_int(rng, 1, 8192 if N <= 22016 else 4096), "K": K, "N": N, "residual": rng.random() < 0.5}
    if op == "quantize":
        K, N = rng.choice(PROJECTIONS)
        return {"op": op, "K": K, "N": N, "fp32": rng.random() < 0.25}
    if op == "ffn":
        if rng.random() < 0.5:
            return {"op": op, "B": _log_int(rng, 1, 64), "S": 1, "hidden": hidden}
        S = _log_int(rng, 8, 1024)
        return {"op": op, "B": _log_int(rng, 1, max(1, min(8, 4096 // S))), "S": S, "hidden": hidden}
    S = _log_int(rng, 16, 2048 if op == "attention" else 1024)
    if op == "model":
        return {"op": op, "B": _log_int(rng, 1, max(1, min(32, 4096 // S))), "S": S, "hidden": hidden,
                "alibi": hidden == 5120, "layers": rng.choice((2, 3))}
    B, decode = _log_int(rng, 1, max(1, min(32, 4096 // S))), rng.random() < 0.5
    alibi = hidden == 5120
    return {"op": op, "B": B, "S": S, "hidden": hidden, "alibi": alibi, "decode": decode,
            "padded": not alibi and rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _half(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).half()


def _int8(gen, K, N):
    """A quantized N(0, 0.02^2) matrix: int8 values of which the largest of a column is near 127, and its scales."""
    q = (torch.randn(K, N, generator=gen, device="cuda") * 30).round_().clamp_(-127, 127).to(torch.int8)
    return q, ((1 + 0.1 * torch.rand(N, generator=gen, device="cuda")) * (0.02 / 30)).half()


def _gamma(gen, n):
    return (1 + 0.1 * torch.randn(n, generator=gen, device="cuda")).half()


def _pads(case):
    """Left padding of each prompt: none for the first, up to a third of the prompt for the last."""
    B, S = case["B"], case["S"]
    return torch.tensor([[b * (S // 3) // max(1, B - 1)] for b in range(B)], dtype=torch.int64, device="cuda")


def _slopes(n):
    def pow2(m):
        return [2.0 ** (-8.0 * (i + 1) / m) for i in range(m)]
    c = 2 ** int(math.log2(n))
    return pow2(n) if c == n else pow2(c) + pow2(2 * c)[0::2][: n - c]


def _bias(heads, rows, cols):
    """fp16 ALiBi bias [heads, len(rows), cols]: slope * position of the key, -inf above the diagonal."""
    s = torch.tensor(_slopes(heads), dtype=torch.float32, device="cuda")
    t = torch.arange(cols, device="cuda")
    m = (s[:, None, None] * t[None, None, :].float()).expand(heads, len(rows), cols)
    return m.masked_fill((t[None, :] > torch.tensor(list(rows), device="cuda")[:, None])[None], float("-inf")).half().contiguous()


def _layer(gen, hidden):
    f = WIDTHS[hidden][1]
    return {"ln1": _gamma(gen, hidden), "qkv": _int8(gen, hidden, 3 * hidden), "out": _int8(gen, hidden, hidden),
            "ln2": _gamma(gen, hidden), "gate": _int8(gen, hidden, f), "up": _int8(gen, hidden, f), "down": _int8(gen, f, hidden)}


def _inputs(case, seed):
    gen, op = _gen(seed), case["op"]
    if op == "linear":
        q, s = _int8(gen, case["K"], case["N"])
        return {"x": _half(gen, case["M"], case["K"]), "q": q, "s": s,
                "residual": _half(gen, case["M"], case["N"]) if case["residual"] else None}
    if op == "quantize":
        w = torch.randn(case["K"], case["N"], generator=gen, device="cuda") * 0.02
        return {"w": w if case["fp32"] else w.half()}
    h = case["hidden"]
    if op == "ffn":
        f = WIDTHS[h][1]
        return {"x": _half(gen, case["B"], case["S"], h), "ln": _gamma(gen, h), "gate": _int8(gen, h, f),
                "up": _int8(gen, h, f), "down": _int8(gen, f, h)}
    if op == "attention":
        return {"prompt": _half(gen, case["B"], case["S"], h), "token": _half(gen, case["B"], 1, h), "ln": _gamma(gen, h),
                "qkv": _int8(gen, h, 3 * h), "out": _int8(gen, h, h)}
    return {"layers": [_layer(gen, h) for _ in range(case["layers"])], "ln": _gamma(gen, h),
            "embed": _half(gen, VOCAB, h, std=0.5), "head": _half(gen, VOCAB, h, std=0.02),
            "prompt": torch.randint(0, VOCAB, (case["B"], case["S"]), generator=gen, device="cuda"),
            "token": torch.randint(0, VOCAB, (case["B"], 1), generator=gen, device="cuda")}


# ---------------------------------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------------------------------
_NONE = torch.empty(0)


def _pack(qs):
    return EET.preprocess_weights(qs[0]), qs[1]


def prepare(case, seed):
    i, op = _inputs(case, seed), case["op"]
    if op == "linear":
        w, s = _pack((i["q"], i["s"]))
        return {"case": case, "x": i["x"], "w": w, "s": s, "residual": i["residual"]}
    if op == "quantize":
        return {"case": case, "w": i["w"]}
    h = case["hidden"]
    heads, f = WIDTHS[h]
    if op == "ffn":
        desc = EET.MetaDesc(torch.float16, case["B"], heads, h, 1, case["S"], case["S"], "silu", D, f, "cuda:0", False, EPS, True)
        (w0, s0), (w1, s1), (w2, s2) = (_pack(i[k]) for k in ("gate", "up", "down"))
        ffn = EET.GatedFeedForwardNetworkInt8(desc, w0, s0, _NONE, w1, s1, _NONE, w2, s2, _NONE, i["ln"], _NONE)
        return {"case": case, "x": i["x"], "ffn": ffn}
    B, S = case["B"], case["S"]
    if op == "attention":
        desc = EET.MetaDesc(torch.float16, B, heads, h, 1, S, S + 32, "silu", D, f, "cuda:0", False, EPS, True)
        (w0, s0), (w1, s1) = _pack(i["qkv"]), _pack(i["out"])
        cls = EET.BaichuanMmha if case["alibi"] else EET.LlamaMmha
        mmha = cls(desc, w0, s0, _NONE, _NONE, _NONE, w1, s1, _NONE, i["ln"], _NONE)
        state = {"case": case, "mmha": mmha, "pad": _pads(case) if case["padded"] else _NONE, "x": i["prompt"]}
        state["bias"] = _bias(heads, range(S), S) if case["alibi"] else _NONE
        if case["decode"]:
            mmha.forward(i["prompt"], state["pad"], _NONE, True, True, True, state["bias"])
            state["x"] = i["token"]
            state["bias"] = _bias(heads, [S], S + 1) if case["alibi"] else _NONE
        return state
    cfg = types.SimpleNamespace(hidden_size=h, num_attention_heads=heads, num_hidden_layers=case["layers"], intermediate_size=f,
                                vocab_size=VOCAB, rms_norm_eps=EPS, hidden_act="silu", pad_token_id=None)
    weights = {"embed_tokens.weight": i["embed"], "norm.weight": i["ln"], "lm_head.weight": i["head"]}
    names = {"qkv": "self_attn.qkv_proj", "out": "self_attn.out_proj", "gate": "ffn.intermediate_0", "up": "ffn.intermediate_1",
             "down": "ffn.output"}
    for n, layer in enumerate(i["layers"]):
        p = "layer.%d." % n
        weights[p + "self_attn.layernorm.weight"], weights[p + "ffn.layernorm.weight"] = layer["ln1"], layer["ln2"]
        for k, name in names.items():
            weights[p + name + ".weight"], weights[p + name + ".scale"] = _pack(layer[k])
    cls = modeling.EETBaichuanForCausalLM if case["alibi"] else modeling.EETLlamaForCausalLM
    model = cls.from_eet(weights, cfg, B, S, S + 128, torch.int8, lm_head_int8=True)
    model.model(i["prompt"], first_pass=True)
    # the step behind the prompt is captured with its position on the device, as a server does that replays it while the
    # position advances; here the position stays, so that every replay is the same step (the eager call before it, which
    # sizes the pooled buffers, is that step too)
    ops = [layer.attention for layer in model.model.layers]
    model.decode_logits(i["token"])
    for op_ in ops:
        op_.sync_device_step()
        op_.use_device_step = True
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = model.decode_logits(i["token"])
    return {"case": case, "model": model, "token": i["token"], "graph": graph, "logits": logits}


# ---------------------------------------------------------------------------------------------------
# the call
# ---------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "linear":
        return EET.gemm_w8a16(state["x"], state["w"], state["s"], residual=state["residual"])
    if op == "quantize":
        return EET.quant_weights(state["w"])
    if op == "ffn":
        return state["ffn"].forward(state["x"], True, True)
    if op == "attention":
        mmha, S = state["mmha"], case["S"]
        if case["decode"]:
            mmha.step_ = S   # the same step again
            out = mmha.forward(state["x"], state["pad"], _NONE, True, True, False, state["bias"])
            return out, mmha.k_cache[:, :, S], mmha.v_cache[:, :, S]
        out = mmha.forward(state["x"], state["pad"], _NONE, True, True, True, state["bias"])
        return out, mmha.k_cache[:, :, :S], mmha.v_cache[:, :, :S]
    state["graph"].replay()
    return state["logits"]


# ---------------------------------------------------------------------------------------------------
# what the call cannot do without
# ---------------------------------------------------------------------------------------------------
def _gemm_work(M, K, N):
    return {"bytes": K * N + 2 * N + 2 * M * K + 2 * M * N, "flops": 2 * M * K * N}


def _add(*works):
    return {k: sum(w[k] for w in works) for k in ("bytes", "flops")}


def _attention_work(B, S, h, decode, bias):
    heads = WIDTHS[h][0]
    if decode:
        core = {"bytes": 4 * B * S * h + 8 * B * h, "flops": 4 * B * (S + 1) * h}
        rows = B
    else:
        core = {"bytes": 8 * B * S * h, "flops": 2 * B * S * (S + 1) * h}   # Q, K, V in, context out; causal half
        rows = B * S
    if bias:
        core["bytes"] += 2 * heads * (S + 1 if decode else S * (S + 1) // 2)
    return _add(_gemm_work(rows, h, 3 * h), core, _gemm_work(rows, h, h), {"bytes": 2 * rows * h, "flops": 0})


def _ffn_work(M, h):
    # x (norm and residual read the same bytes) -> gate, up -> down + residual
    f = WIDTHS[h][1]
    return {"bytes": 3 * h * f + 2 * (2 * f + h) + 4 * M * h, "flops": 6 * M * h * f}


def work(case):
    op = case["op"]
    if op == "linear":
        w = _gemm_work(case["M"], case["K"], case["N"])
        return _add(w, {"bytes": 2 * case["M"] * case["N"] if case["residual"] else 0, "flops": 0})
    if op == "quantize":
        return {"bytes": ((4 if case["fp32"] else 2) + 1) * case["K"] * case["N"], "flops": 0}
    if op == "ffn":
        return _ffn_work(case["B"] * case["S"], case["hidden"])
    if op == "attention":
        return _attention_work(case["B"], case["S"], case["hidden"], case["decode"], case["alibi"])
    B, S, h = case["B"], case["S"], case["hidden"]
    layer = _add(_attention_work(B, S, h, True, False), _ffn_work(B, h))
    return _add(*([layer] * case["layers"] + [_gemm_work(B, h, VOCAB)]))


def tolerance(case):
    """About four times the distance from the 64-bit result that a correct run shows; that distance is at each line."""
    op = case["op"]
    if op == "quantize":
        return "exact"
    if op == "linear":
        return {"rel": 1e-3}                              # 2.1e-4 to 2.9e-4: one rounding to fp16, two with a residual
    if op == "ffn":
        return {"rel": 2.5e-3}                            # 6.2e-4 to 6.4e-4
    if op == "attention":
        return {"rel": 3e-3 if case["alibi"] else 2e-3}   # 6.8e-4 with ALiBi, 4.0e-4 to 5.4e-4 without
    return {"rel": 2e-2 if case["alibi"] else 1e-2}       # 1.7e-3 to 2.4e-3; with ALiBi logits are rounded in fp16 beside
                                                          # a bias of hundreds, where a last bit is 0.125


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------
def _lin(x, qs, cols=slice(None)):
    q, s = qs[0][:, cols], qs[1][cols]
    out = torch.empty(x.shape[0], q.shape[1], dtype=torch.float64, device=x.device)
    for n in range(0, q.shape[1], 4096):
        out[:, n:n + 4096] = (x @ q[:, n:n + 4096].double()) * s[n:n + 4096].double()
    return out


def _norm(x, gamma):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * gamma.double()


def _rope(x, first):
    """x [B, H, S, D] rotated at positions first, first + 1, ..."""
    t = torch.arange(first, first + x.shape[2], dtype=torch.float64, device=x.device)
    a = t[:, None] / ROPE_BASE ** (torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    c, s = a.cos(), a.sin()
    u, v = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _heads(y, B, S):
    return y.view(B, S, -1, D).transpose(1, 2)


def _softmax_v(q, k, v, keep, bias):
    """Softmax of q k^T / sqrt(D) (+ bias) over the positions in `keep`; rows that keep nothing are zero."""
    out = torch.empty_like(q)
    scale = float(torch.tensor(math.sqrt(1.0 / D)).half())
    for b in range(q.shape[0]):
        for h in range(q.shape[1]):
            s = (q[b, h] @ k[b, h].t()) * scale
            if bias is not None:
                s = s + bias[h].double()
            s = s.masked_fill(~keep[b], float("-inf"))
            p = torch.exp(s - s.amax(-1, keepdim=True).clamp_min(-1e20))
            out[b, h] = (p / p.sum(-1, keepdim=True).clamp_min(1e-6)) @ v[b, h]
    return out


def _attention(x, ln, qkv, out, cache, pad, alibi, need_out=True):
    """One attention block for x [B, S, h] behind the history in `cache` (a list [k, v] or empty), which it extends."""
    B, S, h = x.shape
    heads = h // D
    xn = _norm(x.reshape(B * S, h), ln)
    first = cache[0].shape[2] if cache else 0
    k, v = (_heads(_lin(xn, qkv, slice(n * h, (n + 1) * h)), B, S) for n in (1, 2))
    if not alibi:
        k = _rope(k, first)
    cache[:] = [torch.cat([cache[0], k], 2), torch.cat([cache[1], v], 2)] if cache else [k, v]
    if not need_out:
        return None
    q = _heads(_lin(xn, qkv, slice(0, h)), B, S)
    q = q if alibi else _rope(q, first)
    i = torch.arange(first, first + S, device=x.device)
    j = torch.arange(first + S, device=x.device)
    keep = (j[None, :] <= i[:, None])[None].expand(B, -1, -1)
    if pad is not None:
        keep = keep & (j[None, None, :] >= pad.view(B, 1, 1))
    ctx = _softmax_v(q, *cache, keep, _bias(heads, range(first, first + S), first + S) if alibi else None)
    return x + _lin(ctx.transpose(1, 2).reshape(B * S, h), out).view(B, S, h)


def _ffn(x, ln, gate, up, down):
    x2 = x.reshape(-1, x.shape[-1])
    xn = _norm(x2, ln)
    return (x2 + _lin(torch.nn.functional.silu(_lin(xn, gate)) * _lin(xn, up), down)).view(x.shape)


def _quantize(w):
    """Symmetric per column: scale = amax / 128 in fp32, halves away from zero, [-128, 127]."""
    s = w.float().abs().amax(0) * (1.0 / 128.0)
    r = w.float() / s
    return torch.where(r < 0, torch.ceil(r - 0.5), torch.floor(r + 0.5)).clamp(-128, 127).to(torch.int8), s


def exact(case, seed):
    op = case["op"]
    if op == "quantize":
        return None   # whole numbers and scales of 16 or 32 bits, compared bit for bit
    i = _inputs(case, seed)
    if op == "linear":
        y = _lin(i["x"].double(), (i["q"], i["s"]))
        return y if i["residual"] is None else y + i["residual"].double()
    if op == "ffn":
        return _ffn(i["x"].double(), i["ln"], i["gate"], i["up"], i["down"])
    B, S = case["B"], case["S"]
    if op == "attention":
        pad, cache = _pads(case) if case["padded"] else None, []
        args = (i["ln"], i["qkv"], i["out"], cache, pad, case["alibi"])
        out = _attention(i["prompt"].double(), *args, need_out=not case["decode"])
        if not case["decode"]:
            return out, cache[0], cache[1]
        out = _attention(i["token"].double(), *args)
        return out, cache[0][:, :, S], cache[1][:, :, S]
    caches = [[] for _ in i["layers"]]
    x = None
    for ids, last in ((i["prompt"], False), (i["token"], True)):
        x = i["embed"][ids].double()
        for n, (layer, cache) in enumerate(zip(i["layers"], caches)):
            final = n + 1 < case["layers"] or last
            x = _attention(x, layer["ln1"], layer["qkv"], layer["out"], cache, None, case["alibi"], need_out=final)
            if final:
                x = _ffn(x, layer["ln2"], layer["gate"], layer["up"], layer["down"])
    q, s = _quantize(i["head"].t().contiguous())
    return _lin(_norm(x[:, -1], i["ln"]), (q, s.half())).view(B, 1, VOCAB)
