"""The work that users of this framework have it do, as measurable cases through its public entry points.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call: inputs, weights, engines
    run(state)          one pass
    work(case)          bytes and operations the pass cannot do without
    tolerance(case)     how far two correct implementations of the same precision may lie apart
    exact(case, seed)   the outputs of run() in 64 bits, by plain torch

Kinds of cases:
  linear        a quantised weight times activation rows (zig-nn's linear layers; one row per decoded token, several when
                sequences are decoded together, many for a prompt)
  tune          forward and backward to the activations through a frozen quantised weight (adapter training)
  gpt2, gemma3  a prompt, a greedy continuation on the device and one further step: `generate` of the command line
  gemma3_batch  several sequences: their prompts, then steps of all of them together
  decoder       Lenisun and Vepinex (bf16 weights): prompts, then steps whose tokens the program picks from the logits itself;
                one sequence or several
"""
import math

import numpy as np
import torch

from zignn_b200 import api, ggml, hostmodel

DEVICE = "cuda"
BLOCK_BYTES = {"q4_0": 18, "q4_1": 20, "q8_0": 34}

# Mixers, feed-forward parts and heads of the two bf16 designs by width: the `small` and `1b` columns of bench.py.
WIDTHS = {768: dict(heads=12, kv_heads=4, dim=64, ff=3072, wide=64), 1152: dict(heads=4, kv_heads=1, dim=256, ff=6912, wide=128)}
EXPERTS = dict(experts=32, top=4, ff=512)
RANK = 64  # low-rank parts of decays and gates


def listed():
    return [
        # One decoded token in the smallest matrix of the GPT-2 loop, bias included: launch and latency.
        dict(name="row_gpt2_qkv", kind="linear", type="q4_0", k=768, n=2304, rows=1, act="f32", bias=True),
        # One decoded token's logits: the Gemma-3 vocabulary head, the headline of bench.py.
        dict(name="row_vocabulary_head", kind="linear", type="q4_0", k=1152, n=262144, rows=1, act="f32", bias=False),
        # Sixteen sequences decoded together, Gemma-3's deepest matrix, 8-bit activations (bit-exact to the CPU path).
        dict(name="rows16_ffn_down_q8", kind="linear", type="q8_0", k=6912, n=1152, rows=16, act="q8", bias=False),
        # A short prompt, nothing a multiple of a tile: 37 blocks per row, an odd number of weight rows.
        dict(name="rows45_ragged", kind="linear", type="q4_1", k=1184, n=5003, rows=45, act="f32", bias=True),
        # A long prompt through the up projection of an 8B-sized model: the largest single product.
        dict(name="rows2048_ffn_up", kind="linear", type="q4_0", k=4096, n=14336, rows=2048, act="f32", bias=False),
        # One micro-batch of adapter training through Gemma-3's up projection.
        dict(name="tune_ffn_up", kind="tune", type="q8_0", k=1152, n=6912, rows=512),
        # A chat turn: short prompt, most of the time goes to decoded tokens.
        dict(name="gpt2_chat", kind="gpt2", type="q4_0", layers=12, prompt=32, tokens=64),
        # A document nearly as long as the context, few tokens after it: most of the time goes to the prompt.
        dict(name="gpt2_document", kind="gpt2", type="q8_0", layers=12, prompt=900, tokens=4),
        # Gemma-3-1B behind a prompt longer than its sliding window.
        dict(name="gemma3_generate", kind="gemma3", type="q8_0", layers=26, prompt=600, tokens=16),
        # Gemma-3-1B with 4-bit weights serving several short requests at once.
        dict(name="gemma3_batch", kind="gemma3_batch", type="q4_1", layers=26, prompt=40, tokens=12, sequences=8),
        # Attention and recurrent layers behind a long prompt.
        dict(name="lenisun_generate", kind="decoder", design="lenisun", width=1152, layers=12, experts=False, vocab=50304,
             prompt=1500, tokens=24, sequences=1),
        # Matrix memories, delta rules and latent attention serving several requests, every second pair of layers with experts.
        dict(name="vepinex_serve", kind="decoder", design="vepinex", width=768, layers=12, experts=True, vocab=50304,
             prompt=200, tokens=16, sequences=6),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["tune", "gpt2", "gpt2", "gemma3", "gemma3_batch", "decoder", "decoder"])
    kinds = ("q4_0", "q4_1", "q8_0")
    if kind in ("linear", "tune"):
        act = rng.choice(("f32", "f32", "q8")) if kind == "linear" else "f32"
        while True:
            k, n, rows = 32 * _log(rng, 8, 448), _log(rng, 256, 262144), _log(rng, 1, 2048)
            n -= n % 8 if kind == "tune" else 0  # the transposed product takes whole groups of eight weight rows
            if k * n <= 1152 * 262144 and rows * n <= 1 << 25 and rows * n * k <= (1 << 36 if act == "f32" else 1 << 34):
                break
        case = dict(kind=kind, type=rng.choice(kinds), k=k, n=n, rows=rows)
        return dict(case, act=act, bias=rng.random() < 0.5) if kind == "linear" else case
    if kind == "gpt2":
        return dict(kind=kind, type=rng.choice(kinds), layers=rng.randint(2, 12), prompt=_log(rng, 2, 900), tokens=rng.randint(1, 64))
    if kind == "gemma3":
        return dict(kind=kind, type=rng.choice(kinds), layers=rng.randint(4, 26), prompt=_log(rng, 2, 600), tokens=rng.randint(1, 16))
    if kind == "gemma3_batch":
        return dict(kind=kind, type=rng.choice(kinds), layers=rng.randint(4, 26), prompt=_log(rng, 2, 40), tokens=rng.randint(1, 12),
                    sequences=rng.randint(2, 8))
    sequences = rng.choice((1, 1, rng.randint(2, 6)))
    return dict(kind=kind, design=rng.choice(("lenisun", "vepinex")), width=rng.choice((768, 1152)), layers=rng.randint(4, 12),
                experts=rng.random() < 0.3, vocab=50304, prompt=_log(rng, 2, 1500 if sequences == 1 else 200), tokens=rng.randint(1, 16),
                sequences=sequences)


# ---- inputs --------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _linear_inputs(case, seed):
    g = _generator(seed)
    k, n, rows = case["k"], case["n"], case["rows"]
    raw = ggml.quantize(ggml.TYPE_IDS[case["type"]], torch.randn(n, k, generator=g, device=DEVICE) * 0.02)
    x = torch.randn(rows, k, generator=g, device=DEVICE)
    bias = torch.randn(n, generator=g, device=DEVICE) * 0.1 if case.get("bias") else None
    grad = torch.randn(rows, n, generator=g, device=DEVICE) * 1e-3 if case["kind"] == "tune" else None
    return raw, x, bias, grad


def _mlp(case, i, limit):
    ff = WIDTHS[case["width"]]["ff"]
    if case["experts"] and i % 4 >= 2:
        return dict(kind="moe", router=dict(experts=EXPERTS["experts"], top=EXPERTS["top"]),
                    expert=dict(ff=EXPERTS["ff"], limit=7.0), shared=dict(ff=EXPERTS["ff"], limit=7.0))
    return dict(kind="dense", ff=ff, **limit)


def _lenisun_cfg(case):
    E, w = case["width"], WIDTHS[case["width"]]
    layers = []
    for i in range(case["layers"]):
        mixer = (dict(heads=E // 64, dim=64) if i % 2 else
                 dict(heads=w["heads"], kv_heads=w["kv_heads"], dim=w["dim"], vdim=w["dim"], scale=w["dim"] ** -0.5, v_mix=True,
                      q_temp=dict(coef=0.1, every=512)))
        layers.append(dict(type="wkv" if i % 2 else "attention", mixer=mixer, mlp=_mlp(case, i, dict(limit=7.0))))
    return dict(architecture="Lenisun", vocab=case["vocab"], width=E, norm=dict(eps=1e-6), embedding=dict(scale=1.0), layers=layers)


def _vepinex_cfg(case):
    E, wide = case["width"], WIDTHS[case["width"]]["wide"]
    layers, own = [], None
    for i in range(case["layers"]):
        if i % 3 == 0:
            kind, mixer = "channel_delta", dict(heads=E // wide, kv_heads=E // wide, dim=wide, vdim=wide, conv=4)
        elif i % 3 == 1:
            kind, mixer = "mlstm", dict(heads=E // 128, dim=64, vdim=128, gate_cap=10.0)
        else:
            kind, r = "latent_attention", wide // 2
            mixer = dict(heads=E // wide, dim=wide, rot_dim=r, vdim=wide, kv_rank=4 * wide, scale=(wide + r) ** -0.5,
                         rot=dict(base=1e4, dims=r))
            if i % 6 == 5:
                mixer["kv_from"] = own
            else:
                own = i
        layers.append(dict(type=kind, mixer=mixer, mlp=_mlp(case, i, {})))
    return dict(architecture="Vepinex", vocab=case["vocab"], width=E, norm=dict(eps=1e-6), layers=layers)


def _host(case, seed):
    """The model of a case as a loader hands it over."""
    if case["kind"] == "gpt2":
        cfg = dict(hostmodel.GPT2_SMALL, layer=case["layers"])
        host = hostmodel.Gpt2Host.synthetic(cfg, qtype=ggml.TYPE_IDS[case["type"]], seed=seed, device=DEVICE)
        return host.randomize_small_params(seed=seed)
    if case["kind"] in ("gemma3", "gemma3_batch"):
        cfg = dict(hostmodel.GEMMA3_1B, layer=case["layers"])
        host = hostmodel.Gemma3Host.synthetic(cfg, qtype=ggml.TYPE_IDS[case["type"]], seed=seed, device=DEVICE)
        return host.randomize_small_params(seed=seed)
    if case["design"] == "lenisun":
        return hostmodel.LenisunHost.synthetic(_lenisun_cfg(case), seed=seed, device=DEVICE, decay_rank=RANK)
    return hostmodel.VepinexHost.synthetic(_vepinex_cfg(case), seed=seed, device=DEVICE, a_rank=RANK, g_rank=RANK)


def _vocab(case):
    return {"gpt2": hostmodel.GPT2_SMALL["vocab"], "decoder": case.get("vocab")}.get(case["kind"], hostmodel.GEMMA3_1B["vocab"])


def _tokens(case, seed):
    """(prompts, the tokens that the program feeds per step): prompts of requests served together differ in length."""
    rng = np.random.default_rng(seed)
    sequences = case.get("sequences", 1)
    longest = case["prompt"]
    lengths = [longest if s == 0 else int(rng.integers(max(1, longest // 2), longest + 1)) for s in range(sequences)]
    prompts = [rng.integers(0, _vocab(case), size=t) for t in lengths]
    return prompts, rng.integers(0, _vocab(case), size=(case["tokens"], sequences))


def prepare(case, seed):
    state = dict(case=case)
    if case["kind"] in ("linear", "tune"):
        raw, state["x"], state["bias"], state["grad"] = _linear_inputs(case, seed)
        state["weight"] = api.QuantWeight(raw, ggml.TYPE_IDS[case["type"]], case["n"], case["k"])
        if case["kind"] == "tune":
            state["x"].requires_grad_(True)
        return state
    host = _host(case, seed)
    state["prompts"], state["steps"] = _tokens(case, seed)
    if case["kind"] == "gpt2":
        state["engine"] = api.Gpt2(host)
    elif case["kind"] == "gemma3":
        state["engine"] = api.Gemma3(host)
    elif case["kind"] == "gemma3_batch":
        state["engine"] = api.Gemma3Batch(host, case["sequences"])
    else:
        engine = api.Lenisun if case["design"] == "lenisun" else api.Vepinex
        state["engine"] = engine(host, ctx=2048, n_seq=case["sequences"])
    return state


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    return {"linear": _run_linear, "tune": _run_tune, "gpt2": _run_greedy, "gemma3": _run_greedy, "gemma3_batch": _run_batch,
            "decoder": _run_decoder}[case["kind"]](case, state)


def _run_linear(case, s):
    mode = api.ACT_F32 if case["act"] == "f32" else api.ACT_Q8
    return api.quant_matmul_no_grad(s["x"], s["weight"], mode, bias=s["bias"])


def _run_tune(case, s):
    y = api.quant_matmul_no_grad(s["x"], s["weight"])
    grad_x, = torch.autograd.grad(y, s["x"], s["grad"])
    return y.detach(), grad_x


def _run_greedy(case, s):
    engine = s["engine"]
    first = engine.prefill(s["prompts"][0])
    tokens = engine.decode_greedy(int(api.argmax(first).item()), case["tokens"])
    return dict(first=first, tokens=tokens.astype(np.int64), last=engine.decode_next(int(tokens[-1])))


def _run_batch(case, s):
    engine = s["engine"]
    engine.reset_cache()
    logits = [torch.stack([engine.prefill(i, p) for i, p in enumerate(s["prompts"])])]
    for step in s["steps"]:
        logits.append(engine.decode_next(step))
    return torch.stack(logits)


def _run_decoder(case, s):
    engine = s["engine"]
    if case["sequences"] == 1:
        logits = [engine.prefill(s["prompts"][0])]
        for step in s["steps"]:
            logits.append(engine.decode_next(int(step[0])))
        return torch.stack(logits)[:, None]
    slots = list(range(case["sequences"]))
    engine.reset_cache()
    logits = [torch.cat([engine.extend(p, [len(p) - 1], seq=i) for i, p in enumerate(s["prompts"])])]
    for step in s["steps"]:
        logits.append(engine.decode_next_batch(slots, step))
    return torch.stack(logits)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _model_sizes(case):
    """(bytes of the weights that a token needs, multiply-adds per prompt token, multiply-adds and bytes of the head, bytes of
    keys and values per context token, score and value multiply-adds per pair of tokens, most tokens a window sees)."""
    if case["kind"] == "gpt2":
        c = hostmodel.GPT2_SMALL
        E, params = c["embed"], case["layers"] * (4 * c["embed"] ** 2 + 2 * c["embed"] * c["ffn"])
        return params // 32 * BLOCK_BYTES[case["type"]], params, c["vocab"] * E, 4 * c["vocab"] * E, case["layers"] * 8 * E, case["layers"] * 2 * E
    if case["kind"] != "decoder":
        c = hostmodel.GEMMA3_1B
        E, q, kv = c["embed"], c["head"] * c["head_dim"], c["head_kv"] * c["head_dim"]
        params = case["layers"] * ((q + 2 * kv) * E + E * q + 3 * E * c["ffn"])
        per = BLOCK_BYTES[case["type"]]
        return (params // 32 * per, params, c["vocab"] * E, c["vocab"] * E // 32 * per, case["layers"] * 8 * kv, case["layers"] * 2 * q)
    cfg = _lenisun_cfg(case) if case["design"] == "lenisun" else _vepinex_cfg(case)
    E, params, cache, pair = case["width"], 0, 0, 0
    for layer in cfg["layers"]:
        m, f, H = layer["mixer"], layer["mlp"], layer["mixer"]["heads"]
        d, e = m["dim"], m.get("vdim", m["dim"])
        if layer["type"] == "attention":
            params += E * (H * d + m["kv_heads"] * (d + e) + H * e)
            cache, pair = cache + 2 * m["kv_heads"] * (d + e), pair + H * (d + e)
        elif layer["type"] == "latent_attention":
            own, R = m.get("kv_from") is None, m["kv_rank"]
            params += E * (H * (d + m["rot_dim"]) + own * (R + m["rot_dim"]) + H * e) + R * H * (d + e)
            cache, pair = cache + 2 * own * (R + m["rot_dim"]), pair + H * (d + m["rot_dim"] + e)
        else:
            params += E * {"wkv": 5 * H * d, "mlstm": H * (2 * d + 3 * e), "channel_delta": H * (2 * d + 2 * e)}[layer["type"]]
            params += 0 if layer["type"] == "mlstm" else RANK * (2 * E + H * (d + e))
        units = E * f["ff"] if f["kind"] == "dense" else E * (EXPERTS["top"] + 1) * EXPERTS["ff"]
        params += 3 * units
    return 2 * params, params, E * case["vocab"], 2 * E * case["vocab"], cache, pair


def work(case):
    if case["kind"] in ("linear", "tune"):
        k, n, rows = case["k"], case["n"], case["rows"]
        weight, passes = n * (k // 32) * BLOCK_BYTES[case["type"]], 2 if case["kind"] == "tune" else 1
        extra = 4 * n if case.get("bias") else 0
        return dict(bytes=passes * (weight + 4 * rows * (k + n)) + extra, flops=passes * 2 * rows * n * k)
    weights, params, head, head_bytes, cache, pair = _model_sizes(case)
    sequences, steps = case.get("sequences", 1), case["tokens"] + (case["kind"] in ("gpt2", "gemma3"))
    P = case["prompt"]  # requests served together are three quarters of it on average, but for the first
    mean = P if sequences == 1 else (P + 0.75 * P * (sequences - 1)) / sequences
    logits = 4 * _vocab(case) * sequences
    nbytes = sequences * (weights + head_bytes + cache * mean) + logits
    nbytes += steps * (weights + head_bytes + sequences * cache * (mean + steps / 2) + logits)
    flops = 2 * sequences * (mean * params + head + pair * mean * mean / 2) + 2 * steps * sequences * (params + head + pair * mean)
    return dict(bytes=int(nbytes), flops=int(flops))


# ---- how far correct implementations lie apart ---------------------------------------------------------------------
def tolerance(case):
    if case["kind"] == "linear" and case["act"] == "q8":
        return "exact"  # whole-number block dots whose scaled sums have one order: the bits are part of the interface
    if case["kind"] in ("gemma3", "gemma3_batch"):
        return "exact"  # the same, through every layer: 8-bit rounding would multiply any difference
    if case["kind"] == "linear":
        # up to 16 rows (and more, on small matrices) in 32 bits; many rows round weights and activations to 11 bits once
        return dict(rel=1e-5, max=1e-4) if case["rows"] <= 16 else dict(rel=1.2e-3, max=1.2e-2)
    if case["kind"] == "tune":
        return dict(rel=1.2e-3, max=1.2e-2)
    if case["kind"] == "gpt2":
        return dict(rel=1e-5, max=1e-4)
    return dict(rel=3e-2, max=0.3)  # bf16 operands through every layer


# ---- the same in 64 bits -------------------------------------------------------------------------------------------
def _dequantised(raw, kind, n, k):
    """f64 values of GGUF blocks."""
    raw = torch.as_tensor(raw, device=DEVICE).reshape(-1, BLOCK_BYTES[kind])
    half = lambda i: raw[:, i:i + 2].contiguous().view(torch.float16).double()
    if kind == "q8_0":
        return (raw[:, 2:].contiguous().view(torch.int8).double() * half(0)).reshape(n, k)
    packed = raw[:, 2:] if kind == "q4_0" else raw[:, 4:]
    q = torch.cat([packed & 15, packed >> 4], dim=1).double()
    return ((q - 8) * half(0) if kind == "q4_0" else q * half(0) + half(2)).reshape(n, k)


def _rounded_to_q8(x):
    """The values that 8-bit activations stand for: blocks of 32, scale = largest / 127, halves away from zero."""
    b = x.reshape(-1, 32)
    scale = b.abs().amax(dim=1, keepdim=True) / 127.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    r = b / scale
    q = torch.trunc(r.double() + torch.sign(r).double() * 0.5).clamp(-127, 127)
    return (q * scale.double()).reshape(x.shape)


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] in ("linear", "tune"):
            raw, x, bias, grad = _linear_inputs(case, seed)
            w = _dequantised(raw, case["type"], case["n"], case["k"])
            if case["kind"] == "tune":
                return x.double() @ w.T, grad.double() @ w
            x = x.double() if case["act"] == "f32" else _rounded_to_q8(x)
            return x @ w.T + (bias.double() if bias is not None else 0)
        if case["kind"] == "gpt2":
            return _exact_gpt2(case, seed)
        if case["kind"] == "decoder":
            return _exact_decoder(case, seed)
    return None  # Gemma-3's activations are rounded to 8 bits in every layer: its result is a string of bits, not a limit


def _norm(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _causal(q, k, v, scale):
    """q [H, T, d], k [H, T, d], v [H, T, e] -> [T, H * e]."""
    s = q @ k.transpose(1, 2) * scale
    s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=DEVICE).triu(1), -math.inf)
    return (torch.softmax(s, dim=-1) @ v).transpose(0, 1).reshape(q.shape[1], -1)


def _exact_gpt2(case, seed):
    host = _host(case, seed)
    f64 = lambda a: torch.as_tensor(a, device=DEVICE).double()
    wte, wpe = f64(host.wte), f64(host.wpe)
    blocks = [{n: (_dequantised(v.raw, case["type"], v.out_dim, v.in_dim) if hasattr(v, "raw") else f64(v)) for n, v in b.items()}
              for b in host.blocks]
    E, H = wte.shape[1], host.cfg["head"]

    def layer_norm(x, w, b):
        x = x - x.mean(dim=-1, keepdim=True)
        return _norm(x, 1e-5) * w + b

    def logits(tokens):
        x = wte[torch.as_tensor(tokens, device=DEVICE)] + wpe[:len(tokens)]
        for b in blocks:
            h = layer_norm(x, b["ln1_weight"], b["ln1_bias"]) @ b["attn_qkv_weight"].T + b["attn_qkv_bias"]
            q, k, v = (h[:, i * E:(i + 1) * E].reshape(-1, H, E // H).transpose(0, 1) for i in range(3))
            x = x + _causal(q, k, v, (E // H) ** -0.5) @ b["attn_proj_weight"].T + b["attn_proj_bias"]
            h = layer_norm(x, b["ln2_weight"], b["ln2_bias"]) @ b["mlp_fc_weight"].T + b["mlp_fc_bias"]
            x = x + torch.nn.functional.gelu(h, approximate="tanh") @ b["mlp_proj_weight"].T + b["mlp_proj_bias"]
        return wte @ layer_norm(x[-1], f64(host.ln_f_weight), f64(host.ln_f_bias))

    tokens = [int(t) for t in _tokens(case, seed)[0][0]]
    first = logits(tokens)
    step, found = first, []
    for _ in range(case["tokens"]):
        tokens.append(int(step.argmax()))
        step = logits(tokens)
        found.append(int(step.argmax()))
    return dict(first=first, tokens=np.array(found), last=logits(tokens + found[-1:]))


def _exact_decoder(case, seed):
    host = _host(case, seed)
    weights = {n: torch.as_tensor(a, device=DEVICE).double() for n, a in host.as_f32().items()}
    prompts, steps = _tokens(case, seed)
    out = []
    for s, prompt in enumerate(prompts):
        tokens = torch.as_tensor(np.concatenate([prompt, steps[:, s]]), device=DEVICE)
        x = (_lenisun if case["design"] == "lenisun" else _vepinex)(host.cfg, weights, tokens)
        head = weights["head" if case["design"] == "lenisun" else "embed"]
        out.append(x[len(prompt) - 1:] @ head.T)
    return torch.stack(out, dim=1)


def _under(weights, prefix):
    return {n[len(prefix):]: w for n, w in weights.items() if n.startswith(prefix)}


def _clamped(g, u, limit):
    g = g.clamp(max=limit)
    return g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1)


def _lenisun(cfg, weights, tokens):
    eps, first = cfg["norm"]["eps"], None
    silu = torch.nn.functional.silu
    x = weights["embed"][tokens] * cfg["embedding"]["scale"]
    T = len(tokens)
    for i, layer in enumerate(cfg["layers"]):
        L, m, f = _under(weights, "l%d." % i), layer["mixer"], layer["mlp"]
        W, F = _under(L, "mix."), _under(L, "mlp.")
        h = _norm(x, eps) * (1 + L["norm1"])
        if layer["type"] == "attention":
            H, G = m["heads"], m["kv_heads"]
            q, k, v = ((h @ W[n].T).reshape(T, heads, -1).transpose(0, 1) for n, heads in (("q", H), ("k", G), ("v", G)))
            at = torch.arange(T, device=DEVICE, dtype=torch.float64)
            q = _norm(q, eps) * W["q.norm"] * (1 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1))[:, None]
            k = _norm(k, eps) * W["k.norm"]
            if first is None:
                first = v
            else:
                v = (1 - W["vmix"]) * v + W["vmix"] * first
            k, v = (t.repeat_interleave(H // G, dim=0) for t in (k, v))
            y = _causal(q, k, v, m["scale"]) @ W["o"].T
        else:
            H, d = m["heads"], m["dim"]
            back = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
            mix = {n: h + (back - h) * W["mu." + n] for n in "rkvgw"}
            r, k, v = ((mix[n] @ W[n].T).reshape(T, H, d) for n in "rkv")
            keep = torch.exp(-torch.exp(torch.tanh(mix["w"] @ W["w1"].T) @ W["w2"].T + W["w0"])).reshape(T, H, d, 1)
            kv = k[..., None] * v[:, :, None, :]
            S, o = torch.zeros(H, d, d, dtype=torch.float64, device=DEVICE), []
            for t in range(T):
                o.append((r[t][:, None, :] @ (S + W["u"][:, :, None] * kv[t]))[:, 0])
                S = keep[t] * S + kv[t]
            y = (_norm(torch.stack(o), eps).reshape(T, H * d) * W["norm"] * silu(mix["g"] @ W["g"].T)) @ W["o"].T
        x = x + _norm(y, eps) * (1 + L["norm1b"])
        h = _norm(x, eps) * (1 + L["norm2"])
        if f["kind"] == "dense":
            y = _clamped(h @ F["gate"].T, h @ F["up"].T, f["limit"]) @ F["down"].T
        else:
            scores, ids = torch.sigmoid(h @ F["router"].T).topk(f["router"]["top"], dim=1)
            y = (silu(h @ F["shared.gate"].T) * (h @ F["shared.up"].T)) @ F["shared.down"].T * torch.sigmoid(h @ F["shared.sg"].T)
            for e in range(f["router"]["experts"]):
                t, place = torch.nonzero(ids == e, as_tuple=True)
                z, p = h[t] * scores[t, place, None], "e%d." % e
                y[t] += (silu(z @ F[p + "gate"].T) * (z @ F[p + "up"].T)) @ F[p + "down"].T
        x = x + _norm(y, eps) * (1 + L["norm2b"])
    return _norm(x, eps) * (1 + weights["final.norm"])


def _rotated(x, base):
    """x [..., T, r]: neighbours turned by position * base^(-2i / r)."""
    r = x.shape[-1]
    freq = base ** (-torch.arange(0, r, 2, device=DEVICE, dtype=torch.float64) / r)
    a = torch.arange(x.shape[-2], device=DEVICE, dtype=torch.float64)[:, None] * freq
    return torch.view_as_real(torch.view_as_complex(x.reshape(*x.shape[:-1], -1, 2).contiguous()) * torch.polar(torch.ones_like(a), a)).flatten(-2)


def _memory(h, W, m, eps):
    T, H, d, e, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = ((h @ W[n].T).reshape(T, H, -1) for n in "qkv")
    capped = lambda n: cap * torch.tanh((h @ W[n].T + W[n + ".b"]) / cap)
    gate_in, forget = capped("i"), torch.nn.functional.logsigmoid(capped("f"))
    new = torch.zeros(H, dtype=torch.float64, device=DEVICE)
    S, n, o = new.new_zeros(H, d, e), new.new_zeros(H, d), []
    for t in range(T):
        old, new = new, torch.maximum(forget[t] + new, gate_in[t])
        keep, add = torch.exp(forget[t] + old - new)[:, None], torch.exp(gate_in[t] - new)[:, None]
        n = keep * n + add * k[t]
        S = keep[..., None] * S + (add * k[t])[..., None] * v[t][:, None, :]
        qt = q[t] * d ** -0.5
        size = torch.maximum((n * qt).sum(dim=1).abs(), torch.exp(-new)) + 1e-6
        o.append((qt[:, None, :] @ S)[:, 0] / size[:, None])
    return (_norm(torch.stack(o), eps).reshape(T, H * e) * W["norm"] * torch.sigmoid(h @ W["g"].T)) @ W["o"].T


def _delta(h, W, m, eps):
    T, H, G, d, e, taps = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]

    def conv(n):
        z = torch.nn.functional.pad(h @ W[n].T, (0, 0, taps - 1, 0))
        return torch.nn.functional.silu(sum(z[j:j + T] * W[n + ".conv"][:, j] for j in range(taps)))
    q, k = (conv(n).reshape(T, G, d).repeat_interleave(H // G, dim=1) for n in "qk")
    q, k = (t / torch.sqrt((t * t).sum(dim=-1, keepdim=True) + 1e-6) for t in (q, k))
    v, beta = conv("v").reshape(T, H, e), torch.sigmoid(h @ W["b"].T)[..., None]
    rate = torch.nn.functional.softplus(((h @ W["a1"].T) @ W["a2"].T).reshape(T, H, d) + W["dt_bias"].reshape(H, d))
    keep = torch.exp(-torch.exp(W["A_log"])[:, None] * rate)[..., None]
    S, o = torch.zeros(H, d, e, dtype=torch.float64, device=DEVICE), []
    for t in range(T):
        S = keep[t] * S
        S = S + k[t][..., None] * (beta[t] * (v[t] - (k[t][:, None, :] @ S)[:, 0]))[:, None, :]
        o.append((q[t][:, None, :] @ S)[:, 0] * d ** -0.5)
    gate = torch.sigmoid((h @ W["g1"].T) @ W["g2"].T)
    return ((_norm(torch.stack(o), eps) * W["norm"]).reshape(T, H * e) * gate) @ W["o"].T


def _vepinex(cfg, weights, tokens):
    eps, kept, T = cfg["norm"]["eps"], {}, len(tokens)
    x = _norm(weights["embed"][tokens], eps) * weights["embed.norm"]
    for i, layer in enumerate(cfg["layers"]):
        L, m, f = _under(weights, "l%d." % i), layer["mixer"], layer["mlp"]
        W, F = _under(L, "mix."), _under(L, "mlp.")
        h = _norm(x, eps) * L["norm1"]
        if layer["type"] == "mlstm":
            y = _memory(h, W, m, eps)
        elif layer["type"] == "channel_delta":
            y = _delta(h, W, m, eps)
        else:
            H, d, R, base = m["heads"], m["dim"], m["kv_rank"], m["rot"]["base"]
            if m.get("kv_from") is None:
                z = h @ W["dkv"].T
                kept[i] = _norm(z[:, :R], eps) * W["dkv.norm"], _rotated(z[:, R:], base)
            c, kr = kept[i if m.get("kv_from") is None else m["kv_from"]]
            q = (h @ W["q"].T).reshape(T, H, -1).transpose(0, 1)
            q = torch.cat([q[..., :d], _rotated(q[..., d:], base)], dim=-1)
            k, v = ((c @ W[n].T).reshape(T, H, -1).transpose(0, 1) for n in ("uk", "uv"))
            y = _causal(q, torch.cat([k, kr.expand(H, -1, -1)], dim=-1), v, m["scale"]) @ W["o"].T
        if f["kind"] == "dense":
            y = y + (torch.nn.functional.silu(h @ F["gate"].T) * (h @ F["up"].T)) @ F["down"].T
        else:
            z, ids = (h @ F["router"].T + F["router.b"]).topk(f["router"]["top"], dim=1)
            z = torch.softmax(z, dim=1)
            unit = lambda a, p, limit: _clamped(a @ F[p + "gate"].T, a @ F[p + "up"].T, limit) @ F[p + "down"].T
            y = y + unit(h, "shared.", f["shared"]["limit"])
            for e in range(f["router"]["experts"]):
                t, place = torch.nonzero(ids == e, as_tuple=True)
                y[t] += z[t, place, None] * unit(h[t], "e%d." % e, f["expert"]["limit"])
        x = x + y
    return _norm(x, eps) * weights["final.norm"]
