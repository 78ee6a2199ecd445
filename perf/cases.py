"""The work that users of this framework have it do, as cases that can be timed and compared.

Two families run here.  The integer model: DeepSeek-V3 layers in int64 fixed point, at the widths of the full model and at
the two magnitudes of the benchmark: small (activations near 2^16, weights near 2^16 / sqrt(fan-in), shifts 16, the gate's
9; three limbs hold an activation) and the reference's own (2^21, 2^30 / sqrt(fan-in), shifts 29 and 30; four limbs).  Its
outputs are compared word for word.  And the floating-point decoder designs Munalorn and Vifelix, two layers at the sizes
of the benchmark, in bfloat16 (how they are served) and float32.

A state is what a serving program holds: a loaded model with its weights laid out, and its tokens.  Integer models have run
once on a few tokens before, as they have in a program that serves.
"""
import importlib
import math
import zlib

import numpy as np
import torch

PACKAGE = "zk-deepseek_b200"
DEVICE = "cuda"

# width, heads, q_rank, kv_rank, feed-forward of Munalorn's layers; heads of 128 + 64 rotated, values of 128
MUNALORN = {"w7168": (7168, 128, 1536, 512, 18432), "w4096": (4096, 32, 1024, 512, 14336), "w2048": (2048, 16, 768, 512, 8192)}
# width, attention heads, key heads, retention heads, Mamba-2 heads, feed-forward of Vifelix's layers
VIFELIX = {"w7168": (7168, 128, 16, 28, 224, 18432), "w4096": (4096, 32, 8, 16, 128, 14336), "w2048": (2048, 16, 4, 8, 64, 8192)}


def listed():
    return [
        # the reference's own call for one projection, operands unprepared: wkv_a of 32 tokens
        {"name": "projection_32", "kind": "projection", "rows": 32, "inner": 7168, "outer": 576, "weight_bits": 64},
        # the element-wise and row kernels by themselves, on one attention block's activations
        {"name": "fixedpoint_2048", "kind": "fixedpoint", "tokens": 2048},
        # the attention layer on a long prompt: what prefill costs
        {"name": "attention_4096", "kind": "attention", "tokens": 4096, "scales": "small"},
        # a whole dense block on a prompt of odd length, at the reference's own magnitudes
        {"name": "block_777", "kind": "block", "tokens": 777, "scales": "reference"},
        # the routed layer as one GPU of eight holds it, an odd number of tokens
        {"name": "experts_1001", "kind": "experts", "tokens": 1001, "experts": 32},
        # batched decoding: a dense and a routed block, final norm and head
        {"name": "decode_64", "kind": "decode", "batch": 64, "cache": 2048, "experts": 64, "vocab": 16160},
        # one sequence decoding, the reference's own use: latency
        {"name": "decode_1", "kind": "decode", "batch": 1, "cache": 500, "experts": 32, "vocab": 16160},
        # prompts and decoding of the floating-point designs
        {"name": "munalorn_prompt_4096", "kind": "munalorn_prompt", "size": "w7168", "tokens": 4096, "window": 4096, "dtype": "bfloat16"},
        {"name": "munalorn_prompt_f32", "kind": "munalorn_prompt", "size": "w2048", "tokens": 300, "window": 4096, "dtype": "float32"},
        {"name": "munalorn_decode_1", "kind": "munalorn_decode", "size": "w4096", "batch": 1, "cache": 4095, "dtype": "bfloat16"},
        {"name": "vifelix_prompt_3001", "kind": "vifelix_prompt", "size": "w4096", "tokens": 3001, "window": 1024, "dtype": "bfloat16"},
        # a small batch from its prompts through its first tokens
        {"name": "vifelix_request_4", "kind": "vifelix_request", "size": "w2048", "batch": 4, "prompt": 150, "new": 16, "dtype": "bfloat16"},
    ]


def _between(rng, low, high):
    """a whole number spread over the logarithm of the range, often odd"""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return max(low, min(high, n | rng.randrange(2)))


def draw(rng):
    kind = rng.choice(["projection", "fixedpoint", "attention", "block", "experts", "decode", "munalorn_prompt",
                       "munalorn_decode", "vifelix_prompt", "vifelix_request"])
    dtype = "float32" if rng.random() < 0.2 else "bfloat16"
    case = {"kind": kind}
    if kind == "projection":
        case.update(rows=_between(rng, 1, 512), inner=rng.choice([512, 1536, 2048, 7168, 7000]), outer=_between(rng, 64, 2112),
                    weight_bits=rng.choice([32, 64]))
    elif kind == "fixedpoint":
        case.update(tokens=_between(rng, 32, 2047))
    elif kind == "attention":
        case.update(tokens=_between(rng, 17, 2500), scales=rng.choice(["small", "reference"]))
    elif kind == "block":
        case.update(tokens=_between(rng, 17, 2048), scales=rng.choice(["small", "reference"]))
    elif kind == "experts":
        case.update(tokens=_between(rng, 9, 2048), experts=rng.choice([16, 32]))
    elif kind == "decode":
        case.update(batch=_between(rng, 1, 64), cache=_between(rng, 100, 2048), experts=rng.choice([16, 32, 64]), vocab=16160)
    elif kind == "munalorn_prompt":
        case.update(size=rng.choice(sorted(MUNALORN)) if dtype == "bfloat16" else "w2048",
                    tokens=_between(rng, 17, 4096 if dtype == "bfloat16" else 700), window=rng.choice([4096, 1024, 300]), dtype=dtype)
    elif kind == "munalorn_decode":
        case.update(size=rng.choice(sorted(MUNALORN)) if dtype == "bfloat16" else "w2048", batch=_between(rng, 1, 4),
                    cache=_between(rng, 20, 4095 if dtype == "bfloat16" else 700), dtype=dtype)
    elif kind == "vifelix_prompt":
        case.update(size=rng.choice(sorted(VIFELIX)) if dtype == "bfloat16" else "w2048",
                    tokens=_between(rng, 17, 4096 if dtype == "bfloat16" else 700), window=rng.choice([4096, 1024, 300]), dtype=dtype)
    else:
        case.update(size=rng.choice(["w2048", "w4096"]) if dtype == "bfloat16" else "w2048", batch=_between(rng, 1, 4),
                    prompt=_between(rng, 17, 400), new=_between(rng, 4, 32), dtype=dtype)
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------------
def _module(name):
    return importlib.import_module(PACKAGE + "." + name)


def _generator(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((zlib.crc32(name.encode()) << 24) ^ seed)


def _whole(seed, name, shape, scale, dtype=torch.int64):
    """round(N(0, 1) * scale)"""
    g, out = _generator(seed, name), torch.empty(shape, dtype=dtype, device=DEVICE)
    flat, step = out.view(-1), 1 << 27
    for i in range(0, flat.numel(), step):
        part = flat[i:i + step]
        part.copy_(torch.randn(part.numel(), generator=g, device=DEVICE).mul_(scale).round_())
    return out


def _weight(seed, name, outer, inner, dtype=torch.int32, bits=16):
    return _whole(seed, name, (outer, inner), 2.0 ** bits / math.sqrt(inner), dtype)


def _norm_weight(seed, name, n, dtype=torch.int32, bits=16):
    return (2 ** bits + _whole(seed, name, (n,), 2.0 ** (bits - 8))).to(dtype)


# magnitudes: bits of activations, of weights at fan-in 1, of the norms inside attention; shift; limbs of an activation
_SCALES = {"small": (16, 16, 16, 16, 3), "reference": (21, 30, 19, 30, 4)}


def _integer_modules(scales="small"):
    """kernel and model module, set up as a serving program sets them up: with the limbs promised that activations fit"""
    k, m = _module("kernel"), _module("model")
    m.world_size, m.rank, m.ACT_LIMBS = 1, 0, _SCALES[scales][4]
    k.SOFTMAX_WRITES_WEIGHTS = False
    k.softmax_init_q19()
    k.silu_init_q23()
    return k, m


def _integer_args(m, positions, layers=1, dense=1, experts=32, vocab=1024):
    return m.ModelArgs(max_seq_len=positions, vocab_size=vocab, dim=7168, inter_dim=18432, moe_inter_dim=2048, n_layers=layers,
                       n_dense_layers=dense, n_heads=128, n_routed_experts=experts, n_shared_experts=1, n_activated_experts=8,
                       n_expert_groups=8, n_limited_groups=4, score_func="sigmoid", route_scale=2.5, q_lora_rank=1536,
                       kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128)


def _shift(n):
    return torch.tensor(n, dtype=torch.int32, device=DEVICE)


def _fill_attention(at, seed, a, p, scales="small"):
    H, (_, bits, norm, shift, limbs) = a.n_heads, _SCALES[scales]
    for name, outer, inner in (("wq_a", a.q_lora_rank, a.dim), ("wkv_a1", a.kv_lora_rank, a.dim), ("wkv_a2", a.qk_rope_head_dim, a.dim),
                               ("wq_b1", H * a.qk_nope_head_dim, a.q_lora_rank), ("wq_b2", H * a.qk_rope_head_dim, a.q_lora_rank)):
        lin = getattr(at, name)
        lin.weight = _weight(seed, p + name, outer, inner, bits=bits)
        if scales == "small":                # otherwise the shifts that the reference fixes
            lin.res_rescale = shift
    for name, outer, inner in (("wkv_b_1", H * a.qk_nope_head_dim, a.kv_lora_rank), ("wkv_b_2", H * a.v_head_dim, a.kv_lora_rank),
                               ("wo", a.dim, H * a.v_head_dim)):
        lin = getattr(at, name)
        lin.weight, lin.scale = _weight(seed, p + name, outer, inner, bits=bits), _shift(shift)
    at.q_norm.weight = _norm_weight(seed, p + "q_norm", a.q_lora_rank, bits=norm)
    at.kv_norm.weight = _norm_weight(seed, p + "kv_norm", a.kv_lora_rank, bits=norm)
    at.score_limbs = (limbs, limbs)


def _fill_mlp(mlp, seed, dim, inter, p, scales="small"):
    for name, outer, inner in (("w1", inter, dim), ("w3", inter, dim), ("w2", dim, inter)):
        lin = getattr(mlp, name)
        lin.weight, lin.scale = _weight(seed, p + name, outer, inner, bits=_SCALES[scales][1]), _shift(_SCALES[scales][3])


def _fill_experts(moe, seed, a, p):
    E, D, I = a.n_routed_experts, a.dim, a.moe_inter_dim
    moe.gate.weight, moe.gate.scale = _weight(seed, p + "gate", E, D), _shift(9)
    moe.gate.bias = _whole(seed, p + "bias", (E,), 2.0 ** 15).abs_().to(torch.int32)
    _fill_mlp(moe.shared_experts, seed, D, I, p + "shared.")
    moe.experts_w13 = _whole(seed, p + "w13", (E, 2 * I, D), 2.0 ** 16 / math.sqrt(D), torch.int32)
    moe.experts_w2 = _whole(seed, p + "w2", (E, D, I), 2.0 ** 16 / math.sqrt(I), torch.int32)
    moe.experts_shift.fill_(16)


def _fill_block(blk, seed, a, p, scales="small"):
    blk.attn_norm.weight = _norm_weight(seed, p + "attn_norm", a.dim, bits=_SCALES[scales][0])
    blk.ffn_norm.weight = _norm_weight(seed, p + "ffn_norm", a.dim, bits=_SCALES[scales][0])
    _fill_attention(blk.attn, seed, a, p, scales)
    if hasattr(blk.ffn, "gate"):
        _fill_experts(blk.ffn, seed, a, p)
    else:
        _fill_mlp(blk.ffn, seed, a.dim, a.inter_dim, p, scales)


def _causal(n):
    mask = torch.full((n, n), -(64 << 36), dtype=torch.int64, device=DEVICE).triu_(1)
    mask._zkds_causal = True          # as Transformer.layer_inference marks the mask that it builds
    return mask


def _rotation_table(tokens):
    """cos and sin at 2^42, base 10000, 64 rotated dimensions"""
    ang = np.outer(np.arange(tokens), 10000.0 ** (-np.arange(0, 64, 2) / 64.0))
    tab = np.rint(np.stack([np.cos(ang), np.sin(ang)], -1) * 2.0 ** 42).astype(np.int64)
    return torch.from_numpy(tab).to(DEVICE).view(1, tokens, 1, 32, 2)


def _prepare_projection(case, seed):
    k, _ = _integer_modules()
    g = _generator(seed, "projection")
    x = torch.randint(-2 ** 20, 2 ** 20, (1, case["rows"], case["inner"]), generator=g, device=DEVICE)
    w = torch.randint(-2 ** 15, 2 ** 15, (case["outer"], case["inner"]), generator=g, device=DEVICE)
    return {"k": k, "x": x, "w": w if case["weight_bits"] == 64 else w.to(torch.int32)}


def _run_projection(s):
    return s["k"].int64_bmm_broadcast(s["x"], s["w"], 1, 1, 16)


def _prepare_fixedpoint(case, seed):
    k, _ = _integer_modules()
    T = case["tokens"]
    scores = _whole(seed, "scores", (1, T, 128, T), 2.0 ** 18)
    scores += _causal(T)[:, None, :]
    s = {"k": k, "x": _whole(seed, "x", (T, 7168), 2.0 ** 16), "w": _norm_weight(seed, "w", 7168), "scores": scores,
         "q": _whole(seed, "q", (1, T, 128, 32, 2), 2.0 ** 16), "table": _rotation_table(T),
         "act": _whole(seed, "act", (1, T, 18432), 2.0 ** 16)}
    s["probs"], s["silu"] = torch.empty_like(scores), torch.empty_like(s["act"])
    return s


def _run_fixedpoint(s):
    k = s["k"]
    normed, rms = k.rms_norm_int64_device(s["x"], s["w"], 1, 7168)
    turned = k.complex_int64_mul_broadcast(s["q"], s["table"])
    k.softmax_q19(s["scores"], s["probs"])
    k.silu_q23(s["act"], s["silu"])
    return [normed, rms, turned, s["probs"], s["silu"]]


def _prepare_attention(case, seed):
    _, m = _integer_modules(case["scales"])
    T = case["tokens"]
    a = _integer_args(m, T)
    with torch.device(DEVICE):
        at = m.MLA(0, a)
    _fill_attention(at, seed, a, "l0.", case["scales"])
    s = {"layer": at, "x": _whole(seed, "x", (1, T, a.dim), 2.0 ** _SCALES[case["scales"]][0]), "freqs": m.precompute_freqs_cis(a).to(DEVICE), "mask": _causal(T)}
    at(s["x"][:, :16].contiguous(), 0, s["freqs"][:16], _causal(16))
    return s


@torch.inference_mode()
def _run_attention(s):
    at = s["layer"]
    return [at(s["x"], 0, s["freqs"], s["mask"]), at.kv_cache, at.pe_cache]


def _prepare_block(case, seed):
    _, m = _integer_modules(case["scales"])
    T = case["tokens"]
    a = _integer_args(m, T)
    with torch.device(DEVICE):
        blk = m.Block(0, a)
    _fill_block(blk, seed, a, "l0.", case["scales"])
    s = {"layer": blk, "x": _whole(seed, "x", (1, T, a.dim), 2.0 ** _SCALES[case["scales"]][0]), "freqs": m.precompute_freqs_cis(a).to(DEVICE), "mask": _causal(T)}
    blk(s["x"][:, :16].contiguous(), 0, s["freqs"][:16], _causal(16))
    return s


@torch.inference_mode()
def _run_block(s):
    blk = s["layer"]
    return [blk(s["x"], 0, s["freqs"], s["mask"]), blk.attn.kv_cache, blk.attn.pe_cache]


def _prepare_experts(case, seed):
    _, m = _integer_modules()
    a = _integer_args(m, 64, experts=case["experts"])
    with torch.device(DEVICE):
        moe = m.MoE(3, a)
    _fill_experts(moe, seed, a, "l3.")
    s = {"layer": moe, "x": _whole(seed, "x", (1, case["tokens"], a.dim), 2.0 ** 16)}
    moe(0, s["x"][:, :9].contiguous())
    return s


@torch.inference_mode()
def _run_experts(s):
    return s["layer"](0, s["x"])


def _prepare_decode(case, seed):
    _, m = _integer_modules()
    B, C = case["batch"], case["cache"]
    a = _integer_args(m, C + 64, layers=2, dense=1, experts=case["experts"], vocab=case["vocab"])
    with torch.device(DEVICE):
        model = m.Transformer(a)
    model.embed.weight = _whole(seed, "embed", (a.vocab_size, a.dim), 2.0 ** 16)
    model.norm.weight = _norm_weight(seed, "norm", a.dim, torch.int64)
    model.head.weight, model.head.weight_rescale, model.head.res_rescale = _weight(seed, "head", a.vocab_size, a.dim, torch.int64), 1, 16
    for i in range(a.n_layers):
        with torch.device(DEVICE):
            blk = m.Block(i, a, cache_batch=B)
        _fill_block(blk, seed, a, "l%d." % i)
        blk.attn.kv_cache[:, :C] = _whole(seed, "kv%d" % i, (B, C, a.kv_lora_rank), 2.0 ** 16)
        blk.attn.pe_cache[:, :C] = _whole(seed, "pe%d" % i, (B, C, a.qk_rope_head_dim), 2.0 ** 16)
        model.layers[i] = blk
    tokens = torch.randint(0, a.vocab_size, (2, B, 1), generator=_generator(seed, "tokens"), device=DEVICE)
    batch = model.begin_batch(B)
    model.step(tokens[0], C - 1, batch)
    return {"model": model, "tokens": tokens[1], "position": C, "batch": batch}


def _run_decode(s):
    model, at = s["model"], s["position"]
    logits, _ = model.step(s["tokens"], at, s["batch"])
    held = [t[:, at] for blk in model.layers for t in (blk.attn.kv_cache, blk.attn.pe_cache)]
    return [logits, logits[0].argmax(dim=-1)] + held


# ---- floating-point designs ----------------------------------------------------------------------------------------------
def _vocab(case):
    return 32768


def _config(case):
    window = case.get("window", 4096)
    cfg = {"vocab": _vocab(case), "norm": {"eps": 1e-6}}
    if case["kind"].startswith("munalorn"):
        w, H, q, c, ff = MUNALORN[case["size"]]
        mixer = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": q, "kv_rank": c, "scale": 192 ** -0.5,
                 "mask": {"size": window}, "rot": {"base": 10000.0, "dims": 64}}
        ff = {"kind": "dense", "ff": ff}
        # the second layer reads the latents of the first
        layers = [{"type": "latent_attention", "mixer": mixer, "mlp": ff},
                  {"type": "latent_attention", "mixer": dict(mixer, kv_from=0), "mlp": ff}]
        return dict(cfg, architecture="Munalorn", width=w, layers=layers)
    w, H, G, R, M, ff = VIFELIX[case["size"]]
    left = {"heads": H, "kv_heads": G, "dim": 128, "mask": {"size": window}, "rot": {"base": 10000.0, "dims": 128}, "scale": 128 ** -0.5}
    right = {"heads": R, "dim": 128, "vdim": 256, "decay": [1 - 2.0 ** (-5 - i % 8) for i in range(R)],
             "rot": {"base": 10000.0, "dims": 128}}
    mamba = {"heads": M, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    return dict(cfg, architecture="Vifelix", width=w, embedding={"scale": 1.0}, layers=[
        {"type": "mamba2", "mlp": None, "mixer": mamba},
        {"type": "parallel", "mlp": {"kind": "dense", "ff": ff},
         "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}}])


def _weights(case, seed):
    """name, shape -> bfloat16 weights as a checkpoint holds them"""
    around_zero = case["kind"].startswith("vifelix")

    def weight(name, shape):
        t = torch.randn(shape, generator=_generator(seed, name), device=DEVICE, dtype=torch.bfloat16)
        if name.endswith((".A_log", ".dt_bias")):
            return t * 0.5 - 2.0
        if len(shape) == 1:
            zero = name.endswith(".b") or around_zero and not name.endswith((".q.norm", ".k.norm", "mix.norm", ".D"))
            return t * 0.1 if zero else t * 0.1 + 1
        return t if name == "embed" else t * shape[1] ** -0.5
    return weight


def _tokens(case, seed, length):
    return torch.randint(0, _vocab(case), (case.get("batch", 1), length), generator=_generator(seed, "tokens"), device=DEVICE)


def _float_model(case, seed, positions):
    build = _module("build")
    build.build(library=build.FLOAT_LIBRARY)
    fm, fc = _module("float_model"), _module("float_config")
    args = fc.parse_config(_config(case))
    args.max_seq_len, args.max_batch_size = positions, case.get("batch", 1)
    return fm.FloatTransformer(args, getattr(torch, case["dtype"])).load_weights(_weights(case, seed), torch.device(DEVICE))


def _held(model, slots, begin, end):
    """what the model keeps of the sequences: entries of positions begin .. end - 1, recurrent sums"""
    cache = model.cache
    rows = [b[slots, begin:end] for b in cache.buffers if b is not None]
    return rows + [st["sums"][slots] for st in cache.states if "sums" in st]


def _prepare_prompt(case, seed):
    T = case["tokens"]
    return {"model": _float_model(case, seed, T + 64), "tokens": _tokens(case, seed, T)}


def _run_prompt(s):
    model, tokens = s["model"], s["tokens"]
    slots = model.begin_batch(1)
    logits, _ = model.step(tokens, 0, slots)
    out = [logits] + _held(model, slots, 0, tokens.shape[1])
    model.end_batch(slots)
    return out


def _prepare_munalorn_decode(case, seed):
    C = case["cache"]
    model, tokens = _float_model(case, seed, C + 64), _tokens(case, seed, C + 1)
    slots = model.begin_batch(case["batch"])
    model.step(tokens[:, :C], 0, slots, want=[])
    return {"model": model, "tokens": tokens[:, C:].contiguous(), "position": C, "slots": slots}


def _run_munalorn_decode(s):
    model, at, slots = s["model"], s["position"], s["slots"]
    for slot in slots:
        model.cache.truncate(slot, at)      # as a program does that tries another continuation
    logits, _ = model.step(s["tokens"], at, slots)
    return [logits] + _held(model, slots, at, at + 1)


def _prepare_request(case, seed):
    n = case["prompt"] + case["new"]
    return {"model": _float_model(case, seed, 512), "tokens": _tokens(case, seed, n), "prompt": case["prompt"]}


def _run_request(s):
    model, tokens, P = s["model"], s["tokens"], s["prompt"]
    slots = model.begin_batch(tokens.shape[0])
    logits = [model.step(tokens[:, :P], 0, slots)[0]]
    for p in range(P, tokens.shape[1]):
        logits.append(model.step(tokens[:, p:p + 1], p, slots)[0])
    out = logits + _held(model, slots, 0, tokens.shape[1])
    model.end_batch(slots)
    return out


_KINDS = {"projection": (_prepare_projection, _run_projection), "fixedpoint": (_prepare_fixedpoint, _run_fixedpoint),
          "attention": (_prepare_attention, _run_attention), "block": (_prepare_block, _run_block),
          "experts": (_prepare_experts, _run_experts), "decode": (_prepare_decode, _run_decode),
          "munalorn_prompt": (_prepare_prompt, _run_prompt), "munalorn_decode": (_prepare_munalorn_decode, _run_munalorn_decode),
          "vifelix_prompt": (_prepare_prompt, _run_prompt), "vifelix_request": (_prepare_request, _run_request)}


def prepare(case, seed):
    make, go = _KINDS[case["kind"]]
    with torch.inference_mode():
        return go, make(case, seed)


def run(state):
    go, s = state
    return go(s)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def _attention_work(T, B, keys):
    """(multiply-adds, weights, other words) of the integer attention layer for B * T tokens that see `keys` positions"""
    D, q, C, R, H, n, v = 7168, 1536, 512, 64, 128, 128, 128
    weights = D * q + q * H * (n + R) + D * (C + R) + H * n * C + H * C * v + H * v * D
    rows = B * T
    seen = rows * keys if T == 1 else B * T * (T + 1) // 2
    return rows * weights + seen * H * (2 * C + R), weights, rows * (2 * D + C + R) + B * (keys - T) * (C + R)


def _float_work(case):
    """(multiply-adds, weight elements, element bytes) of all the tokens that a pass runs"""
    size, request = 2 if case["dtype"] == "bfloat16" else 4, case["kind"].endswith("request")
    B = case.get("batch", 1)
    if case["kind"].endswith("decode"):
        T, start = 1, case["cache"]
    else:
        T, start = case["prompt"] + case["new"] if request else case["tokens"], 0
    window = case.get("window", 4096)
    seen = sum(min(window, start + t + 1) for t in range(T))
    if case["kind"].startswith("munalorn"):
        w, H, q, c, ff = MUNALORN[case["size"]]
        layer = w * q + H * 192 * q + H * 256 * c + 2 * H * 128 * w + 3 * w * ff
        weights, mixing = 2 * layer + w * (c + 64), 2 * seen * H * 320
        held = B * (start + T) * (c + 64)
    else:
        w, H, G, R, M, ff = VIFELIX[case["size"]]
        mamba = w * (2 * M * 64 + 2 * 8 * 128 + M) + M * 64 * w
        weights = mamba + w * (2 * H + G) * 128 + H * 128 * w + R * w * (256 + 512) + R * 256 * w + 3 * w * ff
        mixing = seen * H * 256 + 2 * T * (M * 128 * 64 + R * 128 * 256)
        held = B * (start + T) * 2 * G * 128 + 2 * (M * 128 * 64 + R * 128 * 256)
    steps = case["new"] + 1 if request else 1
    head = w * _vocab(case)
    macs = B * T * weights + B * mixing + B * steps * head
    if not request:
        return macs, weights + head, size, held * size + 4 * B * _vocab(case)
    # every token after the prompt needs the weights again
    return macs, steps * (weights + head), size, held * size + 4 * B * steps * _vocab(case)


def work(case):
    """Integer weights that a program has laid out count two bytes each, or four at the reference's
    magnitudes: the bits of their values.  Operations are the
    multiply-adds of the products themselves, whatever an exact product on narrow units splits them into."""
    kind = case["kind"]
    if kind == "projection":
        M, K, N = case["rows"], case["inner"], case["outer"]
        return {"bytes": 8 * M * K + case["weight_bits"] // 8 * N * K + 16 * M * N, "flops": 2 * M * K * N}
    if kind == "fixedpoint":
        T = case["tokens"]
        return {"bytes": 16 * T * (7168 + 128 * 64 + 128 * T + 18432), "flops": 0}
    if kind in ("attention", "block"):
        T = case["tokens"]
        macs, weights, words = _attention_work(T, 1, T)
        if kind == "block":
            macs, weights = macs + T * 3 * 7168 * 18432, weights + 3 * 7168 * 18432
        return {"bytes": (2 if case["scales"] == "small" else 4) * weights + 8 * words, "flops": 2 * macs}
    if kind == "experts":
        T, each = case["tokens"], 3 * 7168 * 2048
        E = min(case["experts"], 8 * T)
        return {"bytes": 2 * ((E + 1) * each + 7168 * case["experts"]) + 16 * T * 7168,
                "flops": 2 * T * (9 * each + 7168 * case["experts"])}
    if kind == "decode":
        B, each = case["batch"], 3 * 7168 * 2048
        macs, weights, words = _attention_work(1, B, case["cache"] + 1)
        hit = min(case["experts"], 8 * B)
        head = 7168 * case["vocab"]
        return {"bytes": 2 * (2 * weights + 3 * 7168 * 18432 + (hit + 1) * each + head) + 8 * (2 * words + B * case["vocab"]),
                "flops": 2 * (2 * macs + B * (3 * 7168 * 18432 + 9 * each + head))}
    macs, weights, size, other = _float_work(case)
    return {"bytes": weights * size + other, "flops": 2 * macs}


def tolerance(case):
    if case["kind"] in ("projection", "fixedpoint", "attention", "block", "experts", "decode"):
        return "exact"
    # bfloat16: activations are rounded between products, which puts results 5e-3 off exact(); float32: sums in 32 bits, 2e-6
    # off.  About four times that
    return {"rel": 2e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-5}


# ---- the floating-point designs in 64 bits -------------------------------------------------------------------------------
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, base, half):
    """x [batch, tokens, ..., R], turned by its position: pairs (2i, 2i + 1), or with `half` (i, i + R / 2)"""
    R, T = x.shape[-1], x.shape[1]
    f = float(base) ** (-torch.arange(0, R, 2, dtype=torch.float64, device=x.device) / R)
    ang = torch.arange(T, dtype=torch.float64, device=x.device)[:, None] * f
    ang = ang.view((1, T) + (1,) * (x.dim() - 3) + (R // 2,))
    u, v = (x[..., :R // 2], x[..., R // 2:]) if half else (x[..., 0::2], x[..., 1::2])
    a, b = u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()
    return torch.cat([a, b], -1) if half else torch.stack([a, b], -1).flatten(-2)


def _softmax(q, k, v, scale, window):
    """q, k, v [tokens, size] of one head"""
    T = q.shape[0]
    back = torch.arange(T, device=q.device)[:, None] - torch.arange(T, device=q.device)[None, :]
    s = (q @ k.T * scale).masked_fill_((back < 0) | (back >= window), -math.inf)
    return torch.softmax(s, -1) @ v


def _sums(q, k, v, decay):
    """S_t = decay_t S_{t-1} + k_t v_t^T, o_t = S_t^T q_t; q, k [B, T, H, N], v [B, T, H, P], decay [B, T, H]"""
    B, T, H, P = v.shape
    S = torch.zeros(B, H, k.shape[-1], P, dtype=torch.float64, device=v.device)
    o = torch.empty_like(v)
    for t in range(T):
        S = S * decay[:, t, :, None, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        o[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :]
    return o, S


def _adjacent(x):
    """pairs (i, i + R / 2) of the last dimension side by side, as the cache holds them"""
    R = x.shape[-1]
    return torch.stack([x[..., :R // 2], x[..., R // 2:]], -1).flatten(-2)


def _munalorn(case, W, x):
    cfg, c = _config(case), None
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        H, D, R, C, w = m["heads"], 128, 64, m["kv_rank"], cfg["width"]
        if i == 0:
            y = x @ W(p + "mix.dkv", (C + R, w)).T
            c, kr = _rms(y[..., :C], 1e-6) * W(p + "mix.dkv.norm", (C,)), _turn(y[..., C:], 1e4, False)
        cq = _rms(x @ W(p + "mix.dq", (m["q_rank"], w)).T, 1e-6) * W(p + "mix.dq.norm", (m["q_rank"],))
        q = (cq @ W(p + "mix.uq", (H * (D + R), m["q_rank"])).T).unflatten(-1, (H, D + R))
        q = torch.cat([q[..., :D], _turn(q[..., D:], 1e4, False)], -1)
        uk, uv = (W(p + "mix." + n, (H * D, C)).view(H, D, C) for n in ("uk", "uv"))
        o = torch.empty(*x.shape[:2], H, D, dtype=torch.float64, device=x.device)
        for b in range(x.shape[0]):
            for h in range(H):
                o[b, :, h] = _softmax(q[b, :, h], torch.cat([c[b] @ uk[h].T, kr[b]], -1), c[b] @ uv[h].T, m["scale"], m["mask"]["size"])
        gate = torch.sigmoid(x @ W(p + "mix.g", (H * D, w)).T)
        x = x + _rms((o.flatten(2) * gate) @ W(p + "mix.o", (w, H * D)).T, 1e-6) * W(p + "norm1", (w,))
        ff = layer["mlp"]["ff"]
        hidden = torch.nn.functional.silu(x @ W(p + "mlp.gate", (ff, w)).T) * (x @ W(p + "mlp.up", (ff, w)).T)
        x = x + _rms(hidden @ W(p + "mlp.down", (w, ff)).T, 1e-6) * W(p + "norm2", (w,))
    return x, [torch.cat([c, kr], -1)]


def _vifelix(case, W, x):
    cfg = _config(case)
    w, silu = cfg["width"], torch.nn.functional.silu
    norm = lambda t, name: _rms(t, 1e-6) * (1 + W(name, (w,)))
    # Mamba-2
    m = cfg["layers"][0]["mixer"]
    H, P, N, G = m["heads"], 64, 128, 8
    inner, p = H * P, "l0.mix."
    y = norm(x, "l0.norm1") @ W(p + "in", (2 * inner + 2 * G * N + H, w)).T
    z, u, dt = y[..., :inner], y[..., inner:2 * inner + 2 * G * N], y[..., 2 * inner + 2 * G * N:]
    taps = W(p + "conv", (inner + 2 * G * N, 4))
    padded = torch.nn.functional.pad(u, (0, 0, 3, 0))
    u = silu(sum(padded[:, j:j + u.shape[1]] * taps[:, j] for j in range(4)) + W(p + "conv.b", (inner + 2 * G * N,)))
    v = u[..., :inner].unflatten(-1, (H, P))
    spread = lambda t: t.unflatten(-1, (G, N)).repeat_interleave(H // G, dim=2)
    Bm, Cm = spread(u[..., inner:inner + G * N]), spread(u[..., inner + G * N:])
    dt = torch.nn.functional.softplus(dt + W(p + "dt_bias", (H,)))
    o, state = _sums(Cm, Bm * dt[..., None], v, torch.exp(-torch.exp(W(p + "A_log", (H,))) * dt))
    del Bm, Cm
    o = ((o + W(p + "D", (H,))[:, None] * v).flatten(2) * silu(z)).unflatten(-1, (m["norm_groups"], -1))
    o = _rms(o, 1e-6).flatten(2) * W(p + "norm", (inner,))
    x = x + norm(o @ W(p + "o", (w, inner)).T, "l0.norm1b")
    # attention beside retention
    layer = cfg["layers"][1]
    m, p, h = layer["mixer"]["left"], "l1.mix.left.", norm(x, "l1.norm1")
    H, G, D = m["heads"], m["kv_heads"], 128
    q = (h @ W(p + "q", (H * D, w)).T + W(p + "q.b", (H * D,))).unflatten(-1, (H, D))
    v = (h @ W(p + "k", (G * D, w)).T + W(p + "k.b", (G * D,))).unflatten(-1, (G, D))
    q = _turn(_rms(q, 1e-6) * W(p + "q.norm", (D,)), 1e4, True)
    k = _turn(_rms(v, 1e-6) * W(p + "k.norm", (D,)), 1e4, True)
    o = torch.empty_like(q)
    for b in range(x.shape[0]):
        for j in range(H):
            o[b, :, j] = _softmax(q[b, :, j], k[b, :, j // (H // G)], v[b, :, j // (H // G)], m["scale"], m["mask"]["size"])
    mixed = (o.flatten(2) * torch.sigmoid(h @ W(p + "g", (H * D, w)).T)) @ W(p + "o", (w, H * D)).T
    rows = torch.cat([_adjacent(k).flatten(2), _adjacent(v).flatten(2)], -1)
    m, p = layer["mixer"]["right"], "l1.mix.right."
    R, V = m["heads"], m["vdim"]
    q, k = (_turn((h @ W(p + n, (R * D, w)).T).unflatten(-1, (R, D)), 1e4, True) for n in ("q", "k"))
    v = (h @ W(p + "v", (R * V, w)).T).unflatten(-1, (R, V))
    decay = torch.tensor(m["decay"], dtype=torch.float64, device=x.device).expand(*x.shape[:2], R)
    o, sums = _sums(q, k * D ** -0.5, v, decay)
    o = _rms(o, 1e-6).flatten(2) * silu(h @ W(p + "g", (R * V, w)).T)
    mixed = mixed + o @ W(p + "o", (w, R * V)).T
    x = x + norm(mixed, "l1.norm1b")
    ff, h = layer["mlp"]["ff"], norm(x, "l1.norm2")
    hidden = silu(h @ W("l1.mlp.gate", (ff, w)).T + W("l1.mlp.gate.b", (ff,))) * (h @ W("l1.mlp.up", (ff, w)).T + W("l1.mlp.up.b", (ff,)))
    x = x + norm(hidden @ W("l1.mlp.down", (w, ff)).T + W("l1.mlp.down.b", (w,)), "l1.norm2b")
    return x, [rows, state, _adjacent(sums.transpose(-1, -2)).transpose(-1, -2)]


@torch.inference_mode()
def exact(case, seed):
    """None for the integer model: its outputs are whole numbers, compared word for word"""
    kind = case["kind"]
    if not kind.startswith(("munalorn", "vifelix")):
        return None
    weight = _weights(case, seed)
    W = lambda name, shape: weight(name, shape).double()
    first = {"munalorn_decode": "cache", "vifelix_request": "prompt"}.get(kind)
    length = case["tokens"] if first is None else case["cache"] + 1 if first == "cache" else case["prompt"] + case["new"]
    tokens = _tokens(case, seed, length)
    munalorn = kind.startswith("munalorn")
    w, V = _config(case)["width"], _vocab(case)
    embed = W("embed", (V, w))
    x, held = (_munalorn if munalorn else _vifelix)(case, W, embed[tokens])
    final = W("final.norm", (w,)) + (0 if munalorn else 1)
    head = embed if munalorn else W("head", (V, w))
    wanted = range(case["prompt"] - 1, length) if kind == "vifelix_request" else [length - 1]
    logits = [_rms(x[:, t], 1e-6) * final @ head.T for t in wanted]
    if kind == "munalorn_decode":
        held = [t[:, -1:] for t in held]
    return logits + held
