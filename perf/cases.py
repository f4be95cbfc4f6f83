"""What a user of this package has it do, as cases that can be timed and compared.

Seven kinds of work, each through its public entry points:

* ``matvec``      one NVFP4 projection of one token (``kernels.nvfp4_gemv``): the smallest call there is;
* ``blocks``      the three mixer and expert blocks of the operator table on one token, at a cached context;
* ``step``        one token through the fused step of the NVFP4 hybrid MoE model;
* ``prompt``      ``Engine.prefill`` of the NVFP4 model, with NVFP4 or static-FP8 mixers;
* ``batch``       one step of a batch of sequences (``BatchDecode.graph_step``), each at its own state;
* ``projection``  a chunk of tokens through one NVFP4 projection, exact (``kernels.matmul``) or with both operands NVFP4
                  (``kernels.quantize_act`` and ``kernels.matmul_w4a4``);
* ``hybrid``      a bf16-weight model (Fezopel or Dokulix): a prompt or one more token through ``Engine.extend``.

The models have the layer sizes of the whole ones and fewer layers.  ``exact`` is the same mathematics in 64 bits in plain
torch; where a value depends on which experts a router with 16-bit inputs picked, there is no such value (None).
"""

import math

import torch

from quickdraw_b200 import kernels, synthetic
from quickdraw_b200.batch import BatchDecode, BatchState
from quickdraw_b200.engine import Engine
from quickdraw_b200.fused import FusedStep
from quickdraw_b200.loader import hybrid_shapes
from quickdraw_b200.state import DecodeState

DEVICE = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
VOCAB = 151936             # of the NVFP4 model
MOE_LAYERS = 4             # one group: three gated-DeltaNet layers and one of attention


def listed():
    return [
        # one projection of one token through the operator table: latency
        {"name": "matvec_1024x2048", "kind": "matvec", "out": 1024, "inp": 2048},
        # a caller with a step of its own over the operator table, one layer's blocks at a long context
        {"name": "blocks_context_8192", "kind": "blocks", "context": 8192},
        # chat decoding: one token behind a 512-token prompt and some answer
        {"name": "step_8_layers_context_639", "kind": "step", "layers": 8, "context": 639, "fp8": False},
        # a short prompt of no particular length
        {"name": "prompt_511", "kind": "prompt", "tokens": 511, "fp8": False},
        # a long document
        {"name": "prompt_8192", "kind": "prompt", "tokens": 8192, "fp8": False},
        # the published checkpoint's number formats (static-FP8 mixers, NVFP4 head)
        {"name": "prompt_2048_fp8_mixers", "kind": "prompt", "tokens": 2048, "fp8": True},
        # a small server
        {"name": "batch_32_context_8192", "kind": "batch", "batch": 32, "context": 8192},
        # a projection of a chunk on the FP4 tensor cores
        {"name": "projection_8192_w4a4", "kind": "projection", "tokens": 8192, "out": 8192, "inp": 2048, "w4a4": True},
        # prompts of the bf16-weight models: recurrences and windows, latents and chunks
        {"name": "fezopel_prompt_2048", "kind": "hybrid", "design": "fezopel", "width": 2048, "layers": 6, "span": 1024, "context": 0,
         "tokens": 2048, "fp32": False},
        {"name": "dokulix_prompt_8192", "kind": "hybrid", "design": "dokulix", "width": 2048, "layers": 6, "span": 1024, "context": 0,
         "tokens": 8192, "fp32": False},
        # the same model in true fp32, as a check of a conversion runs it
        {"name": "fezopel_prompt_777_fp32", "kind": "hybrid", "design": "fezopel", "width": 2048, "layers": 6, "span": 1024, "context": 0,
         "tokens": 777, "fp32": True},
        # decoding of a bf16-weight model
        {"name": "dokulix_token_context_512", "kind": "hybrid", "design": "dokulix", "width": 2048, "layers": 12, "span": 1024,
         "context": 512, "tokens": 1, "fp32": False},
    ]


def _log(rng, low, high):
    """A whole number between low and high, spread over its logarithm, odd ones among them."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["matvec", "blocks", "step", "prompt", "prompt", "batch", "projection", "projection", "hybrid", "hybrid", "hybrid", "token"])
    if kind == "matvec":
        return {"kind": kind, "out": _log(rng, 16, 131072), "inp": rng.choice([512, 1536, 2048, 2048, 4096, 4096])}
    if kind == "blocks":
        return {"kind": kind, "context": _log(rng, 16, 32768)}
    if kind == "step":
        return {"kind": kind, "layers": rng.choice([4, 8]), "context": _log(rng, 16, 32767), "fp8": rng.random() < 0.3}
    if kind == "prompt":
        return {"kind": kind, "tokens": _log(rng, 24, 8192), "fp8": rng.random() < 0.4}
    if kind == "batch":
        return {"kind": kind, "batch": rng.randint(2, 32), "context": _log(rng, 64, 8192)}
    if kind == "projection":
        w4a4 = rng.random() < 0.5
        return {"kind": kind, "tokens": _log(rng, 33, 8192), "out": 128 * _log(rng, 1, 64) if w4a4 else 8 * _log(rng, 16, 1024),
                "inp": 256 * _log(rng, 2, 16), "w4a4": w4a4}
    design, fp32 = rng.choice(["fezopel", "dokulix"]), rng.random() < 0.25
    case = {"kind": "hybrid", "design": design, "width": rng.choice([1024, 2048, 2048]), "span": rng.choice([256, 1024, 1024, 2048])}
    if kind == "token":
        return case | {"layers": rng.choice([6, 12]), "context": _log(rng, 16, 4096), "tokens": 1, "fp32": fp32}
    return case | {"layers": 6, "context": 0, "tokens": _log(rng, 24, 1024 if fp32 else 8192), "fp32": fp32}


# --------------------------------------------------------------------------------- what a program has in hand
def _generator(seed, salt):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 64 + salt)
    return g


def _normal(seed, salt, *shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=_generator(seed, salt), device=DEVICE, dtype=F32) * std).to(dtype)


def _tokens(seed, salt, count, vocab):
    return torch.randint(0, vocab, (count,), generator=_generator(seed, salt), device=DEVICE)


def _moe_config(case):
    return synthetic.model_config(num_layers=case.get("layers", MOE_LAYERS), vocab_size=VOCAB)


def _moe_checkpoint(case, seed):
    """Random weights whose tensor scales let every layer add about a twentieth to the stream, as a layer of a trained deep
    model does.  (With scales of one each layer outweighs all before it, and one near-tie of a router in bf16 decides
    everything behind it.)"""
    fp8 = case.get("fp8", False)
    ckpt = synthetic.make_checkpoint(_moe_config(case), seed, DEVICE, fp8_mixers=fp8, nvfp4_head=fp8)
    ckpt.embed_tokens.mul_(50.0)                                # a stream of about one
    for layer in ckpt.layers:
        out = layer.attn.o_proj if layer.layer_type == "full_attention" else layer.attn.out_proj
        for w, factor in ((out, 2.0 ** -9), (layer.moe.experts_down, 2.0 ** -10), (layer.moe.shared_down, 2.0 ** -10)):
            (w.weight_scale if w.weight.dtype != torch.uint8 else w.weight_scale_2).mul_(factor)
    return ckpt


def _hybrid_config(case):
    make = synthetic.fezopel_config if case["design"] == "fezopel" else synthetic.dokulix_config
    spans = {"window": case["span"]} if case["design"] == "fezopel" else {"window": case["span"], "chunk": case["span"]}
    return make(case["layers"], hidden=case["width"], heads=case["width"] // 128, kv_heads=case["width"] // 512, **spans)


def _hybrid_checkpoint(case, seed):
    return (synthetic.make_fezopel if case["design"] == "fezopel" else synthetic.make_dokulix)(_hybrid_config(case), seed, DEVICE)


def _hybrid_rows(case):
    """Positions that the caches are made for: some more than the case begins with, a token at a time goes on."""
    return case["tokens"] if not case["context"] else case["context"] + 32768


def _sequence_state(ckpt, seed, context, rows):
    """The history of a request that has ``context`` tokens behind it."""
    state = DecodeState.allocate(ckpt.config, rows, DEVICE)
    state.kv_k.copy_(_normal(seed, 1, *state.kv_k.shape))
    state.kv_v.copy_(_normal(seed, 2, *state.kv_v.shape))
    state.rec_state.copy_(_normal(seed, 3, *state.rec_state.shape, std=0.01, dtype=F32))
    state.conv_state.copy_(_normal(seed, 4, *state.conv_state.shape, std=4.0))
    return state


@torch.inference_mode()
def prepare(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        src = synthetic.Source(seed, DEVICE)
        return {"kind": kind, "x": src.normal("x", case["inp"]), "w": src.nvfp4("w", case["out"], case["inp"])}
    if kind == "projection":
        src = synthetic.Source(seed, DEVICE)
        return {"kind": kind, "w4a4": case["w4a4"], "x": src.normal("x", case["tokens"], case["inp"]), "w": src.nvfp4("w", case["out"], case["inp"])}
    if kind == "blocks":
        cfg, src = synthetic.model_config(num_layers=2, interval=2), synthetic.Source(seed, DEVICE)
        rows = case["context"] + 1
        return {"kind": kind, "config": cfg, "table": kernels.kernels(), "position": case["context"], "x": src.normal("x", cfg.hidden_size),
                "attn": synthetic.make_attention(cfg, src), "gdn": synthetic.make_gdn(cfg, src), "moe": synthetic.make_moe(cfg, src),
                "cache": (_normal(seed, 1, rows, 2, 256), _normal(seed, 2, rows, 2, 256)),
                "rec": _normal(seed, 3, 32, 128, 128, std=0.01, dtype=F32), "conv": _normal(seed, 4, cfg.conv_channels, 3, std=4.0)}
    if kind == "step":
        ckpt = _moe_checkpoint(case, seed)
        state = _sequence_state(ckpt, seed, case["context"], case["context"] + 1)
        return {"kind": kind, "ckpt": ckpt, "step": FusedStep(ckpt), "state": state, "token": _tokens(seed, 5, 1, VOCAB)[0],
                "position": case["context"], "rec": list(state.rec_state), "conv": list(state.conv_state), "k": list(state.kv_k), "v": list(state.kv_v)}
    if kind == "prompt":
        engine = Engine(_moe_checkpoint(case, seed), max_context=case["tokens"], device=DEVICE)
        s = engine.state
        return {"kind": kind, "engine": engine, "tokens": _tokens(seed, 5, case["tokens"], VOCAB).tolist(), "rec": list(s.rec_state),
                "conv": list(s.conv_state), "k": list(s.kv_k), "v": list(s.kv_v)}
    if kind == "batch":
        ckpt, batch, context = _moe_checkpoint(case, seed), case["batch"], case["context"]
        state = BatchState(ckpt.config, batch, 32768, DEVICE)      # room for the steps that follow
        for salt, buffer in ((1, state.kv_k), (2, state.kv_v)):
            for b in range(batch):
                buffer[b, :, :context] = _normal(seed, 100 * (b + 1) + salt, *buffer[b, :, :context].shape)
        state.rec_state.copy_(_normal(seed, 3, *state.rec_state.shape, std=0.01, dtype=F32))
        state.conv_state.copy_(_normal(seed, 4, *state.conv_state.shape, std=4.0))
        state.positions.fill_(context)
        return {"kind": kind, "decode": BatchDecode(ckpt), "state": state, "tokens": _tokens(seed, 5, batch, VOCAB),
                "rec": list(state.rec_state.unbind(1)), "conv": list(state.conv_state.unbind(1)),
                "k": list(state.kv_k[:, :, context].unbind(1)), "v": list(state.kv_v[:, :, context].unbind(1))}
    config = _hybrid_config(case)
    engine = Engine(_hybrid_checkpoint(case, seed), max_context=_hybrid_rows(case), device=DEVICE, dtype=F32 if case["fp32"] else BF16)
    tokens = _tokens(seed, 5, case["context"] + case["tokens"], config.vocab_size).tolist()
    filled = case["context"] + case["tokens"]
    history = []
    for layer in engine.state.layers:
        views = {name: getattr(layer, name) for name in ("k", "v", "latent", "rec", "conv") if getattr(layer, name) is not None}
        history.append({name: t if name in ("rec", "conv") else t[:min(filled, t.shape[0])] for name, t in views.items()})
    if case["context"]:
        engine.extend(tokens[:case["context"]])
    return {"kind": kind, "engine": engine, "continues": case["context"] > 0, "tokens": tokens[case["context"]:], "history": history}


# ------------------------------------------------------------------------------------------- one pass
@torch.inference_mode()
def run(state):
    kind = state["kind"]
    if kind == "matvec":
        return kernels.nvfp4_gemv(state["x"], state["w"])
    if kind == "projection":
        if not state["w4a4"]:
            return kernels.matmul(state["x"], state["w"])
        codes, scales, scale = kernels.quantize_act(state["x"])
        return {"codes": codes, "scales": scales.view(torch.uint8), "scale": scale, "y": kernels.matmul_w4a4((codes, scales, scale), state["w"])}
    if kind == "blocks":
        table, cfg, x = state["table"], state["config"], state["x"]
        return {"attention": table["full_attention_block"](state["attn"], x, state["cache"], state["position"], config=cfg),
                "delta": table["gated_delta_net_block"](state["gdn"], x, state["rec"], state["conv"], state["position"], config=cfg),
                "experts": table["moe_block"](state["moe"], x, config=cfg), "rec": state["rec"], "conv": state["conv"],
                "k": state["cache"][0], "v": state["cache"][1]}
    histories = {name: state[name] for name in ("rec", "conv", "k", "v") if name in state}
    if kind == "step":
        return {"logits": state["step"](state["ckpt"], state["token"], state["position"], state["state"]), **histories}
    if kind == "prompt":
        return {"logits": state["engine"].prefill(state["tokens"]), **histories}
    if kind == "batch":
        _, logits = state["decode"].graph_step(state["tokens"], state["state"])
        return {"logits": logits, **histories}
    engine = state["engine"]
    if not state["continues"]:
        engine.reset()
    return {"logits": engine.extend(state["tokens"], [len(state["tokens"]) - 1]), "history": state["history"]}


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def _nvfp4_bytes(out, inp):
    return out * inp // 2 + out * inp // 16


def _moe_sizes(cfg, fp8):
    """(dense weights, their bytes) of a DeltaNet layer and of an attention layer, without the experts; one expert's weights."""
    h = cfg.hidden_size
    delta, attention = 8192 * h + 4096 * h + 4096 * h, 8192 * h + 2 * 512 * h + 4096 * h
    shared, small = 3 * 512 * h, (cfg.num_experts + 1) * h
    per = 1.0 if fp8 else 0.5625
    return [(n + shared + small, n * per + shared * 0.5625 + 2 * small) for n in (delta + 64 * h, attention)], 3 * 512 * h


def _moe_work(case, tokens, pairs, state_bytes, heads_rows):
    cfg = _moe_config(case)
    (delta, attention), expert = _moe_sizes(cfg, case.get("fp8", False))
    full = cfg.layer_types.count("full_attention")
    linear = cfg.num_hidden_layers - full
    touched = cfg.num_experts * (1 - (1 - cfg.num_experts_per_tok / cfg.num_experts) ** tokens)
    head = VOCAB * cfg.hidden_size
    size = (linear * delta[1] + full * attention[1] + cfg.num_hidden_layers * touched * expert * 0.5625
            + head * (0.5625 if case.get("fp8") else 2) + state_bytes + heads_rows * VOCAB * 2)
    flops = 2 * tokens * (linear * delta[0] + full * attention[0] + cfg.num_hidden_layers * cfg.num_experts_per_tok * expert)
    flops += 2 * heads_rows * head + full * pairs * 16 * 4 * 256 + linear * tokens * 32 * 8 * 128 * 128
    return {"bytes": size, "flops": flops}


def _pairs(tokens, context, span, chunked):
    """(query, key) pairs that a window or a chunk of ``span`` lets see each other."""
    if chunked:
        return sum((context + i) % span + 1 for i in range(tokens))
    return sum(min(context + i + 1, span) for i in range(tokens))


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        return {"bytes": _nvfp4_bytes(case["out"], case["inp"]) + 2 * (case["out"] + case["inp"]), "flops": 2 * case["out"] * case["inp"]}
    if kind == "projection":
        t, o, i = case["tokens"], case["out"], case["inp"]
        more = _nvfp4_bytes(t, i) if case["w4a4"] else 0
        return {"bytes": _nvfp4_bytes(o, i) + 2 * t * (o + i) + more, "flops": 2 * t * o * i}
    if kind == "blocks":
        (delta, attention), expert = _moe_sizes(synthetic.model_config(num_layers=2, interval=2), False)
        rows = case["context"] + 1
        shared = 3 * 512 * 2048 * 0.5625 + 2 * 257 * 2048
        return {"bytes": delta[1] + attention[1] - shared + 8 * expert * 0.5625 + rows * 2048 + 2 * 32 * 128 * 128 * 4 + 6 * 8192,
                "flops": 2 * (delta[0] + attention[0] + 7 * expert) + rows * 16 * 4 * 256 + 32 * 8 * 128 * 128}
    if kind in ("step", "batch"):
        cfg, count = _moe_config(case), case.get("batch", 1)
        full = cfg.layer_types.count("full_attention")
        state = count * (full * (case["context"] + 1) * 2048 + (cfg.num_hidden_layers - full) * (2 * 32 * 128 * 128 * 4 + 2 * 8192 * 6))
        return _moe_work(case, count, count * (case["context"] + 1), state, count)
    if kind == "prompt":
        cfg, t = _moe_config(case), case["tokens"]
        full = cfg.layer_types.count("full_attention")
        state = full * t * 2048 + (cfg.num_hidden_layers - full) * (32 * 128 * 128 * 4 + 8192 * 6)
        return _moe_work(case, t, t * (t + 1) // 2, state, 1)
    config = _hybrid_config(case)
    rank = lambda _: 16
    shapes = hybrid_shapes(config, rank) if case["design"] == "fezopel" else hybrid_shapes(config)
    weights = sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and n not in ("embed", "head") and not n.endswith(".conv"))
    t, act = case["tokens"], 4 if case["fp32"] else 2
    size, flops = 2 * (weights + shapes["head"][0] * shapes["head"][1]) + t * case["width"] * 2, 2 * t * weights + 2 * shapes["head"][0] * case["width"]
    for layer in config.layers:
        m = layer.mixer
        if hasattr(m, "span"):
            pairs = _pairs(t, case["context"], m.span, case["design"] == "dokulix" and not hasattr(m, "kv_rank"))
            row = m.row if hasattr(m, "kv_rank") else m.kv_heads * (m.dim + m.vdim)
            flops += 2 * pairs * m.heads * (m.dim + getattr(m, "rot_dim", 0) + m.vdim)
            size += act * row * (t + min(case["context"], m.span))
        else:
            flops += 8 * t * m.heads * m.dim * m.vdim
            size += 4 * m.heads * m.dim * m.vdim * (1 if not case["context"] else 2)
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """About four times what the same work shows with its sums in another order (a prompt in other portions, a batch through the
    products of a prompt, a step as one launch per phase) or against 64 bits."""
    kind = case["kind"]
    if kind in ("matvec", "projection"):
        return {"rel": 4e-3}                 # one bf16 rounding of a sum in fp32
    if kind == "blocks":
        return {"rel": 1e-2}
    if kind == "hybrid":                     # portions: 0.8e-2 in bf16; 64 bits: 2e-6 in fp32
        return {"rel": 1e-5} if case["fp32"] else {"rel": 2e-2}
    return {"rel": 3e-2, "max": 0.6}         # 1e-2 and 0.17: a router's near-tie that falls the other way changes a token's rows


# ------------------------------------------------------------------------------------------- the same in 64 bits
E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _codes(packed):
    table = torch.tensor([*E2M1, *(-v for v in E2M1)], dtype=F64, device=packed.device)
    return table[torch.stack((packed & 15, packed >> 4), -1).long()].flatten(-2)


def _matrix(w):
    """A weight container as a 64-bit matrix."""
    if isinstance(w, torch.Tensor):
        return w.double()
    if w.weight.dtype != torch.uint8:
        return w.weight.double() * w.weight_scale.double()
    return _codes(w.weight) * w.weight_scale.double().repeat_interleave(16, -1) * w.weight_scale_2.double()


def _expert(bank, e):
    return _codes(bank.weight[e]) * bank.weight_scale[e].double().repeat_interleave(16, -1) * bank.weight_scale_2.double()


def _times(x, w):
    """x W^T; a static-FP8 projection rounds its input to E4M3 as its definition says."""
    if hasattr(w, "input_scale") and w.weight.dtype != torch.uint8:
        x = (x.to(BF16).float() / w.input_scale).clamp(-448, 448).to(torch.float8_e4m3fn).double() * w.input_scale.double()
    return x @ _matrix(w).T


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _layer_norm(x, n, eps):
    c = x - x.mean(-1, keepdim=True)
    return _rms(c, eps) * n.w.double() + n.b.double()


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale, first, *, offset=0, slopes=None, sink=None):
    """q [T, H, d], k [S, G, d], v [S, G, dv]: query i (position offset + i) sees the keys first(position) .. its own."""
    tokens, heads, _ = q.shape
    share = heads // k.shape[1]
    out = torch.empty((tokens, heads, v.shape[2]), dtype=F64, device=q.device)
    for a in range(0, tokens, 256):
        b = min(tokens, a + 256)
        at = torch.arange(offset + a, offset + b, device=q.device)
        low = first(at)
        lo, hi = int(low.min()), offset + b
        keys = torch.arange(lo, hi, device=q.device)
        seen = (keys[None] <= at[:, None]) & (keys[None] >= low[:, None])
        for g in range(k.shape[1]):
            part = q[a:b, g * share:(g + 1) * share].transpose(0, 1)                     # [share, queries, d]
            s = part @ k[lo:hi, g].T * scale
            if slopes is not None:
                s = s - slopes[g * share:(g + 1) * share, None, None] * (at[:, None] - keys[None])
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                extra = sink[g * share:(g + 1) * share, None, None].expand(-1, b - a, 1)
                p = torch.softmax(torch.cat([s, extra], -1), -1)[..., :-1]
            else:
                p = torch.softmax(s, -1)
            out[a:b, g * share:(g + 1) * share] = (p @ v[lo:hi, g]).transpose(0, 1)
    return out


def _angles(positions, base, dims):
    freq = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)
    a = positions.double()[:, None] * freq
    return a.cos()[:, None], a.sin()[:, None]


def _rotate_half(x, positions, base, dims):
    c, s = _angles(positions, base, dims)
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _rotate_pairs(x, positions, base, dims):
    c, s = _angles(positions, base, dims)
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)


def _delta_net(w, h, rec, conv, cfg):
    """Gated DeltaNet over h [T, B, width]; rec [B, 32, 128, 128], conv [B, channels, taps - 1]: (out, rec, conv)."""
    hk, dk, hv, dv = cfg.linear_num_key_heads, cfg.linear_key_head_dim, cfg.linear_num_value_heads, cfg.linear_value_head_dim
    mixed, z = _times(h, w.in_proj_qkv), _times(h, w.in_proj_z)
    a, b = _times(h, w.in_proj_a), _times(h, w.in_proj_b)
    tokens, taps = h.shape[0], w.conv1d.reshape(mixed.shape[-1], -1).double()
    window = torch.cat([conv.permute(2, 0, 1), mixed])
    x = _silu(sum(window[j:j + tokens] * taps[:, j] for j in range(taps.shape[1])))
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q, k, v = x.split([hk * dk, hk * dk, hv * dv], -1)
    q = unit(q.unflatten(-1, (hk, dk))).repeat_interleave(hv // hk, 2) / dk ** 0.5
    k = unit(k.unflatten(-1, (hk, dk))).repeat_interleave(hv // hk, 2)
    v = v.unflatten(-1, (hv, dv))
    beta, decay = torch.sigmoid(b), torch.exp(-w.A_log.double().exp() * torch.nn.functional.softplus(a + w.dt_bias.double()))
    out = torch.empty_like(v)
    for t in range(tokens):
        rec = rec * decay[t, ..., None, None]
        u = beta[t, ..., None] * (v[t] - (k[t, ..., None, :] @ rec)[..., 0, :])
        rec = rec + k[t, ..., None] * u[..., None, :]
        out[t] = (q[t, ..., None, :] @ rec)[..., 0, :]
    y = _rms(out, cfg.rms_norm_eps) * w.norm.double() * _silu(z.unflatten(-1, (hv, dv)))
    return _times(y.flatten(-2), w.out_proj), rec, window[-conv.shape[-1]:].permute(1, 2, 0)


def _exact_blocks(case, seed):
    s = prepare(case, seed)
    cfg, x, eps = s["config"], s["x"].double(), s["config"].rms_norm_eps
    w, position = s["attn"], torch.tensor([case["context"]], device=DEVICE)
    packed = _times(x, w.q_proj).view(1, 16, 512)
    rot = int(cfg.head_dim * cfg.partial_rotary_factor)
    q = _rotate_half(_rms(packed[..., :256], eps) * (1 + w.q_norm.double()), position, cfg.rope_theta, rot)
    k = _rotate_half(_rms(_times(x, w.k_proj).view(1, 2, 256), eps) * (1 + w.k_norm.double()), position, cfg.rope_theta, rot)
    keys, values = (t.double() for t in s["cache"])
    keys[case["context"]], values[case["context"]] = k[0], _times(x, w.v_proj).view(2, 256)
    heads = _attend(q, keys, values, 256 ** -0.5, torch.zeros_like, offset=case["context"])
    attention = _times((heads * torch.sigmoid(packed[..., 256:])).flatten(), w.o_proj)
    delta, rec, conv = _delta_net(s["gdn"], x[None, None], s["rec"].double()[None], s["conv"].double()[None], cfg)
    w = s["moe"]
    logits = _times(x, w.router).to(BF16).double()             # a router's logits are bf16 by definition: they decide
    ids = logits.argsort(descending=True, stable=True)[:cfg.num_experts_per_tok]
    p = torch.softmax(logits, 0)[ids]
    experts = sum(weight * (_silu(x @ _expert(w.experts_gate, e).T) * (x @ _expert(w.experts_up, e).T)) @ _expert(w.experts_down, e).T
                  for e, weight in zip(ids.tolist(), p / p.sum()))
    shared = _times(_silu(_times(x, w.shared_gate)) * _times(x, w.shared_up), w.shared_down)
    experts = experts + shared * torch.sigmoid(_times(x, w.shared_expert_gate))
    return {"attention": attention, "delta": delta.flatten(), "experts": experts, "rec": rec[0], "conv": conv[0], "k": keys, "v": values}


def _exact_moe(case, seed):
    """The histories of the first layer: what lies behind a router depends on 16-bit ties."""
    kind = case["kind"]
    s = prepare(case, seed)
    ckpt = s["ckpt"] if kind == "step" else s["engine"].ckpt if kind == "prompt" else s["decode"].ckpt
    layer, cfg = ckpt.layers[0], ckpt.config
    batch = case.get("batch", 1)
    ids = torch.tensor(s["tokens"], device=DEVICE)[:, None] if kind == "prompt" else s["tokens"][None] if kind == "batch" else s["token"].view(1, 1)
    h = _rms(ckpt.embed_tokens[ids].double(), cfg.rms_norm_eps) * (1 + layer.input_layernorm.double())
    if kind == "prompt":
        rec, conv = torch.zeros((1, 32, 128, 128), dtype=F64, device=DEVICE), torch.zeros((1, cfg.conv_channels, 3), dtype=F64, device=DEVICE)
    else:
        rec, conv = (s[name][0].double().reshape(batch, *shape) for name, shape in (("rec", (32, 128, 128)), ("conv", (-1, 3))))
    _, rec, conv = _delta_net(layer.attn, h, rec, conv, cfg)
    first = (lambda t: t) if kind == "batch" else (lambda t: t[0])
    return {"logits": None, "rec": [first(rec)] + [None] * (len(s["rec"]) - 1), "conv": [first(conv)] + [None] * (len(s["conv"]) - 1),
            "k": [None] * len(s["k"]), "v": [None] * len(s["v"])}


def _ring(rows, capacity):
    """Rows of positions 0 .. as a ring of ``capacity`` holds them."""
    if rows.shape[0] <= capacity:
        return rows
    at = torch.arange(rows.shape[0] - capacity, rows.shape[0], device=rows.device)
    out = torch.empty_like(rows[:capacity])
    out[at % capacity] = rows[at]
    return out


def _window(span):
    return lambda at: (at - span + 1).clamp(min=0)


def _fezopel_mixer(w, m, h, eps, capacity):
    tokens, at = h.shape[0], torch.arange(h.shape[0], device=DEVICE)
    if hasattr(m, "window"):
        q = (_rms(_times(h, w.q), eps) * w.q_norm.double()).view(tokens, m.heads, m.dim)
        k = (_rms(_times(h, w.k), eps) * w.k_norm.double()).view(tokens, m.kv_heads, m.dim)
        q, k = (_rotate_pairs(t, at, m.rotary_base, m.rotary_dims) for t in (q, k))
        v = _times(h, w.v).view(tokens, m.kv_heads, m.vdim)
        out = _attend(q, k, v, m.scale, _window(m.window), sink=w.sink.double())
        out = out * torch.sigmoid(_times(h, w.g))[..., None]
        return _times(out.flatten(1), w.o), {"k": _ring(k, capacity), "v": _ring(v, capacity)}
    z = _times(_times(h, w.a1), w.a2)
    state = torch.zeros((m.heads, m.dim, m.vdim), dtype=F64, device=DEVICE)
    out = torch.empty((tokens, m.heads, m.vdim), dtype=F64, device=DEVICE)
    if hasattr(m, "tau"):
        q = _times(h, w.q).view(tokens, m.heads, 1, m.dim) * m.dim ** -0.5
        k, v = _times(h, w.k).view(tokens, m.heads, m.dim, 1), _times(h, w.v).view(tokens, m.heads, 1, m.vdim)
        decay = torch.sigmoid(z + w.a2_b.double()).pow(1 / m.tau).view(tokens, m.heads, m.dim, 1)
        for t in range(tokens):
            state = decay[t] * state + k[t] * v[t]
            out[t] = (q[t] @ state)[:, 0]
        gate, history = _silu(_times(h, w.g)), {}
    else:
        raw = [_times(h, x) for x in (w.q, w.k, w.v)]
        conv = []
        for x, taps in zip(raw, (w.q_conv, w.k_conv, w.v_conv)):
            padded = torch.cat([x.new_zeros((m.conv - 1, x.shape[1])), x])
            conv.append(_silu(sum(padded[j:j + tokens] * taps.double()[:, j] for j in range(m.conv))))
        unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
        share = m.heads // m.kv_heads
        q = (unit(conv[0].view(tokens, m.kv_heads, m.dim)) * m.dim ** -0.5).repeat_interleave(share, 1)[:, :, None]
        k = unit(conv[1].view(tokens, m.kv_heads, m.dim)).repeat_interleave(share, 1)[:, :, None]
        v, beta = conv[2].view(tokens, m.heads, 1, m.vdim), torch.sigmoid(_times(h, w.b))[..., None, None]
        z = (z + w.dt_bias.double()).view(tokens, m.heads, m.dim)
        decay = torch.exp(-w.A_log.double().exp()[:, None] * torch.nn.functional.softplus(z))[..., None]
        for t in range(tokens):
            state = decay[t] * state
            state = state + k[t].transpose(1, 2) * (beta[t] * (v[t] - k[t] @ state))
            out[t] = (q[t] @ state)[:, 0]
        gate, history = torch.sigmoid(_times(_times(h, w.g1), w.g2)), {"conv": _ring(torch.cat(raw, 1), m.conv)}
        if tokens < m.conv:
            history["conv"] = torch.cat([history["conv"], history["conv"].new_zeros((m.conv - tokens, history["conv"].shape[1]))])
    out = (_rms(out, eps) * w.norm.double()).flatten(1)
    return _times(out * gate, w.o), {"rec": state, **history}


def _fezopel(ckpt, tokens, capacities):
    eps, x = ckpt.config.norm_eps, ckpt.embed_tokens[tokens].double()
    results, histories = [x], []

    def sublayer(x, around, mix):
        h = _layer_norm(x, around.norm, eps)
        y = mix(h) * torch.sigmoid(_times(h, around.gate) + around.gate_b.double())
        return x + _layer_norm(y, around.post, eps)

    for layer, cfg, capacity in zip(ckpt.layers, ckpt.config.layers, capacities):
        def mixer(h):
            y, history = _fezopel_mixer(layer.mixer, cfg.mixer, h, eps, capacity)
            histories.append(history)
            return y
        x = sublayer(x, layer.around_mixer, mixer)
        if layer.mlp is not None:
            x = sublayer(x, layer.around_mlp, lambda h: _times(torch.nn.functional.gelu(_times(h, layer.mlp.up)), layer.mlp.down))
        results.append(x)
        x = sum(c * r for c, r in zip(layer.depth.double(), results))
    return _layer_norm(x[-1:], ckpt.final_norm, eps) @ ckpt.lm_head.double().T, histories


def _dokulix_mixer(w, m, h, eps, capacity):
    tokens, at = h.shape[0], torch.arange(h.shape[0], device=DEVICE)
    if hasattr(m, "kv_rank"):
        dkv = _times(h, w.dkv)
        q = _times(_rms(_times(h, w.dq), eps) * w.dq_norm.double(), w.uq).view(tokens, m.heads, m.dim + m.rot_dim)
        q = torch.cat([q[..., :m.dim], _rotate_half(q[..., m.dim:], at, m.rotary_base, m.rot_dim)], -1)
        latent = _rms(dkv[:, :m.kv_rank], eps) * w.dkv_norm.double()
        shared = _rotate_half(dkv[:, None, m.kv_rank:], at, m.rotary_base, m.rot_dim)
        k = torch.cat([_times(latent, w.uk).view(tokens, m.heads, m.dim), shared.expand(-1, m.heads, -1)], -1)
        out = _attend(q, k, _times(latent, w.uv).view(tokens, m.heads, m.vdim), m.scale, _window(m.window)).flatten(1)
        row = latent.new_zeros((tokens, m.row))
        row[:, :m.kv_rank], row[:, m.rot_column:m.rot_column + m.rot_dim] = latent, shared[:, 0]
        return _times(out * torch.sigmoid(_times(h, w.g)), w.o), {"latent": _ring(row, capacity)}
    q = (_rms((_times(h, w.q) + w.q_b.double()).view(tokens, m.heads, m.dim), eps)) * w.q_norm.double()
    k = (_rms((_times(h, w.k) + w.k_b.double()).view(tokens, m.kv_heads, m.dim), eps)) * w.k_norm.double()
    v = (_times(h, w.v) + w.v_b.double()).view(tokens, m.kv_heads, m.vdim)
    slopes = torch.tensor([2.0 ** (-8.0 * (i + 1) / m.heads) for i in range(m.heads)], dtype=F64, device=DEVICE)
    out = _attend(q, k, v, m.scale, lambda p: p // m.span * m.span, slopes=slopes, sink=torch.zeros_like(slopes))
    return _times(out.flatten(1), w.o) + w.o_b.double(), {"k": _ring(k, capacity), "v": _ring(v, capacity)}


def _dokulix(ckpt, tokens, capacities):
    eps, x, histories = ckpt.config.norm_eps, ckpt.embed_tokens[tokens].double(), []
    for layer, cfg, capacity in zip(ckpt.layers, ckpt.config.layers, capacities):
        y, history = _dokulix_mixer(layer.mixer, cfg.mixer, _rms(x, eps) * (1 + layer.norm1.double()), eps, capacity)
        histories.append(history)
        x = x + y
        if layer.mlp is not None:
            h = _rms(x, eps) * (1 + layer.norm2.double())
            x = x + _times(_times(h, layer.mlp.gate).clamp(min=0) * _times(h, layer.mlp.up), layer.mlp.down)
    return (_rms(x[-1:], eps) * (1 + ckpt.final_norm.double())) @ ckpt.lm_head.double().T, histories


def _exact_hybrid(case, seed):
    ckpt = _hybrid_checkpoint(case, seed)
    tokens = _tokens(seed, 5, case["context"] + case["tokens"], ckpt.config.vocab_size)
    rows = _hybrid_rows(case)
    capacities = [min(rows, layer.mixer.span - 1 + 2048) if hasattr(layer.mixer, "span") else 0 for layer in ckpt.config.layers]
    logits, history = (_fezopel if case["design"] == "fezopel" else _dokulix)(ckpt, tokens, capacities)
    return {"logits": logits, "history": history}


def _quantised(x):
    """bf16 rows as NVFP4: (codes, E4M3 scales, tensor scale), every rounding to nearest even, and the values of the first two."""
    xf = x.float()
    top = xf.abs().max()
    g = top / torch.tensor(6.0 * 448.0, device=DEVICE)
    blocks = xf.unflatten(-1, (-1, 16))
    scale = (blocks.abs().amax(-1) / (torch.tensor(6.0, device=DEVICE) * g)).to(torch.float8_e4m3fn)
    s = scale.float() * g
    scaled = blocks * torch.where(s > 0, 1.0 / s, torch.zeros_like(s))[..., None]
    mag = scaled.abs().clamp(max=6.0)
    grid = torch.tensor(E2M1, device=DEVICE)
    lower = torch.bucketize(mag, grid, right=True) - 1
    upper = (lower + 1).clamp(max=7)
    middle = (grid[lower] + grid[upper]) / 2
    code = torch.where((mag > middle) | ((mag == middle) & (upper % 2 == 0)), upper, lower) + 8 * torch.signbit(scaled).long()
    code = code.flatten(-2).to(torch.uint8)
    packed = code[:, 0::2] | (code[:, 1::2] << 4)
    return packed, scale.view(torch.uint8), g, _codes(packed) * scale.double().repeat_interleave(16, -1)


@torch.inference_mode()
def exact(case, seed):
    kind = case["kind"]
    if kind == "blocks":
        return _exact_blocks(case, seed)
    if kind == "hybrid":
        return _exact_hybrid(case, seed)
    if kind not in ("matvec", "projection"):
        return _exact_moe(case, seed)
    s = prepare(case, seed)
    if not case.get("w4a4"):
        return _times(s["x"].double(), s["w"])
    codes, scales, scale, values = _quantised(s["x"])
    return {"codes": codes, "scales": scales, "scale": scale, "y": values @ _matrix(s["w"]).T * scale.double()}
