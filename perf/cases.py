"""The framework's main path as a set of measured cases.

A case is one call that a serving or control program makes over and over: a decode step of a batch, the prefill of a batch of
prompts, the encoding of images, an action chunk.  ``prepare`` builds the engine (weights drawn from the seed) and everything the
program holds between calls, ``run`` makes the call, ``exact`` is the same computation in plain 64-bit torch.  Decoders of several
billion parameters are cut to a few of their layers: widths, heads, vocabulary and with them every kernel's shape stay.
"""
import math

import torch
import torch.nn.functional as F

DEV = "cuda"
DTYPE = {"fp16": torch.float16, "bf16": torch.bfloat16}
BYTES = 2

# name: vocabulary, width, feed-forward, layers, heads, K/V heads, head size, epsilon, rotary base, tied head, norms on queries and keys
DECODERS = {
    "qwen3-0.6b": (151936, 1024, 3072, 28, 16, 8, 128, 1e-6, 1e6, True, True),
    "qwen3-1.7b": (151936, 2048, 6144, 28, 16, 8, 128, 1e-6, 1e6, True, True),
    "qwen3-4b": (151936, 2560, 9728, 36, 32, 8, 128, 1e-6, 1e6, True, True),
    "qwen3-8b": (151936, 4096, 12288, 36, 32, 8, 128, 1e-6, 1e6, False, True),
    "llama-3.2-1b": (128256, 2048, 8192, 16, 32, 8, 64, 1e-5, 5e5, True, False),
}
# the hybrid of gated attention and Gated-DeltaNet layers, the latent-attention / HGRN2 decoder and the chunked-attention / selective-scan
# decoder with routed experts: width -> heads, K/V heads or latent rank, feed-forward (of one expert)
HYBRID = {1024: (8, 2, 3584), 2048: (16, 4, 6144), 3072: (24, 6, 8192)}
LATENT = {2048: (16, 256, 8192), 3072: (24, 512, 12288)}
ROUTED = {2048: (16, 4, 1024), 3072: (24, 6, 1024)}
MIXED_VOCAB = 32768
ROOM = 256                       # decode steps behind a prompt before the program takes up the next batch of prompts


def listed():
    return [
        # one user of a small assistant, token by token: the smallest call, launches and latency count
        {"name": "step-1-small", "kind": "step", "model": "qwen3-0.6b", "layers": 28, "batch": 1, "context": 300, "dtype": "fp16", "quant": "none"},
        # a full batch of chats: the throughput point of the serving benchmark
        {"name": "step-64", "kind": "step", "model": "qwen3-8b", "layers": 4, "batch": 64, "context": 1024, "dtype": "fp16", "quant": "none"},
        # a handful of users on 8-bit weights
        {"name": "step-12-w8", "kind": "step", "model": "qwen3-8b", "layers": 4, "batch": 12, "context": 517, "dtype": "fp16", "quant": "w8a16"},
        # long documents being answered: K/V reading weighs as much as the weights
        {"name": "step-8-long", "kind": "step", "model": "qwen3-8b", "layers": 2, "batch": 8, "context": 8000, "dtype": "bf16", "quant": "none"},
        # one short question: time to first token
        {"name": "prompt-short", "kind": "prompts", "model": "llama-3.2-1b", "layers": 16, "batch": 1, "context": 93, "dtype": "fp16"},
        # eight prompts of unequal lengths in one launch
        {"name": "prompts-ragged", "kind": "prompts", "model": "qwen3-8b", "layers": 4, "batch": 8, "context": 1021, "dtype": "bf16"},
        # one long document, two chunks of 8192 rows
        {"name": "prompt-long", "kind": "prompts", "model": "qwen3-8b", "layers": 2, "batch": 1, "context": 16000, "dtype": "fp16"},
        # the hybrid decoder reading prompts
        {"name": "hybrid-prompts", "kind": "hybrid", "width": 2048, "layers": 4, "batch": 4, "context": 1500, "dtype": "bf16"},
        # decoders with per-layer mixers: latent attention and HGRN2 reading prompts, routed experts and selective scans in a decode step
        {"name": "latent-prompts", "kind": "latent", "width": 2048, "layers": 4, "batch": 6, "context": 1100, "dtype": "bf16"},
        {"name": "routed-step-32", "kind": "routed", "width": 2048, "layers": 4, "batch": 32, "context": 260, "dtype": "fp16"},
        # a vision tower over a batch of camera frames
        {"name": "images-12", "kind": "images", "images": 12, "dtype": "fp16"},
        # a robot's control step: three cameras, an instruction, ten denoising steps
        {"name": "action-chunk", "kind": "action", "batch": 1, "views": 3, "language": 57, "steps": 10, "dtype": "fp16"},
    ]


def _spread(rng, low, high):
    """A whole number of the range, evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "prompts", "prompts", "hybrid", "latent", "routed", "images", "action"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("step", "prompts"):
        model, layers = rng.choice([("qwen3-0.6b", 28), ("qwen3-1.7b", 12), ("qwen3-4b", 5), ("qwen3-8b", 4), ("llama-3.2-1b", 16)])
        if kind == "step":
            batch = _spread(rng, 1, 64)
            return {"kind": kind, "model": model, "layers": layers, "batch": batch, "context": _spread(rng, 40, min(4000, 65536 // batch)), "dtype": dtype,
                    "quant": rng.choice(["none", "none", "none", "w8a16", "w4a16"])}
        batch = _spread(rng, 1, 8)
        return {"kind": kind, "model": model, "layers": layers // 2, "batch": batch, "context": _spread(rng, 20, 8000 // batch), "dtype": dtype}
    if kind == "hybrid":
        batch = _spread(rng, 1, 6)
        return {"kind": kind, "width": rng.choice(sorted(HYBRID)), "layers": 4, "batch": batch, "context": _spread(rng, 30, 6000 // batch), "dtype": dtype}
    if kind == "latent":
        batch = _spread(rng, 1, 6)
        return {"kind": kind, "width": rng.choice(sorted(LATENT)), "layers": 4, "batch": batch, "context": _spread(rng, 30, 6000 // batch), "dtype": dtype}
    if kind == "routed":
        return {"kind": kind, "width": rng.choice(sorted(ROUTED)), "layers": 4, "batch": _spread(rng, 1, 48), "context": _spread(rng, 30, 300), "dtype": "fp16"}
    if kind == "images":
        return {"kind": kind, "images": _spread(rng, 1, 16), "dtype": dtype}
    return {"kind": kind, "batch": _spread(rng, 1, 2), "views": rng.randint(1, 3), "language": _spread(rng, 8, 200), "steps": rng.choice([5, 10]), "dtype": dtype}


# ---------------------------------------------------------------------------------------------------------------- weights and inputs
def _weights(shapes, seed, dtype):
    """Tensors by name from ``(name, shape, kind)`` rows, drawn on the GPU one behind the other."""
    g = torch.Generator(device=DEV).manual_seed(seed * 1000003 + 17)
    out = {}
    for name, shape, kind in shapes:
        t = torch.empty(shape, dtype=torch.float32, device=DEV)
        if kind == "unit":
            t.uniform_(0, 1, generator=g)
        elif kind == "scale":
            t.uniform_(0.25, 0.75, generator=g)
        elif kind == "log_a":
            t.uniform_(0.0, math.log(16.0), generator=g)
        elif kind == "dt_bias":
            t.uniform_(math.log(1e-3), math.log(1e-1), generator=g).exp_()
            t = t + torch.log(-torch.expm1(-t))
        else:
            t.normal_(0.0, 1.0, generator=g)
            if kind == "norm":
                t.mul_(0.05).add_(1.0)
            elif kind == "fan":
                t.mul_(shape[1] ** -0.5)
            elif kind == "correction":
                t.mul_(0.25 / shape[0])
            elif kind in ("linear", "bias"):
                t.mul_(0.02)
            elif kind == "back":               # into the residual stream: small beside the embedding, as deep models are initialised
                t.mul_(0.005)
            elif kind == "embed":
                t.mul_(0.5)
            elif kind == "norm0":
                t.mul_(0.05)
        out[name] = t.to(dtype)
    return out


def _decoder_shapes(case):
    V, H, I, _, heads, kv, hd, _, _, tied, qk = DECODERS[case["model"]]
    out = [("model.embed_tokens.weight", (V, H), "embed"), ("model.norm.weight", (H,), "norm")]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        out += [(p + "input_layernorm.weight", (H,), "norm"), (p + "post_attention_layernorm.weight", (H,), "norm"),
                (p + "self_attn.q_proj.weight", (heads * hd, H), "linear"), (p + "self_attn.k_proj.weight", (kv * hd, H), "linear"),
                (p + "self_attn.v_proj.weight", (kv * hd, H), "linear"), (p + "self_attn.o_proj.weight", (H, heads * hd), "back"),
                (p + "mlp.gate_proj.weight", (I, H), "linear"), (p + "mlp.up_proj.weight", (I, H), "linear"), (p + "mlp.down_proj.weight", (H, I), "back")]
        if qk:
            out += [(p + "self_attn.q_norm.weight", (hd,), "norm"), (p + "self_attn.k_norm.weight", (hd,), "norm")]
    return out if tied else out + [("lm_head.weight", (V, H), "linear")]


def _hybrid_shapes(case):
    H = case["width"]
    heads, kv, I = HYBRID[H]
    out = [("model.embed_tokens.weight", (MIXED_VOCAB, H), "embed"), ("model.norm.weight", (H,), "norm0")]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        out += [(p + "input_layernorm.weight", (H,), "norm0"), (p + "post_attention_layernorm.weight", (H,), "norm0"),
                (p + "mlp.gate_proj.weight", (I, H), "linear"), (p + "mlp.up_proj.weight", (I, H), "linear"), (p + "mlp.down_proj.weight", (H, I), "back")]
        if i % 2:
            a = p + "linear_attn."
            out += [(a + "in_proj_qkv.weight", (heads * 384, H), "linear"), (a + "in_proj_z.weight", (heads * 128, H), "linear"),
                    (a + "in_proj_b.weight", (heads, H), "linear"), (a + "in_proj_a.weight", (heads, H), "linear"), (a + "out_proj.weight", (H, heads * 128), "back"),
                    (a + "conv1d.weight", (heads * 384, 4), "fan"), (a + "A_log", (heads,), "log_a"), (a + "dt_bias", (heads,), "dt_bias"), (a + "norm.weight", (128,), "norm")]
        else:
            a = p + "self_attn."
            out += [(a + "q_proj.weight", (heads * 256, H), "linear"), (a + "k_proj.weight", (kv * 128, H), "linear"), (a + "v_proj.weight", (kv * 128, H), "linear"),
                    (a + "o_proj.weight", (H, heads * 128), "back"), (a + "q_norm.weight", (128,), "norm0"), (a + "k_norm.weight", (128,), "norm0")]
    return out


def _latent_shapes(case):
    H, L, P = case["width"], case["layers"], 128
    heads, rank, I = LATENT[H]
    out = [("embed", (MIXED_VOCAB, H), "normal"), ("side.embed", (MIXED_VOCAB, L * P), "normal"), ("final.norm", (H,), "norm")]
    for i in range(L):
        p, D = f"l{i}.", heads * 128
        out += [(p + "norm1", (H,), "norm"), (p + "norm2", (H,), "norm"), (p + "shift", (H,), "unit"), (p + "mix.q", (D, H), "fan"), (p + "mix.o", (H, D), "fan"),
                (p + "mlp.up", (I, H), "fan"), (p + "mlp.down", (H, I), "fan"), (p + "side.gate", (P, H), "fan"), (p + "side.proj", (H, P), "fan"), (p + "side.norm", (H,), "norm")]
        if i % 2:
            out += [(p + "mix.f", (D, H), "fan"), (p + "mix.f.b", (D,), "normal"), (p + "mix.lower", (D,), "unit"), (p + "mix.v", (D, H), "fan"), (p + "mix.norm", (128,), "norm")]
        else:
            out += [(p + "mix.dkv", (rank, H), "fan"), (p + "mix.dkv.norm", (rank,), "norm"), (p + "mix.uk", (D, rank), "fan"), (p + "mix.uv", (D, rank), "fan")]
    return out


def _routed_shapes(case):
    H = case["width"]
    heads, kv, ff = ROUTED[H]
    out = [("embed", (MIXED_VOCAB, H), "normal"), ("head", (MIXED_VOCAB, H), "fan"), ("final.norm", (H,), "norm")]
    for i in range(case["layers"]):
        p, D, N = f"l{i}.", heads * 128, 2 * H
        out += [(p + "norm1", (H,), "norm"), (p + "norm2", (H,), "norm"), (p + "ls1", (H,), "scale"), (p + "ls2", (H,), "scale")]
        if i % 2:
            out += [(p + "mix.q", (D, H), "fan"), (p + "mix.k", (kv * 128, H), "fan"), (p + "mix.v", (kv * 128, H), "fan"), (p + "mix.g", (D, H), "fan"), (p + "mix.o", (H, D), "fan"),
                    (p + "mix.q.norm", (128,), "norm"), (p + "mix.k.norm", (128,), "norm"), (p + "mix.sink", (heads,), "normal")]
        else:
            out += [(p + "mix.in", (2 * N, H), "fan"), (p + "mix.conv", (N, 4), "fan"), (p + "mix.conv.b", (N,), "normal"), (p + "mix.x", (H // 16 + 32, N), "fan"),
                    (p + "mix.dt", (N, H // 16), "fan"), (p + "mix.dt.b", (N,), "dt_bias"), (p + "mix.A_log", (N, 16), "log_a"), (p + "mix.D", (N,), "norm"), (p + "mix.o", (H, N), "fan")]
        for e, width in [(f"e{j}", ff) for j in range(16)] + [("shared", 2 * ff)]:
            out += [(f"{p}mlp.{e}.gate", (width, H), "fan"), (f"{p}mlp.{e}.up", (width, H), "fan"), (f"{p}mlp.{e}.down", (H, width), "fan")]
        out += [(p + "mlp.router", (16, H), "fan"), (p + "mlp.correction", (16,), "correction")]
    return out


VIT = (1152, 4304, 27, 16, 14, 256)            # width, feed-forward, layers, heads, patch, patches of a 224 x 224 image


def _tower_shapes(p):
    H, I, L, _, patch, n = VIT
    out = [(p + "embeddings.patch_embedding.weight", (H, 3, patch, patch), "linear"), (p + "embeddings.patch_embedding.bias", (H,), "bias"),
           (p + "embeddings.position_embedding.weight", (n, H), "linear"), (p + "post_layernorm.weight", (H,), "norm"), (p + "post_layernorm.bias", (H,), "bias")]
    for i in range(L):
        b = f"{p}encoder.layers.{i}."
        for x in ("layer_norm1", "layer_norm2"):
            out += [(f"{b}{x}.weight", (H,), "norm"), (f"{b}{x}.bias", (H,), "bias")]
        for x, rows, cols in [(f"self_attn.{t}", H, H) for t in ("q_proj", "k_proj", "v_proj", "out_proj")] + [("mlp.fc1", I, H), ("mlp.fc2", H, I)]:
            out += [(f"{b}{x}.weight", (rows, cols), "linear"), (f"{b}{x}.bias", (rows,), "bias")]
    return out


VLM, EXPERT = "paligemma_with_expert.paligemma.model.", "paligemma_with_expert.gemma_expert.model."
GEMMA_VOCAB, HORIZON, ACTION, DEPTH = 257152, 50, 32, 18


def _action_shapes():
    out = _tower_shapes(VLM + "vision_tower.vision_model.")
    out += [(VLM + "multi_modal_projector.linear.weight", (2048, 1152), "linear"), (VLM + "multi_modal_projector.linear.bias", (2048,), "bias"),
            (VLM + "language_model.embed_tokens.weight", (GEMMA_VOCAB, 2048), "linear")]
    for pre, H, I, ada in ((VLM + "language_model.", 2048, 16384, False), (EXPERT, 1024, 4096, True)):
        for i in range(DEPTH):
            b = f"{pre}layers.{i}."
            out += [(b + "self_attn.q_proj.weight", (2048, H), "linear"), (b + "self_attn.k_proj.weight", (256, H), "linear"), (b + "self_attn.v_proj.weight", (256, H), "linear"),
                    (b + "self_attn.o_proj.weight", (H, 2048), "linear"), (b + "mlp.gate_proj.weight", (I, H), "linear"), (b + "mlp.up_proj.weight", (I, H), "linear"),
                    (b + "mlp.down_proj.weight", (H, I), "linear")]
        for n in [f"layers.{i}.{x}" for i in range(DEPTH) for x in ("input_layernorm", "post_attention_layernorm")] + ["norm"]:
            out += [(f"{pre}{n}.dense.weight", (3 * H, H), "linear"), (f"{pre}{n}.dense.bias", (3 * H,), "bias")] if ada else [(f"{pre}{n}.weight", (H,), "norm0")]
    out += [("action_in_proj.weight", (1024, ACTION), "linear"), ("action_in_proj.bias", (1024,), "bias"), ("action_out_proj.weight", (ACTION, 1024), "linear"),
            ("action_out_proj.bias", (ACTION,), "bias")]
    for n in ("time_mlp_in", "time_mlp_out"):
        out += [(n + ".weight", (1024, 1024), "linear"), (n + ".bias", (1024,), "bias")]
    return out


def _shapes(case):
    kind = case["kind"]
    if kind in ("step", "prompts"):
        return _decoder_shapes(case)
    return {"hybrid": _hybrid_shapes, "latent": _latent_shapes, "routed": _routed_shapes, "images": lambda c: _tower_shapes("vision_model."),
            "action": lambda c: _action_shapes()}[kind](case)


def _vocab(case):
    return DECODERS[case["model"]][0] if "model" in case else MIXED_VOCAB


def _lengths(case):
    """Prompt lengths: the first is the case's, the others between a third of it and all of it."""
    n = case["context"]
    return [max(1, n - (2 * n // 3) * ((7 * i) % case["batch"]) // max(1, case["batch"])) for i in range(case["batch"])]


def _tokens(case, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 3)
    prompts = [torch.randint(0, _vocab(case), (n,), generator=g) for n in _lengths(case)]
    return prompts, torch.randint(0, _vocab(case), (ROOM, case["batch"]), generator=g, dtype=torch.int32)


def _observation(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed * 104729 + 5)
    if case["kind"] == "images":
        return (torch.rand(case["images"], 3, 224, 224, generator=g, device=DEV) * 2 - 1,)
    B = case["batch"]
    images = torch.rand(B, case["views"], 3, 224, 224, generator=g, device=DEV) * 2 - 1
    words = torch.randint(0, GEMMA_VOCAB, (B, 200), generator=torch.Generator().manual_seed(seed * 31 + 1))
    return images, words, torch.randn(B, HORIZON, ACTION, generator=g, device=DEV)


# ---------------------------------------------------------------------------------------------------------------- the calls
def _mixed_config(case):
    from rhinoforge_b200.models.mixed import DenseMLP, GroupedAttention, HGRN2, LatentAttention, Mamba1, MixedConfig, MixedLayer, MoE, Rotary, YarnScaling
    H, half = case["width"], case["layers"] // 2
    if case["kind"] == "latent":
        heads, rank, I = LATENT[H]
        layers = (MixedLayer(LatentAttention(heads, 128, 128, rank, 128 ** -0.5, 1024), DenseMLP(I)), MixedLayer(HGRN2(heads, 128, 128), DenseMLP(I))) * half
        return MixedConfig("latent", MIXED_VOCAB, H, 1e-6, layers, 128)
    heads, kv, ff = ROUTED[H]
    moe = MoE(16, 2, ff, 4, 2, 2 * ff)
    layers = (MixedLayer(Mamba1(2 * H, 16, H // 16, 4), moe),
              MixedLayer(GroupedAttention(heads, kv, 128, 128, 128 ** -0.5, 2048, Rotary(64, 5e5, YarnScaling(8.0, 8192, 32.0, 1.0))), moe)) * half
    return MixedConfig.zulopel("routed", MIXED_VOCAB, H, 1e-6, layers)


def _engine(case, seed):
    from rhinoforge_b200.models.decoder import DecoderConfig
    from rhinoforge_b200.runtime.engine import DecoderEngine
    from rhinoforge_b200.runtime.mixed_engine import MixedDecoderEngine
    w = _weights(_shapes(case), seed, DTYPE[case["dtype"]])
    lengths = _lengths(case)
    size = dict(dtype=DTYPE[case["dtype"]], max_batch=case["batch"], max_seq_len=(max(lengths) + ROOM + 31) // 16 * 16)
    if case["kind"] in ("latent", "routed"):
        return MixedDecoderEngine(_mixed_config(case), w.__getitem__, **size)
    if case["kind"] == "hybrid":
        H, L = case["width"], case["layers"]
        heads, kv, I = HYBRID[H]
        cfg = DecoderConfig("hybrid", MIXED_VOCAB, H, I, L, heads, kv, 128, tie_embeddings=True, norm="rms_gemma", attn_gate=True, model_type="qwen3_5",
                            layer_types=("full_attention", "linear_attention") * (L // 2), gdn_heads_k=heads, gdn_heads_v=heads, gdn_dk=128, gdn_dv=128)
        return DecoderEngine(cfg, w.__getitem__, **size)
    V, H, I, _, heads, kv, hd, eps, base, tied, qk = DECODERS[case["model"]]
    cfg = DecoderConfig(case["model"], V, H, I, case["layers"], heads, kv, hd, rms_eps=eps, rope_theta=base, tie_embeddings=tied, qk_norm=qk)
    quant = case.get("quant", "none")
    return DecoderEngine(cfg, w.__getitem__, quant=None if quant == "none" else quant, **size)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "images":
        from rhinoforge_b200.models.vision import SiglipConfig, SiglipVisionEncoder
        w = _weights(_shapes(case), seed, DTYPE[case["dtype"]])
        return {"kind": kind, "encode": SiglipVisionEncoder(SiglipConfig(), w, dtype=DTYPE[case["dtype"]], max_images=case["images"]), "pixels": _observation(case, seed)[0]}
    if kind == "action":
        from rhinoforge_b200.models.pi05 import Pi05Config, Pi05Engine
        w = _weights(_shapes(case), seed, DTYPE[case["dtype"]])
        images, words, noise = _observation(case, seed)
        B, views = case["batch"], case["views"]
        frames = torch.zeros(B, 3, 3, 224, 224, device=DEV)
        frames[:, :views] = images
        return {"kind": kind, "engine": Pi05Engine(Pi05Config(), w, dtype=DTYPE[case["dtype"]], max_batch=B), "frames": frames, "words": words, "noise": noise,
                "cameras": (torch.arange(3) < views).expand(B, 3).contiguous(), "spoken": (torch.arange(200) < case["language"]).expand(B, 200).contiguous(),
                "steps": case["steps"]}
    engine = _engine(case, seed)
    prompts, ids = _tokens(case, seed)
    if kind not in ("step", "routed"):
        return {"kind": kind, "engine": engine, "prompts": prompts}
    B = case["batch"]
    engine.prefill(prompts)
    engine.capture(B)
    held = [engine.pos, engine.kv_len, engine.step] + (engine.cache.state_tensors() if kind == "routed" else [])
    return {"kind": kind, "engine": engine, "batch": B, "ids": ids.pin_memory(), "out": torch.zeros(B, dtype=torch.int32).pin_memory(), "at": 0,
            "start": [(t, t.clone()) for t in held], "lengths": engine.cache.lengths.copy()}


def run(state):
    kind = state["kind"]
    if kind == "images":
        return state["encode"](state["pixels"])
    engine = state["engine"]
    if kind == "action":
        return engine.predict(state["frames"], state["cameras"], state["words"], state["spoken"], state["noise"], num_steps=state["steps"])
    if kind in ("step", "routed"):
        B = state["batch"]
        if state["at"] == ROOM:                # the answers are complete: back to the end of the prompts
            for t, saved in state["start"]:
                t.copy_(saved)
            engine.cache.lengths[:] = state["lengths"]
            state["at"] = 0
        engine.step_from_host(state["ids"][state["at"]], state["out"])
        state["at"] += 1
        # the step's logits, or where the engine keeps them to itself the stream they are made of and the largest one of each row
        return engine.logits[:B] if kind == "routed" else {"stream": engine.hidden[:B], "top": engine.out_vals[:B]}
    _, logits = engine.prefill(state["prompts"], return_logits=True)
    if kind == "latent":
        return {"logits": logits, "states": [t for t in engine.cache.recurrent if t is not None]}
    rows = sum(int(p.numel()) for p in state["prompts"])
    last = rows - (rows - 1) // engine.max_tokens * engine.max_tokens       # rows of the last chunk: what the stream buffer holds
    out = {"logits": logits, "stream": engine.hidden[:last]}
    if kind == "hybrid":
        out["states"] = list(engine.gdn_rec_state.values())
    return out


# ---------------------------------------------------------------------------------------------------------------- what a call needs
def _params(case):
    """(values of the matrices that every row meets, values of the head's matrix)."""
    n = sum(math.prod(s) for name, s, _ in _shapes(case) if len(s) == 2 and "embed" not in name and "head" not in name and ".e" not in name and "conv" not in name)
    return n, sum(math.prod(s) for name, s, _ in _shapes(case) if name in ("model.embed_tokens.weight", "head", "lm_head.weight", "embed")) // (
        2 if any(name in ("head", "lm_head.weight") for name, _, _ in _shapes(case)) else 1)


def work(case):
    kind = case["kind"]
    if kind in ("images", "action"):
        H, I, L, heads, _, n = VIT
        vit = L * (4 * H * H + 2 * H * I) + H * 588
        count = case["images"] if kind == "images" else case["batch"] * case["views"]
        flops = count * n * (2 * vit + 4 * n * H * L)
        if kind == "images":
            return {"bytes": BYTES * (vit + count * n * H) + 4 * count * 3 * 224 * 224, "flops": flops}
        B, rows = case["batch"], case["views"] * 256 + case["language"]
        layer = lambda w, i: w * 2048 * 2 + 2 * w * 256 + 3 * w * i
        prefix, expert = DEPTH * layer(2048, 16384), DEPTH * layer(1024, 4096)
        flops += count * 256 * 2 * 1152 * 2048 + B * rows * (2 * prefix + 4 * rows * 2048 * DEPTH)
        flops += B * case["steps"] * HORIZON * (2 * expert + 4 * (rows + HORIZON) * 2048 * DEPTH + 4 * 1024 * ACTION)
        return {"bytes": BYTES * (vit + prefix + expert + B * rows * 512 * DEPTH) + 4 * count * 3 * 224 * 224, "flops": flops}
    body, head = _params(case)
    lengths, B, L = _lengths(case), case["batch"], case["layers"]
    if kind in ("step", "prompts"):
        _, H, _, _, heads, kv, hd, _, _, _, _ = DECODERS[case["model"]]
        row, span = BYTES * 2 * kv * hd * L, 4 * heads * hd * L
    elif kind == "hybrid":
        H = case["width"]
        heads, kv, _ = HYBRID[H]
        row, span = BYTES * 2 * kv * 128 * L // 2, 4 * heads * 128 * L // 2
    elif kind == "latent":
        H = case["width"]
        row, span = BYTES * LATENT[H][1] * L // 2, 4 * LATENT[H][0] * 128 * L // 2
    else:
        H = case["width"]
        heads, kv, ff = ROUTED[H]
        row, span = BYTES * 2 * kv * 128 * L // 2, 4 * heads * 128 * L // 2
    if kind in ("step", "routed"):
        scale = {"w8a16": 0.5, "w4a16": 0.25}.get(case.get("quant"), 1.0)
        experts = 0
        if kind == "routed":       # experts that somebody picks (2 of 16 a row) are read once, every row meets two
            experts = 3 * H * ff * L
            seen = 16 * (1 - (1 - 2 / 16) ** B)
            state = 2 * 4 * B * 2 * H * 16 * L // 2
            return {"bytes": BYTES * (body + head + experts * seen) + row * (sum(lengths) + B) + state + 2 * B * head // H,
                    "flops": 2 * B * (body + head + 2 * experts) + span * sum(lengths)}
        return {"bytes": BYTES * (scale * body + (0.5 if case["quant"] == "w8a16" else 1.0) * head + 2 * B * H) + row * (sum(lengths) + B),
                "flops": 2 * B * (body + head) + span * sum(lengths)}
    T = sum(lengths)
    seen = sum(n * (n + 1) // 2 if kind != "latent" else sum(min(i + 1, 1024) for i in range(n)) for n in lengths)
    mixer = 0
    if kind in ("hybrid", "latent"):           # the recurrences: three or two products with a [128, 128] state per token and head
        mixer = T * H // 128 * (6 if kind == "hybrid" else 4) * 128 * 128 * L // 2
    return {"bytes": BYTES * (body + head + 2 * T * H + B * head // H) + row * T, "flops": 2 * T * body + 2 * B * head + span * seen + mixer}


def tolerance(case):
    # about four times the distance from exact(): 16-bit activations are rounded two dozen times on the way through a few layers.  A row whose
    # two best experts are next to equal may take the other one (once in some hundred rows in fp16), which turns a fifth of that row
    return {"rel": 0.03 if case["dtype"] == "bf16" or case["kind"] == "routed" else 0.008}


# ---------------------------------------------------------------------------------------------------------------- 64 bits
def _rms(x, eps, w=None):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _turn(x, base, dims=None, scaling=None):
    """Rotation of ``x [rows, heads, size]`` of positions 0, 1, ...: dimension i of the first ``dims`` pairs with i + dims / 2."""
    dims = dims or x.shape[-1]
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    amp = 1.0
    if scaling is not None:
        factor, original, fast, slow = scaling
        pair = lambda turns: dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(pair(fast)), 0), min(math.ceil(pair(slow)), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=torch.float64, device=x.device) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, amp = f / factor * ramp + f * (1 - ramp), 0.1 * math.log(factor) + 1
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = a.cos() * amp, a.sin() * amp
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat((u * c - v * s, v * c + u * s, x[..., dims:]), -1)


def _attend(q, k, v, scale, causal=True, window=None, sink=None):
    """``q [rows, heads, size]`` over ``k, v [keys, shared heads, size]``, blocks of 256 query rows at a time."""
    n, heads, d = q.shape
    share = heads // k.shape[1]
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    out = torch.empty(n, heads, v.shape[2], dtype=q.dtype, device=q.device)
    for a in range(0, n, 256):
        b = min(n, a + 256)
        lo, hi = (max(0, a - window + 1) if window else 0), (b if causal else k.shape[0])
        s = torch.matmul(q[a:b].view(b - a, -1, share * d).transpose(0, 1).reshape(-1, (b - a) * share, d), kk[:, :, lo:hi]) * scale
        s = s.view(-1, b - a, share, hi - lo)
        if causal:
            i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(lo, hi, device=q.device)[None]
            keep = (j <= i) if window is None else (j <= i) & (j > i - window)
            s = s.masked_fill(~keep[None, :, None], -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.view(-1, 1, share, 1).expand(-1, b - a, -1, 1)), -1)
        p = torch.softmax(s, -1)[..., :hi - lo]
        o = torch.matmul(p.reshape(-1, (b - a) * share, hi - lo), vv[:, lo:hi])
        out[a:b] = o.view(-1, b - a, share, v.shape[2]).transpose(0, 1).reshape(b - a, heads, -1)
    return out


class _Wide:
    """Tensors of ``w`` as float64 on demand, matrices with the rounding of their stored form where ``quant`` says so."""

    def __init__(self, w, quant="none", dtype=None):
        self.w, self.quant, self.dtype = w, quant, dtype

    def __contains__(self, name):
        return name in self.w

    def __getitem__(self, name):
        return self.w[name].double()

    def linear(self, x, name, head=False):
        t = self.w[name]
        if self.quant == "w8a16":
            s = (t.float().abs().amax(1).clamp(min=1e-8) / 127.0).to(self.dtype).double()[:, None]
            t = (t.float() / s.float()).round().clamp(-127, 127).double() * s
        elif self.quant == "w4a16" and not head:
            g = t.float().view(t.shape[0], -1, 64)
            s = (g.abs().amax(-1, keepdim=True) / 7.0).clamp_min(1e-8)
            t = ((g / s).round().clamp(-8, 7).double() * s.to(self.dtype).double()).view(t.shape)
        return x @ t.double().t()


def _split(x, lengths):
    return torch.split(x, lengths, 0)


def _exact_decoder(case, w, rows):
    """Residual stream behind the last layer of all rows, sequence after sequence."""
    V, H, I, _, heads, kv, hd, eps, base, _, qk = DECODERS[case["model"]]
    lengths = [int(r.numel()) for r in rows]
    x = w["model.embed_tokens.weight"][torch.cat(rows).to(DEV)]
    for i in range(case["layers"]):
        p, y = f"model.layers.{i}.", torch.empty_like(x)
        for part, seq in zip(_split(y, lengths), _split(x, lengths)):
            h = _rms(seq, eps, w[p + "input_layernorm.weight"])
            q, k, v = (w.linear(h, f"{p}self_attn.{t}_proj.weight").view(-1, n, hd) for t, n in (("q", heads), ("k", kv), ("v", kv)))
            if qk:
                q, k = _rms(q, eps, w[p + "self_attn.q_norm.weight"]), _rms(k, eps, w[p + "self_attn.k_norm.weight"])
            a = _attend(_turn(q, base), _turn(k, base), v, hd ** -0.5)
            seq = seq + w.linear(a.reshape(-1, heads * hd), p + "self_attn.o_proj.weight")
            h = _rms(seq, eps, w[p + "post_attention_layernorm.weight"])
            part.copy_(seq + w.linear(F.silu(w.linear(h, p + "mlp.gate_proj.weight")) * w.linear(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight"))
        x = y
    return x


def _conv(x, taps, bias=None):
    """Causal convolution per channel over ``x [sequences, rows, channels]``."""
    k = taps.shape[1]
    padded = F.pad(x, (0, 0, k - 1, 0))
    y = sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(k))
    return y if bias is None else y + bias


def _exact_hybrid(case, w, rows):
    H = case["width"]
    heads, kv, _ = HYBRID[H]
    lengths, B, eps = [int(r.numel()) for r in rows], case["batch"], 1e-6
    n, live = max(lengths), torch.tensor([int(r.numel()) for r in rows], device=DEV)
    x = torch.zeros(B, n, H, dtype=torch.float64, device=DEV)
    for b, r in enumerate(rows):
        x[b, :lengths[b]] = w["model.embed_tokens.weight"][r.to(DEV)]
    states = []
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps, 1 + w[p + "input_layernorm.weight"])
        if i % 2:
            a = p + "linear_attn."
            qkv = F.silu(_conv(w.linear(h, a + "in_proj_qkv.weight"), w[a + "conv1d.weight"]))
            q, k, v = (t.view(B, n, heads, 128) for t in qkv.split(heads * 128, -1))
            unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
            q, k = unit(q) * 128 ** -0.5, unit(k)
            beta = torch.sigmoid(w.linear(h, a + "in_proj_b.weight"))
            keep = torch.exp(-torch.exp(w[a + "A_log"]) * F.softplus(w.linear(h, a + "in_proj_a.weight") + w[a + "dt_bias"]))
            S, o = torch.zeros(B, heads, 128, 128, dtype=torch.float64, device=DEV), torch.empty_like(v)
            for t in range(n):
                new = S * keep[:, t, :, None, None]
                d = (v[:, t] - torch.einsum("bhkv,bhk->bhv", new, k[:, t])) * beta[:, t, :, None]
                new = new + k[:, t, :, :, None] * d[:, :, None]
                o[:, t] = torch.einsum("bhkv,bhk->bhv", new, q[:, t])
                S = torch.where((live > t)[:, None, None, None], new, S)
            states.append(S)
            o = _rms(o, eps, w[a + "norm.weight"]).reshape(B, n, -1) * F.silu(w.linear(h, a + "in_proj_z.weight"))
            x = x + w.linear(o, a + "out_proj.weight")
        else:
            a = p + "self_attn."
            qg = w.linear(h, a + "q_proj.weight").view(B, n, heads, 2, 128)
            k, v = (w.linear(h, a + t).view(B, n, kv, 128) for t in ("k_proj.weight", "v_proj.weight"))
            q, k = _rms(qg[:, :, :, 0], eps, 1 + w[a + "q_norm.weight"]), _rms(k, eps, 1 + w[a + "k_norm.weight"])
            o = torch.stack([_attend(_turn(q[b], 1e6), _turn(k[b], 1e6), v[b], 128 ** -0.5) for b in range(B)])
            x = x + w.linear((o * torch.sigmoid(qg[:, :, :, 1])).reshape(B, n, -1), a + "o_proj.weight")
        h = _rms(x, eps, 1 + w[p + "post_attention_layernorm.weight"])
        x = x + w.linear(F.silu(w.linear(h, p + "mlp.gate_proj.weight")) * w.linear(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
    last = torch.stack([x[b, lengths[b] - 1] for b in range(B)])
    return {"logits": w.linear(_rms(last, eps, 1 + w["model.norm.weight"]), "model.embed_tokens.weight"),
            "stream": torch.cat([x[b, :lengths[b]] for b in range(B)]), "states": states}


def _exact_latent(case, w, rows):
    H = case["width"]
    heads, rank, _ = LATENT[H]
    lengths, B, eps = [int(r.numel()) for r in rows], case["batch"], 1e-6
    n, live = max(lengths), torch.tensor([int(r.numel()) for r in rows], device=DEV)
    ids = torch.zeros(B, n, dtype=torch.long, device=DEV)
    for b, r in enumerate(rows):
        ids[b, :lengths[b]] = r.to(DEV)
    x, states = w["embed"][ids], []
    for i in range(case["layers"]):
        p = f"l{i}."
        h = _rms(x, eps, w[p + "norm1"])
        h = h + (F.pad(h, (0, 0, 1, 0))[:, :-1] - h) * w[p + "shift"]
        if i % 2:
            q = F.silu(w.linear(h, p + "mix.q")).view(B, n, heads, 128)
            low = w[p + "mix.lower"]
            f = (low + (1 - low) * torch.sigmoid(w.linear(h, p + "mix.f") + w[p + "mix.f.b"])).view(B, n, heads, 128)
            v = w.linear(h, p + "mix.v").view(B, n, heads, 128)
            S, o = torch.zeros(B, heads, 128, 128, dtype=torch.float64, device=DEV), torch.empty_like(v)
            for t in range(n):
                new = S * f[:, t, :, :, None] + (1 - f[:, t])[:, :, :, None] * v[:, t, :, None]
                o[:, t] = torch.einsum("bhkv,bhk->bhv", new, q[:, t])
                S = torch.where((live > t)[:, None, None, None], new, S)
            states.append(S)
            o = _rms(o, eps, w[p + "mix.norm"])
        else:
            q = w.linear(h, p + "mix.q").view(B, n, heads, 128)
            c = _rms(w.linear(h, p + "mix.dkv"), eps, w[p + "mix.dkv.norm"])
            k, v = (w.linear(c, p + t).view(B, n, heads, 128) for t in ("mix.uk", "mix.uv"))
            o = torch.stack([_attend(q[b], k[b], v[b], 128 ** -0.5, window=1024) for b in range(B)])
        x = x + w.linear(o.reshape(B, n, -1), p + "mix.o")
        x = x + w.linear(torch.relu(w.linear(_rms(x, eps, w[p + "norm2"]), p + "mlp.up")).pow(2), p + "mlp.down")
        side = F.gelu(w.linear(x, p + "side.gate"), approximate="tanh") * w["side.embed"][ids][..., i * 128:(i + 1) * 128]
        x = x + _rms(w.linear(side, p + "side.proj"), eps, w[p + "side.norm"])
    last = torch.stack([x[b, lengths[b] - 1] for b in range(B)])
    return {"logits": w.linear(_rms(last, eps, w["final.norm"]), "embed"), "states": states}


def _exact_routed(case, w, rows):
    H = case["width"]
    heads, kv, _ = ROUTED[H]
    lengths, B, eps, N = [int(r.numel()) for r in rows], case["batch"], 1e-6, 2 * H
    n = max(lengths)
    ids = torch.zeros(B, n, dtype=torch.long, device=DEV)
    for b, r in enumerate(rows):
        ids[b, :lengths[b]] = r.to(DEV)
    x = w["embed"][ids]
    glu = lambda h, e: w.linear(F.silu(w.linear(h, e + "gate")) * w.linear(h, e + "up"), e + "down")
    for i in range(case["layers"]):
        p = f"l{i}."
        if i % 2:
            q, k, v = (w.linear(x, f"{p}mix.{t}").view(B, n, m, 128) for t, m in (("q", heads), ("k", kv), ("v", kv)))
            q, k = _rms(q, eps, w[p + "mix.q.norm"]), _rms(k, eps, w[p + "mix.k.norm"])
            turn = lambda t: _turn(t, 5e5, 64, (8.0, 8192, 32.0, 1.0))
            o = torch.stack([_attend(turn(q[b]), turn(k[b]), v[b], 128 ** -0.5, sink=w[p + "mix.sink"]) for b in range(B)]).reshape(B, n, -1)
            y = w.linear(o * torch.sigmoid(w.linear(x, p + "mix.g")), p + "mix.o")
        else:
            u, z = w.linear(x, p + "mix.in").split(N, -1)
            u = F.silu(_conv(u, w[p + "mix.conv"], w[p + "mix.conv.b"]))
            dt, b_, c_ = w.linear(u, p + "mix.x").split((H // 16, 16, 16), -1)
            dt = F.softplus(w.linear(dt, p + "mix.dt") + w[p + "mix.dt.b"])
            A, S, o = -torch.exp(w[p + "mix.A_log"]), torch.zeros(B, N, 16, dtype=torch.float64, device=DEV), torch.empty_like(u)
            for t in range(n):
                S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * u[:, t])[:, :, None] * b_[:, t, None]
                o[:, t] = (S * c_[:, t, None]).sum(-1)
            y = w.linear((o + w[p + "mix.D"] * u) * F.silu(z), p + "mix.o")
        x = x + _rms(y, eps, w[p + "norm1"]) * w[p + "ls1"]
        h = x.reshape(B * n, H)
        score = torch.softmax(w.linear(h, p + "mlp.router"), -1)
        key = score + w[p + "mlp.correction"]
        best = key.view(-1, 4, 4).amax(-1).topk(2, -1).indices
        allowed = torch.zeros(h.shape[0], 4, dtype=torch.bool, device=DEV).scatter_(1, best, True).repeat_interleave(4, 1)
        picks = key.masked_fill(~allowed, -math.inf).topk(2, -1).indices
        weight = score.gather(1, picks)
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
        y = glu(h, p + "mlp.shared.")
        for e in range(16):
            row, pick = (picks == e).nonzero(as_tuple=True)
            y.index_add_(0, row, weight[row, pick, None] * glu(h[row], f"{p}mlp.e{e}."))
        x = x + _rms(y.view(B, n, H), eps, w[p + "norm2"]) * w[p + "ls2"]
    last = torch.stack([x[b, lengths[b] - 1] for b in range(B)])
    return w.linear(_rms(last, eps, w["final.norm"]), "head")


def _exact_tower(w, p, pixels):
    H, _, L, heads, patch, n = VIT
    B = pixels.shape[0]
    norm = lambda t, name: F.layer_norm(t, (H,), w[name + ".weight"], w[name + ".bias"], 1e-6)
    linear = lambda t, name: w.linear(t, name + ".weight") + w[name + ".bias"]
    x = pixels.double().reshape(B, 3, 16, patch, 16, patch).permute(0, 2, 4, 1, 3, 5).reshape(B, n, -1)
    x = x @ w[p + "embeddings.patch_embedding.weight"].reshape(H, -1).t() + w[p + "embeddings.patch_embedding.bias"] + w[p + "embeddings.position_embedding.weight"]
    for i in range(L):
        b = f"{p}encoder.layers.{i}."
        h = norm(x, b + "layer_norm1")
        q, k, v = (linear(h, f"{b}self_attn.{t}_proj").view(B, n, heads, H // heads) for t in "qkv")
        o = torch.stack([_attend(q[j], k[j], v[j], (H // heads) ** -0.5, causal=False) for j in range(B)]).reshape(B, n, H)
        x = x + linear(o, b + "self_attn.out_proj")
        x = x + linear(F.gelu(linear(norm(x, b + "layer_norm2"), b + "mlp.fc1"), approximate="tanh"), b + "mlp.fc2")
    return norm(x, p + "post_layernorm")


def _exact_action(case, w, images, words, noise):
    B, count = case["batch"], case["language"]
    seen = _exact_tower(w, VLM + "vision_tower.vision_model.", images.flatten(0, 1)) @ w[VLM + "multi_modal_projector.linear.weight"].t()
    seen = (seen + w[VLM + "multi_modal_projector.linear.bias"]).view(B, -1, 2048)
    x = torch.cat((seen, w[VLM + "language_model.embed_tokens.weight"][words[:, :count].to(DEV)] * 2048 ** 0.5), 1)
    n = x.shape[1]

    def layer(b, x, past, norm):
        """One layer over ``x``; ``norm(name, x)`` returns the normalised rows and the factor of the sublayer's output."""
        h, gate = norm("input_layernorm", x)
        q, k, v = (w.linear(h, f"{b}self_attn.{t}_proj.weight").view(B, x.shape[1], -1, 256) for t in "qkv")
        if past is not None:                   # rotations go on behind the prefix
            q, k = (torch.cat((t.new_zeros(B, n, t.shape[2], 256), t), 1) for t in (q, k))
        q, k = (torch.stack([_turn(t[j], 1e4) for j in range(B)])[:, -x.shape[1]:] for t in (q, k))
        keys, values = (k, v) if past is None else (torch.cat((past[0], k), 1), torch.cat((past[1], v), 1))
        o = torch.stack([_attend(q[j], keys[j], values[j], 1 / 16, causal=False) for j in range(B)]).reshape(B, x.shape[1], 2048)
        x = x + gate * w.linear(o, b + "self_attn.o_proj.weight")
        h, gate = norm("post_attention_layernorm", x)
        y = F.gelu(w.linear(h, b + "mlp.gate_proj.weight"), approximate="tanh") * w.linear(h, b + "mlp.up_proj.weight")
        return x + gate * w.linear(y, b + "mlp.down_proj.weight"), (k, v)

    past = []
    for i in range(DEPTH):
        b = f"{VLM}language_model.layers.{i}."
        x, kv = layer(b, x, None, lambda name, t: (_rms(t, 1e-6, 1 + w[f"{b}{name}.weight"]), 1.0))
        past.append(kv)
    a, linear = noise.double(), lambda t, name: w.linear(t, name + ".weight") + w[name + ".bias"]
    period = 4e-3 * (4.0 / 4e-3) ** torch.linspace(0, 1, 512, dtype=torch.float64, device=DEV)
    for s in range(case["steps"]):
        angle = 2 * math.pi / period * (1 - s / case["steps"])
        cond = F.silu(linear(F.silu(linear(torch.cat((angle.sin(), angle.cos())), "time_mlp_in")), "time_mlp_out"))

        def ada(name, t):
            scale, shift, gate = linear(cond, name + ".dense").chunk(3)
            return _rms(t, 1e-6) * (1 + scale) + shift, gate

        h = linear(a, "action_in_proj")
        for i in range(DEPTH):
            b = f"{EXPERT}layers.{i}."
            h, _ = layer(b, h, past[i], lambda name, t: ada(b + name, t))
        a = a - linear(ada(EXPERT + "norm", h)[0], "action_out_proj") / case["steps"]
    return a


@torch.no_grad()
def exact(case, seed):
    kind, dtype = case["kind"], DTYPE[case["dtype"]]
    w = _Wide(_weights(_shapes(case), seed, dtype), case.get("quant", "none"), dtype)
    if kind == "images":
        return _exact_tower(w, "vision_model.", _observation(case, seed)[0].to(dtype))
    if kind == "action":
        images, words, noise = _observation(case, seed)
        return _exact_action(case, w, images.to(dtype), words, noise.to(dtype))
    prompts, ids = _tokens(case, seed)
    if kind in ("step", "routed"):
        prompts = [torch.cat((p, ids[0, b:b + 1].long())) for b, p in enumerate(prompts)]
    if kind != "step" and kind != "prompts":
        return {"hybrid": _exact_hybrid, "latent": _exact_latent, "routed": _exact_routed}[kind](case, w, prompts)
    eps, tied = DECODERS[case["model"]][7], DECODERS[case["model"]][9]
    x = _exact_decoder(case, w, prompts)
    ends = torch.tensor([int(p.numel()) for p in prompts]).cumsum(0) - 1
    logits = w.linear(_rms(x[ends.to(DEV)], eps, w["model.norm.weight"]), "model.embed_tokens.weight" if tied else "lm_head.weight", head=True)
    if kind == "step":
        return {"stream": x[ends.to(DEV)], "top": logits.amax(1)}
    last = x.shape[0] - (x.shape[0] - 1) // 8192 * 8192
    return {"logits": logits, "stream": x[-last:]}
