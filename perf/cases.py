"""The work that users of this package have it do, as cases that can be timed and compared.

``listed()`` holds one case for each way the package is called in earnest, ``draw(rng)`` gives more of the same
ranges.  A case is a dict of plain values; its ``kind`` says which entry point it goes through:

    layer          WindowedAttention / BlockSparseAttention forward under ``no_grad`` (x -> y)
    layer_train    the same module forward + backward: output, gradient of the input and of every weight
    core           the attention core alone on given Q, K, V (``_native.prefill``)
    model_forward  TitanMAC forward of whole sequences (ids -> logits)
    model_train    TitanMAC forward with labels + backward: loss and the gradient of every parameter
    decode         one TitanMAC.decode_step against filled ring caches: logits and the updated rings
    generate       TitanMAC.generate: prompt, then greedy tokens
"""

import math
import os
import sys

import torch

sys.path.insert(1, os.path.join(os.getcwd(), "titanmac-standalone_b200"))

from titanmac_b200 import (BlockSparseAttention, TitanMAC, TitanMACConfig, WindowConfig, WindowedAttention,  # noqa: E402
                           _native)

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
_BLOCK = 64  # block size of the block-sparse class (its default)


def _case(kind, attention, dtype, batch, tokens, d_model, heads, window, persistent, **more):
    """``tokens`` counts sequence rows; the persistent rows come on top.  For decode it is the context length."""
    return dict(kind=kind, attention=attention, dtype=dtype, batch=batch, tokens=tokens, d_model=d_model, heads=heads,
                window=window, persistent=persistent, **more)


def listed():
    return [
        # one short sequence through one layer: nothing but launches and latency
        dict(_case("layer", "windowed", "bf16", 1, 128, 640, 10, 512, 16), name="layer_one_short_sequence"),
        # fp32, the type the module is built in by default, at the smallest benchmark configuration
        dict(_case("layer", "windowed", "fp32", 2, 512, 512, 8, 256, 16), name="layer_fp32"),
        # the default layer over a full batch of long sequences
        dict(_case("layer", "windowed", "bf16", 8, 4096, 640, 10, 512, 16), name="layer_full_batch"),
        # the other attention class (convolutions, block-granular window), a ragged length, the other 16-bit type
        dict(_case("layer", "block_sparse", "fp16", 3, 2731, 640, 10, 512, 16), name="block_sparse_ragged"),
        # training one layer of the default geometry
        dict(_case("layer_train", "windowed", "bf16", 8, 4096, 640, 10, 512, 16), name="layer_train_full_batch"),
        # long context, wide heads, attention only: what a rank of a sequence-sharded prefill runs
        dict(_case("core", "windowed", "bf16", 1, 131072, 2048, 16, 1024, 16), name="core_long_context"),
        # scoring whole sequences with the default 16-layer model
        dict(_case("model_forward", "windowed", "bf16", 2, 8192, 640, 10, 512, 16, layers=16, vocab=50000),
             name="model_long_prompt"),
        # a training step of the small experiment configuration: many small operations
        dict(_case("model_train", "block_sparse", "bf16", 8, 256, 256, 4, 64, 8, layers=4, vocab=8000),
             name="model_train_small"),
        # a training step at the default width
        dict(_case("model_train", "windowed", "bf16", 8, 1024, 640, 10, 512, 16, layers=6, vocab=50000),
             name="model_train_default_width"),
        # serving: one token for each of many sequences, the caches full
        dict(_case("decode", "windowed", "bf16", 256, 2048, 640, 10, 512, 16, layers=16, vocab=50000),
             name="decode_large_batch"),
        # serving: one token for a single sequence
        dict(_case("decode", "windowed", "bf16", 1, 700, 640, 10, 512, 16, layers=16, vocab=50000),
             name="decode_one_sequence"),
        # a handful of prompts continued greedily
        dict(_case("generate", "windowed", "bf16", 8, 300, 640, 10, 512, 16, layers=16, vocab=50000, new_tokens=48),
             name="generate_few_sequences"),
    ]


def _log_int(rng, lo, hi):
    """An integer between lo and hi, evenly over the logarithm; odd ones and powers of two alike."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layer"] * 4 + ["layer_train"] * 2 + ["core"] + ["model_forward"] * 2 + ["model_train"] * 2 +
                      ["decode"] * 3 + ["generate"])
    d_model, heads = rng.choice([(256, 4), (512, 8), (640, 10), (640, 10), (1024, 8)])  # head sizes 64 and 128
    persistent = rng.choice([0, 8, 16, 16])
    attention = rng.choice(["windowed", "windowed", "block_sparse"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    window = _log_int(rng, 64, 1024)
    if kind in ("layer", "layer_train"):
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"]) if kind == "layer" else dtype
        rows = {"layer": 32768, "layer_train": 24576}[kind] if dtype != "fp32" else 2048
        rows = rows * 640 // max(640, d_model)
        tokens = _log_int(rng, 32, min(8192, rows))
        batch = _log_int(rng, 1, max(1, min(16, rows // tokens)))
        return _case(kind, attention, dtype, batch, tokens, d_model, heads, window, persistent)
    if kind == "core":
        d_model, heads = rng.choice([(640, 10), (1024, 8), (2048, 16)])
        tokens = _log_int(rng, 4096, 131072 * 2048 // max(2048, d_model))
        return _case(kind, "windowed", dtype, 1, tokens, d_model, heads, window, persistent)
    if kind == "model_forward":
        tokens = _log_int(rng, 32, 8192)
        batch = _log_int(rng, 1, max(1, min(16, 12288 // tokens)))
        return _case(kind, attention, dtype, batch, tokens, d_model, heads, window, persistent,
                     layers=rng.randint(2, 16), vocab=rng.choice([8000, 32000, 50000]))
    if kind == "model_train":
        tokens = _log_int(rng, 64, 2048)
        batch = _log_int(rng, 1, max(1, min(16, 6144 // tokens)))
        return _case(kind, attention, "bf16", batch, tokens, d_model, heads, min(window, 512), persistent,
                     layers=rng.randint(2, 5 if attention == "block_sparse" else 6), vocab=rng.choice([8000, 32000]))
    layers, vocab = rng.randint(4, 16), rng.choice([8000, 32000, 50000])
    if kind == "decode":
        batch = _log_int(rng, 1, 256)
        return _case(kind, "windowed", dtype, batch, _log_int(rng, 32, 4096), *rng.choice([(512, 8), (640, 10)]),
                     min(window, 640), persistent, layers=layers, vocab=vocab)
    return _case(kind, "windowed", "bf16", _log_int(rng, 1, 32), _log_int(rng, 16, 512), *rng.choice([(512, 8), (640, 10)]),
                 window, persistent, layers=layers, vocab=vocab, new_tokens=rng.randint(8, 48))


# ------------------------------------------------------------------------------------------------ preparation --
def _layer(case):
    if case["attention"] == "block_sparse":
        return BlockSparseAttention(d_model=case["d_model"], n_heads=case["heads"], window_size=case["window"],
                                    block_size=_BLOCK, n_persistent=case["persistent"])
    return WindowedAttention(WindowConfig(window_size=case["window"], num_heads=case["heads"],
                                          head_dim=case["d_model"] // case["heads"], n_persistent=case["persistent"]))


def _model(case, g):
    generating = case["kind"] == "generate"
    cfg = TitanMACConfig(vocab_size=case["vocab"], d_model=case["d_model"], n_heads=case["heads"],
                         n_layers=case["layers"], d_ff=4 * case["d_model"],
                         max_seq_len=max(case["tokens"] + case.get("new_tokens", 1), case["persistent"] + 1),
                         window_size=case["window"], n_persistent=case["persistent"],
                         use_block_sparse=case["attention"] == "block_sparse", block_size=_BLOCK,
                         tie_weights=not generating)
    model = TitanMAC(cfg)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            if name.endswith("scale"):
                prm.fill_(1.0)
            elif name.endswith("bias"):
                prm.zero_()
            elif ".conv_" in name:
                prm.normal_(0.0, 0.3, generator=g)
            else:
                prm.normal_(0.0, 0.02, generator=g)
        if generating:
            # As in a trained model the next token is decided by a clear margin (random weights leave ties, which
            # any rounding decides): the residual stream stays close to the token's embedding, and the head prefers
            # the token that follows it in the vocabulary.
            model.embed_tokens.weight.normal_(0.0, 1.0, generator=g)
            model.lm_head.weight.copy_(model.embed_tokens.weight.roll(1, 0) * 0.05)
            for layer in model.layers:
                for lin in (layer.attention.out_proj, layer.mlp.fc2):
                    lin.weight.mul_((2 * case["layers"]) ** -0.5)
    return model


def prepare(case, seed):
    dev = torch.device("cuda")
    dtype = _DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    kind, B, T, D, H = case["kind"], case["batch"], case["tokens"], case["d_model"], case["heads"]
    L = T + case["persistent"]

    def normal(*shape, std=1.0):
        return torch.randn(shape, generator=g, device=dev).mul_(std).to(dtype)

    if kind == "core":
        qkv = torch.empty((B, L, 3, H, D // H), dtype=dtype, device=dev)
        for part in qkv.unbind(2):
            part.normal_(generator=g)
        return dict(case=case, qkv=tuple(t.permute(0, 2, 1, 3) for t in qkv.unbind(2)))
    with torch.device(dev):
        if kind in ("layer", "layer_train"):
            mod = _layer(case)
            with torch.no_grad():
                for name, prm in mod.named_parameters():
                    prm.normal_(0.0, 0.3 if name.startswith("conv_") else 0.02, generator=g)
        else:
            mod = _model(case, g)
    mod = mod.to(dtype=dtype)
    state = dict(case=case, mod=mod)
    if kind in ("layer", "model_forward", "decode", "generate"):
        mod.eval()
    if kind in ("layer", "layer_train"):
        state["x"] = normal(B, L, D)
        if kind == "layer_train":
            state["x"].requires_grad_(True)
            state["dy"] = normal(B, L, D)
        return state
    ids = torch.randint(0, case["vocab"], (B, T if kind != "decode" else 1), generator=g, device=dev)
    if kind == "model_train":
        state["labels"] = ids
    if kind == "decode":
        state["caches"] = mod.new_caches(B, dev, dtype)
        for cache in state["caches"]:
            for t in (cache.k_ring, cache.v_ring, cache.k_pers, cache.v_pers):
                t.normal_(0.0, 0.5, generator=g)  # keys and values as the projections of normalised rows give them
        state["pos"] = torch.full((B,), T, dtype=torch.int32, device=dev)
        ids = ids[:, 0]
    state["ids"] = ids
    return state


# -------------------------------------------------------------------------------------------------- one pass --
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "core":
        q, k, v = state["qkv"]
        return _native.prefill(q, k, v, case["window"], case["persistent"])
    mod = state["mod"]
    if kind == "layer":
        with torch.no_grad():
            return mod(state["x"])
    if kind == "model_forward":
        with torch.no_grad():
            return mod(state["ids"])["logits"]
    if kind == "decode":
        logits = mod.decode_step(state["ids"], state["pos"], state["caches"])
        return [logits] + [t for c in state["caches"] for t in (c.k_ring, c.v_ring)]
    if kind == "generate":
        return mod.generate(state["ids"], case["new_tokens"])
    mod.zero_grad(set_to_none=True)
    if kind == "layer_train":
        x = state["x"]
        x.grad = None
        y = mod(x)
        y.backward(state["dy"])
        return [y, x.grad] + [p.grad for p in mod.parameters()]
    loss = mod(state["ids"], labels=state["labels"])["loss"]
    loss.backward()
    return [loss] + [p.grad for p in mod.parameters()]


# ------------------------------------------------------------------------------------------------------ work --
def _pairs(case):
    """Visible (query, key) pairs of one sequence and head."""
    T, w, n = case["tokens"], case["window"], case["persistent"]
    if case["attention"] == "block_sparse":
        first = [max(0, b * _BLOCK - w) for b in range((T + _BLOCK - 1) // _BLOCK)]
        return sum(n + t - first[t // _BLOCK] + 1 for t in range(T)) + n * (n + T)
    ramp = min(T, w)
    return ramp * (ramp + 1) // 2 + max(0, T - w) * (w + 1) + n * T + n * n


def work(case):
    kind, B, T, D, H = case["kind"], case["batch"], case["tokens"], case["d_model"], case["heads"]
    esz = 4 if case["dtype"] == "fp32" else 2
    rows = B * (T + case["persistent"])
    core = 4.0 * D * B * _pairs(case) if kind != "decode" else 0.0  # 4 * head_dim per pair and head
    proj = 8.0 * rows * D * D
    conv = 24.0 * rows * D if case["attention"] == "block_sparse" else 0.0
    conv_w = 12 * D if case["attention"] == "block_sparse" else 0
    if kind == "core":
        return {"bytes": 4 * rows * D * esz, "flops": core}
    if kind == "layer":
        return {"bytes": (2 * rows * D + 4 * D * D + conv_w) * esz, "flops": core + proj + conv}
    if kind == "layer_train":
        # x, dy in; y, dx out; the weights and their gradients
        return {"bytes": (4 * rows * D + 2 * (4 * D * D + conv_w)) * esz, "flops": 3.5 * core + 3 * (proj + conv)}
    layers, V = case["layers"], case["vocab"]
    weights = layers * (4 * D * D + 8 * D * D + conv_w + 7 * D) + D
    head = V * D
    if kind == "model_forward":
        return {"bytes": (weights + head + B * T * V) * esz,
                "flops": layers * (core + 3 * proj + conv) + 2.0 * B * T * head}
    if kind == "model_train":
        return {"bytes": 2 * (weights + head + T * D) * esz,
                "flops": layers * (3.5 * core + 9 * proj + 3 * conv) + 6.0 * B * T * head}
    ring = 2 * D * (case["window"] + 1)  # one sequence, one layer: keys and values
    seen = 2 * D * (min(T + 1, case["window"] + 1) + case["persistent"])
    step_flops = B * (2.0 * (layers * 12 * D * D + head) + layers * 2.0 * seen)
    if kind == "decode":
        seen_bytes = 2 * D * min(T, case["window"]) * B * layers + 2 * D * case["persistent"] * layers
        return {"bytes": (weights + head + seen_bytes + 2 * D * B * layers + B * V) * esz, "flops": step_flops}
    # generate: the prompt once, then new_tokens - 1 steps that read the weights and the caches
    n = case["new_tokens"] - 1
    return {"bytes": (weights + head) * esz * (1 + n) + n * layers * B * min(seen, ring) * esz,
            "flops": layers * (core + 3 * proj) + 2.0 * B * head + n * step_flops}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"  # token ids
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    # Rounding to 16 bits: one layer, several layers, several layers there and back (measured between two attention
    # kernels and two GEMMs: 0.0033, 0.0125 and 0.017 in bf16, an eighth of that in fp16)
    rel = {"layer": 1e-2, "layer_train": 1e-2, "core": 1e-2, "model_train": 3e-2}.get(case["kind"], 2e-2)
    return {"rel": rel if case["dtype"] == "bf16" else rel / 5}
