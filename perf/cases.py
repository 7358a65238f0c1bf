"""What a user of this library has it do, as cases whose time is measured.

Families (`what` of a case):

  linear         `QMatMul.forward` on the device: one quantized linear layer over m rows of activations.
  host_linear    `QTensor.matmul_t` with host arrays: the operator boundary of an unchanged CPU engine.
  llama_decode   one greedy decode step of the dense decoder (Q4_K), a CUDA graph of `LlamaDecoder.step`.
  llama_prefill  `LlamaDecoder.prefill` of a prompt.
  moe_decode     the same step of the routed-expert decoder (`MoeDecoder`, Q8_0 attention, Q4_K experts).
  moe_prefill    `MoeDecoder.prefill` of a prompt.
  mla_decode     one step of the latent-attention decoder (`DeepseekDecoder`, IQ2_XXS experts, the rest Q8_0).
  experts        `Moe.forward_dev`: one routed-expert layer of MXFP4 banks with ids given by the caller.

Sizes are those of the benchmark configurations (bench.py) and ragged ones between them.  Weights are raw random
blocks whose scales are set so that a linear layer keeps its input's size and has weights of mean zero, as trained
weights do; activations are N(0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from joshua_b200 import synth
from joshua_b200.bench_experts import zipf_ids
from joshua_b200.deepseek import DeepseekConfig, DeepseekDecoder
from joshua_b200.llama import LlamaConfig, LlamaDecoder
from joshua_b200.moe import GATE_SOFTMAX, Moe, MoeConfig
from joshua_b200.moe_decoder import MoeDecoder, MoeDecoderConfig
from joshua_b200.qtensor import QMatMul, QTensor

TYPES = {"q8_0": synth.Q8_0, "q2_k": synth.Q2_K, "q4_k": synth.Q4_K, "iq2_xxs": synth.IQ2_XXS, "mxfp4": synth.MXFP4,
         "q6_k": synth.Q6_K}

# [rows, columns] of the linear layers of the benchmark configurations
SHAPES = [(4096, 4096), (6144, 4096), (28672, 4096), (4096, 14336), (128256, 4096), (5120, 2048), (2048, 4096),
          (1536, 7168), (24576, 1536), (7168, 16384), (2048, 7168), (7168, 2048)]

MAX_CTX = 1056  # positions the decoders' caches hold


def listed():
    return [
        # one attention projection for one token, called eagerly: the smallest call there is
        {"name": "linear_q4k_b1", "what": "linear", "type": "q4_k", "n": 4096, "k": 4096, "m": 1},
        # a small batch of sequences through a layer whose row count is no multiple of any tile
        {"name": "linear_q8_b20_ragged", "what": "linear", "type": "q8_0", "n": 6145, "k": 4096, "m": 20},
        # the output head of a mixed file: such files keep it in Q6_K while the layers are Q4_K
        {"name": "linear_q6k_head_b1", "what": "linear", "type": "q6_k", "n": 128256, "k": 4096, "m": 1},
        # a prompt of odd length through a 2-bit layer
        {"name": "linear_q2k_m333", "what": "linear", "type": "q2_k", "n": 4096, "k": 14336, "m": 333},
        # the drop-in operator with host slices on both sides
        {"name": "host_q4k_b1", "what": "host_linear", "type": "q4_k", "n": 14336, "k": 4096, "m": 1},
        # token generation for one user, and for a batch of users
        {"name": "llama_decode_b1", "what": "llama_decode", "batch": 1, "ctx": 512},
        {"name": "llama_decode_b8", "what": "llama_decode", "batch": 8, "ctx": 512},
        # reading the prompt
        {"name": "llama_prefill_512", "what": "llama_prefill", "tokens": 512},
        # the same two directions of the routed-expert model
        {"name": "moe_decode_b1", "what": "moe_decode", "batch": 1, "ctx": 128},
        {"name": "moe_prefill_1000", "what": "moe_prefill", "tokens": 1000},
        # a batch between decode and prefill on one large expert layer with skewed routing
        {"name": "experts_mxfp4_256", "what": "experts", "tokens": 256},
        # latent attention, 2-bit experts, a shared expert
        {"name": "mla_decode_b4", "what": "mla_decode", "batch": 4, "ctx": 128},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["linear"] * 5 + ["host_linear", "llama_decode", "llama_prefill", "moe_decode", "moe_prefill",
                                        "experts", "mla_decode"])
    if what in ("linear", "host_linear"):
        n, k = rng.choice(SHAPES)
        if rng.random() < 0.5:
            n = max(1, n - rng.randrange(0, min(n // 2, 1000)))  # ragged row counts
        m = _log_int(rng, 1, 1024) if what == "linear" else _log_int(rng, 1, 64)
        kind = rng.choice(sorted(TYPES))
        if n > 100000:
            m = rng.randrange(1, 17)  # the head sees the last token of each sequence only
        return {"what": what, "type": kind, "n": n, "k": k, "m": m}
    if what in ("llama_decode", "moe_decode"):
        return {"what": what, "batch": _log_int(rng, 1, 16), "ctx": _log_int(rng, 1, 1000)}
    if what in ("llama_prefill", "moe_prefill"):
        return {"what": what, "tokens": _log_int(rng, 16, 1000)}
    if what == "experts":
        return {"what": what, "tokens": _log_int(rng, 1, 4096)}
    return {"what": what, "batch": _log_int(rng, 1, 8), "ctx": _log_int(rng, 1, 1000)}


# ── inputs ──────────────────────────────────────────────────────────────
def blocks(kind, rows, cols, seed, dev):
    """Raw blocks of a [rows, cols] matrix: uniform codes and group scales, block scales such that the weights have
    mean zero and a standard deviation near 1 / sqrt(cols) (MXFP4: the benchmark's exponents)."""
    t = TYPES[kind]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    elems, nbytes = synth.BLOCK[t]
    raw = torch.randint(0, 256, (rows * (cols // elems), nbytes), dtype=torch.uint8, device=dev, generator=gen)
    if kind == "mxfp4":
        raw[:, 0] = torch.randint(118, 131, (raw.shape[0],), dtype=torch.uint8, device=dev, generator=gen)
        return raw.reshape(-1)

    def scale(offset, size, like=None):
        d = torch.empty(raw.shape[0], device=dev).uniform_(0.5, 1.5, generator=gen) * size if like is None else like
        raw[:, offset:offset + 2] = d.to(torch.float16).view(torch.uint8).reshape(-1, 2)
        return d.to(torch.float16).float()

    std = 1.0 / math.sqrt(cols)
    if kind == "q8_0":
        raw[:, 2:][raw[:, 2:] == 128] = 129  # codes in [-127, 127]
        scale(0, std / 73)
    elif kind == "q4_k":  # minima = 7.5 x scales, the middle of the codes
        raw[:, 8:12] = raw[:, 4:8]
        raw[:, 12:16] = (raw[:, 12:16] & 15) * 17
        d = scale(0, std / 168)
        scale(2, 0, like=d * 7.5)
    elif kind == "q2_k":  # minima = 1.5 x scales
        raw[:, :16] = (raw[:, :16] & 15) * 17
        d = scale(80, std / 9.8)
        scale(82, 0, like=d * 1.5)
    elif kind == "iq2_xxs":
        scale(0, std / 67)
    elif kind == "q6_k":
        scale(208, std / 1370)
    return raw.reshape(-1)


def _tensor(kind, rows, cols, seed, dev):
    t = TYPES[kind]
    raw = torch.cat([blocks(kind, rows, cols, seed, dev), torch.zeros(16, dtype=torch.uint8, device=dev)])
    return QTensor.from_device(t, raw[:synth.tensor_bytes(t, rows, cols)])


def _randn(shape, seed, dev):
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32)


def _router(cfg, seed):
    """Scores with a standard deviation of 4: the first experts of a token take most of the weight, the last of the
    chosen ones about a hundredth, so that two experts in a near tie may change places without much effect."""
    gen = np.random.default_rng(seed)
    return (gen.standard_normal((cfg.n_expert, cfg.hidden), dtype=np.float32) * (4.0 / math.sqrt(cfg.hidden)))


def _warm_graph(model, restore):
    """The decode step as a CUDA graph, as a serving loop keeps it."""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        model.step()
        restore()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            model.step()
        restore()
        stream.synchronize()
    return graph


def _decode_state(model, case, seed, dev, vocab):
    batch, ctx = case["batch"], case["ctx"]
    for i, ly in enumerate(model.layers):
        ly["k"].normal_(generator=torch.Generator(device=dev).manual_seed(seed * 131 + 2 * i))
        ly["v"].normal_(generator=torch.Generator(device=dev).manual_seed(seed * 131 + 2 * i + 1))
    token = torch.randint(0, vocab, (batch,), generator=torch.Generator().manual_seed(seed), dtype=torch.int32).to(dev)
    pos = torch.full((batch,), ctx, dtype=torch.int32, device=dev)

    def restore():
        model.token.copy_(token)
        model.pos.copy_(pos)

    restore()
    return {"case": case, "model": model, "token": token, "pos": pos, "graph": _warm_graph(model, restore)}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    what = case["what"]
    if what in ("linear", "host_linear"):
        n, k, m = case["n"], case["k"], case["m"]
        w = _tensor(case["type"], n, k, seed * 1009 + 1, dev)
        x = _randn((m, k), seed * 1009 + 2, dev)
        if what == "linear":
            return {"case": case, "linear": QMatMul(w, n, k), "x": x}
        return {"case": case, "w": w, "x": x.cpu().numpy()}
    if what in ("llama_decode", "llama_prefill"):
        cfg = LlamaConfig()
        model = LlamaDecoder(cfg, dev, batch=case.get("batch", 1), max_ctx=MAX_CTX, seed=seed,
                             weights=lambda name, n, k, s: blocks("q4_k", n, k, s, dev))
    elif what in ("moe_decode", "moe_prefill"):
        cfg = MoeDecoderConfig()
        model = MoeDecoder(cfg, dev, batch=case.get("batch", 1), max_ctx=MAX_CTX, seed=seed, qk_norm=True,
                           weights=lambda name, n, k, s: blocks("q8_0", n, k, s, dev),
                           expert_weights=lambda name, n, k, s: blocks("q4_k", n, k, s + seed, dev),
                           routers=lambda layer: _router(cfg, seed * 97 + layer))
    elif what == "mla_decode":
        cfg = DeepseekConfig()
        names = {v: k for k, v in TYPES.items()}
        model = DeepseekDecoder(cfg, dev, batch=case["batch"], max_ctx=MAX_CTX, seed=seed,
                                weights=lambda name, t, n, k, s: blocks(names[t], n, k, s, dev))
    else:
        experts, used, hidden, inter, tokens = 384, 8, 7168, 2048, case["tokens"]
        banks = [_tensor("mxfp4", experts * r, c, seed * 1009 + i, dev)
                 for i, (r, c) in enumerate([(inter, hidden), (inter, hidden), (hidden, inter)])]
        rng = np.random.default_rng(seed)
        router = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
        layer = Moe(MoeConfig(gating=GATE_SOFTMAX, n_expert=experts, n_used=used, hidden=hidden, inter=inter), router,
                    *banks)
        layer.reserve(tokens, tokens * used)
        ids = zipf_ids(tokens, rng, np.random.default_rng(7).permutation(experts))
        return {"case": case, "layer": layer, "x": _randn((tokens, hidden), seed * 1009 + 5, dev).bfloat16().float(),
                "ids": torch.from_numpy(ids.astype(np.int32)).to(dev), "y": torch.empty(tokens, hidden, device=dev)}
    if what.endswith("prefill"):
        ids = torch.randint(0, cfg.vocab, (case["tokens"],), generator=torch.Generator().manual_seed(seed),
                            dtype=torch.int32)
        return {"case": case, "model": model, "ids": ids}
    return _decode_state(model, case, seed, dev, cfg.vocab)


def run(state):
    what = state["case"]["what"]
    if what == "linear":
        return state["linear"].forward(state["x"])
    if what == "host_linear":
        c = state["case"]
        return state["w"].matmul_t((c["m"], c["k"], c["n"]), state["x"])
    if what == "experts":
        state["layer"].forward_dev(state["x"], state["y"], forced_ids=state["ids"])
        return state["y"]
    model = state["model"]
    if what.endswith("prefill"):
        model.pos.zero_()
        model.prefill(state["ids"])
        if what == "moe_prefill":
            # behind the first router a near tie may go either way: one token's rows of the caches then differ
            return {"logits": model.logits, "k": model.layers[0]["k"], "v": model.layers[0]["v"]}
        return {"logits": model.logits, "token": model.token, "k": model.layers[-1]["k"], "v": model.layers[-1]["v"]}
    model.token.copy_(state["token"])
    model.pos.copy_(state["pos"])
    state["graph"].replay()
    if what == "moe_decode":
        return model.logits
    return {"logits": model.logits, "token": model.token}


# ── what a pass cannot do without ───────────────────────────────────────
def _tb(kind, rows, cols):
    return synth.tensor_bytes(TYPES[kind], rows, cols)


def work(case):
    """Bytes: weights once (of a bank: the experts that are touched), inputs and outputs once, cached positions once.
    flops: two per weight and row, and the attention products."""
    what = case["what"]
    if what in ("linear", "host_linear"):
        n, k, m = case["n"], case["k"], case["m"]
        return {"bytes": _tb(case["type"], n, k) + 4 * m * (n + k), "flops": 2 * m * n * k}
    if what == "experts":
        hidden, inter, t = 7168, 2048, case["tokens"]
        rng = np.random.default_rng(1)
        touched = len(np.unique(zipf_ids(t, rng, np.random.default_rng(7).permutation(384))))
        return {"bytes": touched * 3 * _tb("mxfp4", inter, hidden) + 8 * t * hidden,
                "flops": 2 * t * 8 * 3 * hidden * inter}
    decode = what.endswith("decode")
    rows = case["batch"] if decode else case["tokens"]
    # positions a row attends to, summed over the rows; cached positions read (decode) or written (prefill)
    seen = rows * (case["ctx"] + 1) if decode else rows * (rows + 1) // 2
    cached = seen if decode else rows
    heads_out = case["batch"] if decode else 1
    if what.startswith("llama"):
        c = LlamaConfig()
        per_layer = _tb("q4_k", c.qkv_rows, c.hidden) + _tb("q4_k", c.hidden, c.q_heads * c.head_dim) + \
            2 * _tb("q4_k", c.ffn, c.hidden) + _tb("q4_k", c.hidden, c.ffn)
        weights = c.hidden * (c.qkv_rows + c.q_heads * c.head_dim + 3 * c.ffn)
        head = _tb("q4_k", c.vocab, c.hidden)
        kv, att = 2 * c.kv_heads * c.head_dim, 4 * c.q_heads * c.head_dim
    elif what.startswith("moe"):
        c = MoeDecoderConfig()
        touched = c.n_expert * (1 - (1 - c.n_used / c.n_expert) ** rows)
        per_expert = 2 * _tb("q4_k", c.moe_inter, c.hidden) + _tb("q4_k", c.hidden, c.moe_inter)
        per_layer = _tb("q8_0", c.qkv_rows, c.hidden) + _tb("q8_0", c.hidden, c.q_heads * c.head_dim) + \
            touched * per_expert + 4 * c.n_expert * c.hidden
        weights = c.hidden * (c.qkv_rows + c.q_heads * c.head_dim + c.n_used * 3 * c.moe_inter + c.n_expert)
        head = _tb("q8_0", c.vocab, c.hidden)
        kv, att = 2 * c.kv_heads * c.head_dim, 4 * c.q_heads * c.head_dim
    else:
        c = DeepseekConfig()
        touched = c.n_expert * (1 - (1 - c.n_used / c.n_expert) ** rows)
        dense = [(c.q_lora, c.hidden), (c.n_head * c.qd, c.q_lora), (c.kv_lora + c.qk_rope, c.hidden),
                 (c.n_head * (c.qk_nope + c.v_dim), c.kv_lora), (c.hidden, c.n_head * c.v_dim), (c.moe_inter, c.hidden),
                 (c.moe_inter, c.hidden), (c.hidden, c.moe_inter)]
        per_expert = 2 * _tb("iq2_xxs", c.moe_inter, c.hidden) + _tb("iq2_xxs", c.hidden, c.moe_inter)
        per_layer = sum(_tb("q8_0", n, k) for n, k in dense) + touched * per_expert + 4 * c.n_expert * c.hidden
        weights = sum(n * k for n, k in dense) + c.hidden * (c.n_used * 3 * c.moe_inter + c.n_expert)
        head = _tb("q8_0", c.vocab, c.hidden)
        kv, att = c.n_head * (c.qd + c.v_dim), 2 * c.n_head * (c.qd + c.v_dim)
    return {"bytes": c.layers * (per_layer + 4 * kv * cached) + head + 4 * heads_out * c.vocab,
            "flops": c.layers * (2 * rows * weights + att * seen) + 2 * heads_out * c.vocab * c.hidden}


def tolerance(case):
    """About four times what the default kernels and the exact-decode float kernels (JQ_FORCE_F32_PATH=1, the same
    sums in another order) were seen to differ by: single layers 3e-7 to 1.2e-6, the dense and latent-attention models
    2.5e-6 to 7.2e-6, the routed-expert model 1.4e-5 to 6e-4 (its router turns a rounding difference into one of the
    expert weights, and two experts in a near tie may change places)."""
    what = case["what"]
    if what in ("linear", "host_linear", "experts"):
        return {"rel": 5e-6}
    return {"rel": 3e-3 if what.startswith("moe") else 3e-5}
