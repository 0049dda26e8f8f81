"""Performance cases of the inference runtime, measured through the entry points a program calls: `ExecutionEngine.run`,
`run_host`, `decode_static` (with and without `last_row_only`) and `decode_cached`.

The models are the ones this repository is configured, tested and benchmarked with: the 16-layer MLP of width 512, the
4-layer GPT of width 256, the GPT-2-small shape, the 6 + 6 layer encoder-decoder and ResNet-50.  Weights are fixed per
model (a program loads one model file and feeds it many inputs); token ids, features, images, masks and prompts come from
the seed.  A state is one engine with the inputs of one call: building it is what a program pays when it loads the model.
"""
from __future__ import annotations

import math
import os
from collections import OrderedDict

import numpy as np
import torch

from fxfusion_b200 import lowering, wire
from fxfusion_b200.engine import ExecutionEngine

MLP_OUT = 10
GPT = {"gpt_c2": lowering.GPT_C2, "gpt2_small": lowering.GPT2_SMALL}
ENCDEC = lowering.TRANSFORMER_C4


def listed():
    return [
        # MLP scoring of one request: the smallest call, sixteen dependent layers over a single row.
        {"name": "mlp_b1", "model": "mlp", "call": "run", "precision": "auto", "batch": 1, "depth": 16, "width": 512},
        # The benchmark's MLP configuration, batch 32.
        {"name": "mlp_b32", "model": "mlp", "call": "run", "precision": "auto", "batch": 32, "depth": 16, "width": 512},
        # Bulk scoring with the last, incomplete batch of a data set: many rows, not a multiple of any tile.
        {"name": "mlp_b1500", "model": "mlp", "call": "run", "precision": "auto", "batch": 1500, "depth": 16, "width": 512},
        # The benchmark's small GPT: one forward over batch 8 x 64 positions.
        {"name": "gpt_c2_b8_t64", "model": "gpt_c2", "call": "run", "precision": "auto", "batch": 8, "seq": 64},
        # The small GPT decoding to the loop's default static length of 50 with the projection on the read row only.
        {"name": "gpt_c2_lastrow_b3_t50", "model": "gpt_c2", "call": "decode_last_row", "precision": "auto", "batch": 3, "seq": 50, "steps": 33},
        # Scoring a few documents of an odd length: prefill whose rows and keys are ragged.
        {"name": "gpt2_forward_b5_t197", "model": "gpt2_small", "call": "run", "precision": "auto", "batch": 5, "seq": 197},
        # The headline: full-recompute greedy decode at batch 32, static length 256 (the last 8 tokens of it).
        {"name": "gpt2_decode_b32_t256", "model": "gpt2_small", "call": "decode_static", "precision": "auto", "batch": 32, "seq": 256, "steps": 8},
        # The reduced-precision option on a medium batch.
        {"name": "gpt2_bf16_b16_t256", "model": "gpt2_small", "call": "run", "precision": "bf16", "batch": 16, "seq": 256},
        # Incremental decode with cached keys and values: 255 single-position forwards.
        {"name": "gpt2_cached_b32_t256", "model": "gpt2_small", "call": "decode_cached", "precision": "auto", "batch": 32, "seq": 256, "steps": 128},
        # The benchmark's encoder-decoder: 64 pairs of 256 + 256 positions.
        {"name": "encdec_b64_s256_t256", "model": "encdec", "call": "run", "precision": "auto", "batch": 64, "src": 256, "seq": 256},
        # The benchmark's image classification batch.
        {"name": "resnet50_b256", "model": "resnet50", "call": "run", "precision": "auto", "batch": 256, "image": 224},
        # One image from a request handler: host buffer in, host logits out.
        {"name": "resnet50_host_b1", "model": "resnet50", "call": "run_host", "precision": "auto", "batch": 1, "image": 224},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "gpt_forward", "gpt_forward", "gpt_decode", "gpt_cached", "encdec", "resnet50"])
    if kind == "mlp":
        return {"model": "mlp", "call": rng.choice(["run", "run", "run_host"]), "precision": rng.choice(["auto", "auto", "bf16"]), "batch": _log_int(rng, 1, 2048),
                "depth": rng.randint(4, 16), "width": rng.choice([256, 512, 1024])}
    if kind == "gpt_forward":
        return {"model": rng.choice(["gpt_c2", "gpt2_small"]), "call": "run", "precision": rng.choice(["auto", "auto", "bf16"]), "batch": _log_int(rng, 1, 32),
                "seq": _log_int(rng, 16, 256)}
    if kind == "gpt_decode":
        seq = _log_int(rng, 32, 256)
        return {"model": rng.choice(["gpt_c2", "gpt2_small"]), "call": rng.choice(["decode_static", "decode_last_row"]), "precision": "auto",
                "batch": _log_int(rng, 1, 32), "seq": seq, "steps": rng.randint(2, 8)}
    if kind == "gpt_cached":
        seq = _log_int(rng, 32, 256)
        return {"model": rng.choice(["gpt_c2", "gpt2_small"]), "call": "decode_cached", "precision": "auto", "batch": _log_int(rng, 1, 32), "seq": seq,
                "steps": rng.randint(seq // 4, seq // 2)}
    if kind == "encdec":
        return {"model": "encdec", "call": "run", "precision": "auto", "batch": _log_int(rng, 1, 64), "src": _log_int(rng, 16, 256), "seq": _log_int(rng, 16, 256)}
    return {"model": "resnet50", "call": rng.choice(["run", "run_host"]), "precision": "auto", "batch": _log_int(rng, 1, 128), "image": rng.choice([160, 192, 224])}


# ---- model files -------------------------------------------------------------------------------------------------------
def _transformer_like(shapes, pe_keys, pe):
    """N(0, 0.02) matrices, zero biases, unit LayerNorms, made on the GPU from a fixed seed (163 M values for GPT-2-small)."""
    gen = torch.Generator(device="cuda").manual_seed(0)
    out = {}
    for key, shape in shapes.items():
        if key.endswith(".b"):
            out[key] = np.zeros(shape, np.float32)
        elif ".ln" in key or key.startswith("ln"):
            out[key] = np.ones(shape, np.float32)
        else:
            out[key] = torch.empty(shape, device="cuda").normal_(0.0, 0.02, generator=gen).cpu().numpy()
    for key in pe_keys:
        out[key] = pe
    return out


def _gpt_params(cfg):
    D, F, V = cfg.d_model, cfg.d_ff, cfg.vocab
    shapes = {"emb": (V, D), "head.w": (V, D), "head.b": (V,), "ln_f.w": (D,), "ln_f.b": (D,)}
    for l in range(cfg.layers):
        for key, n_out, n_in in (("qkv", 3 * D, D), ("wo", D, D), ("ff1", F, D), ("ff2", D, F)):
            shapes[f"l{l}.{key}.w"], shapes[f"l{l}.{key}.b"] = (n_out, n_in), (n_out,)
        for key in ("ln1", "ln2"):
            shapes[f"l{l}.{key}.w"], shapes[f"l{l}.{key}.b"] = (D,), (D,)
    return _transformer_like(shapes, ["pe"], lowering.sinusoidal_pe(cfg.pe_len, D))


_PARAMS = {}              # weights of the model used last
_FILES = OrderedDict()    # serialised graphs used last, as anonymous in-memory files


def _params(case):
    model = case["model"]
    key = (model, case.get("depth"), case.get("width"))
    if key not in _PARAMS:
        _PARAMS.clear()
        if model == "mlp":
            _PARAMS[key] = lowering.mlp_params(case["depth"], case["width"], MLP_OUT, seed=0)
        elif model == "encdec":
            _PARAMS[key] = lowering.transformer_params(ENCDEC, 0)
        elif model == "resnet50":
            _PARAMS[key] = lowering.resnet50_params(0)
        else:
            _PARAMS[key] = _gpt_params(GPT[model])
    return _PARAMS[key]


def _graph_path(case):
    model, nb = case["model"], case["batch"]
    key = (model, nb, case.get("seq"), case.get("src"), case.get("image"), case.get("depth"), case.get("width"), case["call"] == "decode_cached")
    if key in _FILES:
        return f"/proc/self/fd/{_FILES[key]}"
    while len(_FILES) >= 2:
        os.close(_FILES.popitem(last=False)[1])
    p = _params(case)
    if model == "mlp":
        g = lowering.mlp_graph(p, batch=nb)
    elif model == "encdec":
        g = lowering.transformer_graph(ENCDEC, p, batch=nb, src_len=case["src"], tgt_len=case["seq"])
    elif model == "resnet50":
        g = lowering.resnet50_graph(p, batch=nb, image=case["image"])
    elif case["call"] == "decode_cached":
        g = lowering.gpt_step_graph(GPT[model], p, batch=nb, max_len=case["seq"])
    else:
        g = lowering.gpt_graph(GPT[model], p, batch=nb, seq=case["seq"])
    fd = os.memfd_create(model)
    wire.dump(g, f"/proc/self/fd/{fd}")
    _FILES[key] = fd
    return f"/proc/self/fd/{fd}"


# ---- states ------------------------------------------------------------------------------------------------------------
def _causal(nb, T):
    return torch.ones(T, T, dtype=torch.bool, device="cuda").tril().view(1, 1, T, T).expand(nb, 1, T, T).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    model, nb, call = case["model"], case["batch"], case["call"]

    def ids(n, vocab):   # id 0 is the pad id
        return torch.randint(1, vocab, (nb, n), generator=gen, device="cuda")

    state = {"call": call, "engine": ExecutionEngine(_graph_path(case), "cuda:0", precision=case["precision"])}
    if model == "mlp":
        state["inputs"] = [torch.randn(nb, case["width"], generator=gen, device="cuda")]
    elif model == "encdec":
        S, T = case["src"], case["seq"]
        state["inputs"] = [ids(S, ENCDEC.vocab), ids(T, ENCDEC.vocab), torch.ones(nb, 1, 1, S, dtype=torch.bool, device="cuda"), _causal(nb, T)]
    elif model == "resnet50":
        state["inputs"] = [torch.randn(nb, 3, case["image"], case["image"], generator=gen, device="cuda")]
    elif call == "run":
        state["inputs"] = [ids(case["seq"], GPT[model].vocab), _causal(nb, case["seq"])]
    else:
        T = case["seq"]
        state["prompt_len"] = T - case["steps"]
        tokens = torch.zeros(nb, T, dtype=torch.int64, device="cuda")
        tokens[:, :state["prompt_len"]] = ids(state["prompt_len"], GPT[model].vocab)
        state["tokens"] = tokens
    if call == "run_host":   # a request handler keeps pinned host buffers for what comes in and what goes out
        state["pinned"] = [t.cpu().pin_memory() for t in state.pop("inputs")]
        descs = state["engine"].output_descs
        state["out"] = [torch.empty([d.shape[i] for i in range(d.rank)], dtype=torch.float32).pin_memory() for d in descs]
        state["host_in"], state["host_out"] = [t.numpy() for t in state["pinned"]], [t.numpy() for t in state["out"]]
    return state


def run(state):
    engine, call = state["engine"], state["call"]
    if call == "run":
        return engine.run(state["inputs"])
    if call == "run_host":
        engine.run_host(state["host_in"], state["host_out"])
        return state["out"]
    if call == "decode_cached":
        return engine.decode_cached(state["tokens"], state["prompt_len"])
    return engine.decode_static(state["tokens"], state["prompt_len"], last_row_only=call == "decode_last_row")


# ---- work --------------------------------------------------------------------------------------------------------------
def _dense(rows, n_in, n_out):
    return 2.0 * rows * n_in * n_out


def _gpt_forward_flops(cfg, nb, T, head_rows):
    M, D, F = nb * T, cfg.d_model, cfg.d_ff
    layer = _dense(M, D, 3 * D) + 4.0 * nb * T * T * D + _dense(M, D, D) + 2.0 * _dense(M, D, F)
    return cfg.layers * layer + _dense(head_rows, D, cfg.vocab)


def work(case):
    """Operations of the call as its contract states them (full recompute per decode step; one position per incremental
    step) and the bytes of weights, inputs and outputs, each once per forward."""
    model, nb, call = case["model"], case["batch"], case["call"]
    if model == "mlp":
        weights = case["width"] ** 2 * (case["depth"] - 1) + case["width"] * MLP_OUT
        return {"bytes": 4.0 * (weights + nb * (case["width"] + MLP_OUT)), "flops": 2.0 * nb * weights}
    if model == "resnet50":
        h = case["image"]
        flops, weights, c_in = 0.0, 0.0, 64

        def conv(n_out, n_in, k, side):
            nonlocal flops, weights
            flops += 2.0 * nb * side * side * n_out * n_in * k * k
            weights += n_out * n_in * k * k

        h = (h - 1) // 2 + 1
        conv(64, 3, 7, h)
        h = (h - 1) // 2 + 1
        for width, blocks, stride in lowering.RESNET50_LAYERS:
            for b in range(blocks):
                out = (h - 1) // (stride if b == 0 else 1) + 1
                conv(width, c_in, 1, h)
                conv(width, width, 3, out)
                conv(4 * width, width, 1, out)
                if b == 0:
                    conv(4 * width, c_in, 1, out)
                h, c_in = out, 4 * width
        flops += _dense(nb, c_in, 1000)
        weights += c_in * 1000
        return {"bytes": 4.0 * (weights + nb * (3 * case["image"] ** 2 + 1000)), "flops": flops}
    if model == "encdec":
        D, F, V, S, T = ENCDEC.d_model, ENCDEC.d_ff, ENCDEC.vocab, case["src"], case["seq"]
        Ms, Mt = nb * S, nb * T
        enc = _dense(Ms, D, 4 * D) + 4.0 * nb * S * S * D + 2.0 * _dense(Ms, D, F)
        dec = _dense(Mt, D, 6 * D) + _dense(Ms, D, 2 * D) + 4.0 * nb * T * (T + S) * D + 2.0 * _dense(Mt, D, F)
        weights = ENCDEC.enc_layers * (4 * D * D + 2 * D * F) + ENCDEC.dec_layers * (8 * D * D + 2 * D * F) + V * D
        return {"bytes": 4.0 * (weights + (Ms + Mt) * D + Mt * V) + 8.0 * (Ms + Mt) + nb * (S + T * T),
                "flops": ENCDEC.enc_layers * enc + ENCDEC.dec_layers * dec + _dense(Mt, D, V)}
    cfg, T = GPT[model], case["seq"]
    D, V = cfg.d_model, cfg.vocab
    weights = cfg.layers * (4 * D * D + 2 * D * cfg.d_ff) + V * D
    if call == "decode_cached":   # T - 1 positions; position p attends over p + 1 keys
        per_pos = cfg.layers * (_dense(nb, D, 4 * D) + 2.0 * _dense(nb, D, cfg.d_ff))
        keys = cfg.layers * nb * D * T * (T - 1) / 2.0
        return {"bytes": 4.0 * (weights * (T - 1) + 2.0 * keys + case["steps"] * nb * V), "flops": per_pos * (T - 1) + 4.0 * keys + case["steps"] * _dense(nb, D, V)}
    head_rows = nb if call == "decode_last_row" else nb * T
    steps = 1 if call == "run" else case["steps"]
    return {"bytes": steps * (4.0 * (weights + nb * T * D + head_rows * V) + 8.0 * nb * T + nb * T * T), "flops": steps * _gpt_forward_flops(cfg, nb, T, head_rows)}


def tolerance(case):
    """fp32 results: products of 21 bits or more and 32-bit sums through the depth of the network.  The bf16 option rounds
    both factors of every product.  Decoded tokens are whole numbers that may differ where two logits are tied to rounding,
    and then to the end of that sequence."""
    if case["call"] in ("decode_static", "decode_last_row", "decode_cached"):
        return {"rel": 0.0, "differ": 0.01}
    if case["precision"] == "bf16":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 4e-5, "max": 1e-3}
