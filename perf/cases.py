"""The work a user of this package has it do, as cases that can be timed.

Four kinds of work, all through the package's public entry points:

* ``linear``  one call of a ``runtime.TexelatorLinear`` -- the module ``runtime.install`` puts in the place
  of an ``nn.Linear``: one token (decode), a few tokens (batched decode, speculative checks), short and
  long prompts; bf16 and fp16; with and without bias; both palettes; dense and pruned weights; the prefill
  kernel an applied profile selected, or (``backend`` 0) the handle as ``install`` leaves it without one.
* ``encode``  a dense matrix to BC4 blocks and scales, as a conversion does it once per projection.
* ``step``    one decoded token per sequence through a captured decoder (one sequence or a batch).
* ``prompt``  a prompt through a decoder, filling its cache.

Matrix shapes are those of ``modeling.CONFIGS`` (hidden 2048, 5120 and 8192), tensor-parallel shares of
them, and ragged ones.  Models keep a configuration's widths, heads and vocabulary; the number of layers is
cut so that a state is made quickly and so that rounding differences do not grow past what one layer's
data types explain (a random-init stack amplifies them from layer to layer).
"""
from __future__ import annotations

import dataclasses
import math
import sys

import torch

from texelator_b200 import modeling, runtime
from texelator_b200.batched import BatchedBC4Decoder


# ---- the cases ------------------------------------------------------------------------------------------

def _linear(name, tokens, m, k, backend=5, dtype="bf16", bias=False, palette="software", pruned=False):
    case = {"kind": "linear", "tokens": tokens, "m": m, "k": k, "backend": backend, "dtype": dtype, "bias": bias,
            "palette": palette, "pruned": pruned}
    return {"name": name, **case} if name else case


def _model(name, kind, model, layers, batch, context):
    case = {"kind": kind, "model": model, "layers": layers, "batch": batch, "context": context}
    return {"name": name, **case} if name else case


def listed():
    return [
        # the smallest projection of the 2048-wide model: a key projection of one decoded token
        _linear("decode_kv_256x2048", 1, 256, 2048, bias=True),
        # the largest matrix a decoded token meets: fused gate and up of the 5120-wide model
        _linear("decode_gate_up_34816x5120", 1, 34816, 5120),
        # a converted checkpoint run in fp16, encoded against the measured texture palette
        _linear("decode_fp16_texture_5120x17408", 1, 5120, 17408, dtype="fp16", palette="hardware"),
        # eight sequences (or draft tokens) in one call
        _linear("decode8_5120x17408", 8, 5120, 17408),
        # a ragged, pruned matrix and an odd number of prompt tokens: low-mode blocks, partial tiles
        _linear("prompt29_pruned_4250x2896", 29, 4250, 2896, backend=8, pruned=True),
        # a prompt on a model that was installed without applying a tuning profile
        _linear("prompt160_untuned_11008x2048", 160, 11008, 2048, backend=0, bias=True),
        # a prompt of usual length through the down projection
        _linear("prompt512_5120x17408", 512, 5120, 17408, backend=9),
        # a long prompt through the widest projection
        _linear("prompt4096_34816x5120", 4096, 34816, 5120, backend=5),
        # converting one square projection
        {"name": "encode_4096x4096", "kind": "encode", "m": 4096, "k": 4096},
        # chat with the 2048-wide model: one token of one sequence
        _model("step1_2048wide", "step", "qwen2.5-3b-shaped", 6, 1, 1500),
        # serving: one token for each of sixteen sequences of the 5120-wide model
        _model("step16_5120wide", "step", "27b-class", 4, 16, 1000),
        # reading a prompt with the 2048-wide model
        _model("prompt700_2048wide", "prompt", "qwen2.5-3b-shaped", 6, 1, 700),
    ]


_LARGEST = 4096 * 34816 * 5120


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _matrix(rng):
    """A projection of one of the configurations (or a two- or four-way share of its rows), or a ragged matrix."""
    if rng.random() < 0.3:
        return _log_int(rng, 200, 20000), 16 * _log_int(rng, 16, 1100)
    c = modeling.CONFIGS[rng.choice(["qwen2.5-3b-shaped", "27b-class", "70b-class"])]
    m, k = rng.choice([(c.q_rows + 2 * c.kv_rows, c.hidden), (c.kv_rows, c.hidden), (c.hidden, c.q_rows),
                       (2 * c.intermediate, c.hidden), (c.intermediate, c.hidden), (c.hidden, c.intermediate)])
    return m // rng.choice([1, 1, 2, 4]), k


def draw(rng):
    kind = rng.choice(["linear"] * 7 + ["encode", "step", "prompt"])
    if kind == "encode":
        return {"kind": kind, "m": _log_int(rng, 100, 12000), "k": 16 * _log_int(rng, 16, 700)}
    if kind != "linear":
        model = rng.choice(["qwen2.5-3b-shaped", "27b-class", "70b-class"])
        layers = rng.randint(2, 6) if model == "qwen2.5-3b-shaped" else rng.randint(1, 3)
        if kind == "prompt":
            return _model("", kind, model, layers, 1, _log_int(rng, 20, 2000))
        return _model("", kind, model, layers, rng.choice([1, 1, _log_int(rng, 2, 32)]), _log_int(rng, 40, 4000))
    m, k = _matrix(rng)
    tokens = rng.choice([1, 1, rng.randint(2, 15), _log_int(rng, 16, 200), _log_int(rng, 200, 4096)])
    tokens = max(1, min(tokens, _LARGEST // (m * k)))
    # what an applied profile selects for this many tokens; without a profile only short prompts are usual
    tuned = rng.choice([8, 7] if tokens <= 64 else [7, 9] if tokens <= 256 else [5, 9, 6])
    backend = 0 if tokens <= 256 and rng.random() < 0.3 else tuned
    return _linear("", tokens, m, k, backend, rng.choice(["bf16", "bf16", "fp16"]), rng.random() < 0.3,
                   rng.choice(["software", "software", "hardware"]), rng.random() < 0.15)


# ---- what a program has in hand -----------------------------------------------------------------------------

class _Owned:
    """Device handles that are given back with the state that uses them."""

    def __init__(self, handles):
        self.handles = handles

    def __del__(self):
        if not sys.is_finalizing():
            runtime.free(self.handles)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weight(m, k, gen, pruned=False):
    """Gaussian rows of different magnitude; ``pruned`` zeroes nine weights of ten, which is what makes blocks whose
    endpoints meet (the palette's second mode)."""
    w = torch.randn(m, k, device="cuda", generator=gen) * (0.01 + 0.02 * torch.rand(m, 1, device="cuda", generator=gen))
    if pruned:
        w *= torch.rand(m, k, device="cuda", generator=gen) < 0.1
    return w


def _moments(k, gen):
    """Second moments of the input columns, a few of them large, as calibration finds them."""
    return torch.exp(0.5 * torch.randn(k, device="cuda", generator=gen)) * (1 + 30 * (torch.rand(k, device="cuda", generator=gen) < 0.005))


def _prepare_linear(case, seed):
    gen, ext = _generator(seed), runtime.extension()
    m, k = case["m"], case["k"]
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float16
    hardware = case["palette"] == "hardware"
    table = ext.hardware_palette().cuda().reshape(255, 255, 8) if hardware else modeling.software_palette_table("cuda")
    moments = _moments(k, gen)
    blocks, scales = ext.encode(_weight(m, k, gen, case["pruned"]), moments, table)
    bias = (torch.randn(m, device="cuda", generator=gen) * 0.1).to(dtype) if case["bias"] else None
    handle = ext.pack_encoded_device(blocks, scales, bias)
    ext.set_lookahead(handle, 3)
    ext.set_palette(handle, runtime.PALETTE_HARDWARE if hardware else runtime.PALETTE_SOFTWARE)
    ext.set_prefill(handle, runtime.PREFILL_THRESHOLD, runtime.PREFILL_TILE_ROWS)
    ext.set_prefill_backend(handle, case["backend"])
    x = (torch.randn(case["tokens"], k, device="cuda", generator=gen) * moments.sqrt()).to(dtype)
    return {"module": runtime.TexelatorLinear([handle]), "x": x, "owner": _Owned([handle])}


def _decoder(case, seed, max_len):
    config = dataclasses.replace(modeling.CONFIGS[case["model"]], layers=case["layers"])
    if case["batch"] == 1:
        return modeling.BC4Decoder(config, "cuda", max_len=max_len, seed=seed, encoder="e3")
    return BatchedBC4Decoder(config, "cuda", max_len=max_len, batch=case["batch"], seed=seed, encoder="e3")


def _prepare_step(case, seed):
    gen = _generator(seed + 1)
    batch, context = case["batch"], case["context"]
    model = _decoder(case, seed, context + 64)
    ids = torch.randint(0, model.config.vocab, (batch, context), device="cuda", generator=gen)
    if batch == 1:
        model.prefill(ids[0])
    else:
        for sequence in range(batch):                   # contexts of different length, as a server has them
            model.fill_context(sequence, 0, context - (sequence * 37) % (context // 2), seed=seed)
        model.tune_decode_kernel()
    tokens, positions = ids[:, -1].contiguous(), model.pos.clone()
    model.tok.copy_(tokens)
    model.capture()
    return {"model": model, "tokens": tokens, "positions": positions, "owner": _Owned(model.handles)}


def _prepare_prompt(case, seed):
    model = _decoder(case, seed, case["context"] + 64)
    ids = torch.randint(0, model.config.vocab, (case["context"],), device="cuda", generator=_generator(seed + 1))
    return {"model": model, "ids": ids, "owner": _Owned(model.handles)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        return {"kind": kind, **_prepare_linear(case, seed)}
    if kind == "encode":
        gen = _generator(seed)
        return {"kind": kind, "weight": _weight(case["m"], case["k"], gen), "moments": _moments(case["k"], gen),
                "table": modeling.software_palette_table("cuda")}
    return {"kind": kind, **(_prepare_step if kind == "step" else _prepare_prompt)(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "encode":
        return runtime.extension().encode(state["weight"], state["moments"], state["table"])
    model = state["model"]
    if kind == "prompt":
        return [model.prefill(state["ids"]), model.k_cache, model.v_cache]
    # the token each sequence continues with and its position, then the captured step; which token follows is left
    # out of the outputs: random-init logits tie in bf16 too often to compare a single arg-max
    model.tok.copy_(state["tokens"])
    model.pos.copy_(state["positions"])
    model.decode_graph()
    return [model.last_hidden, model.k_cache, model.v_cache]


# ---- what a pass cannot do without -----------------------------------------------------------------------------

def work(case):
    if case["kind"] == "linear":
        t, m, k = case["tokens"], case["m"], case["k"]
        return {"bytes": m * k // 2 + 4 * m + (2 * m if case["bias"] else 0) + 2 * t * (m + k), "flops": 2 * t * m * k}
    if case["kind"] == "encode":
        # ten palettes per weight: the nearest entry (about six operations) and its weighted squared error (four)
        m, k = case["m"], case["k"]
        return {"bytes": 4 * m * k + m * k // 2 + 4 * m + 4 * k, "flops": 100 * m * k}
    c = dataclasses.replace(modeling.CONFIGS[case["model"]], layers=case["layers"])
    weights = c.layers * c.hidden * (2 * c.q_rows + 2 * c.kv_rows + 3 * c.intermediate)
    batch, context = case["batch"], case["context"]
    if case["kind"] == "prompt":
        cache = 2 * c.layers * context * c.kv_rows
        return {"bytes": c.bc4_bytes_per_token() + 2 * cache + 4 * context * c.hidden,
                "flops": 2 * context * weights + 2 * c.layers * c.q_rows * context * context}
    if batch == 1:
        keys = context
    else:
        keys = sum(context - (sequence * 37) % (context // 2) for sequence in range(batch))
    head = c.vocab * c.hidden
    return {"bytes": c.bc4_bytes_per_token() + 2 * head + 4 * c.layers * keys * c.kv_rows + 4 * batch * c.hidden,
            "flops": 2 * batch * (weights + head) + 4 * c.layers * keys * c.q_rows}


def tolerance(case):
    if case["kind"] == "encode":
        return "exact"
    if case["kind"] == "linear":
        # one rounding of each output (2^-9 or 2^-12 of it at most) plus the weights' own, which an implementation
        # may round to the activations' type
        return {"rel": 5e-3, "max": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 5e-3}
    # several bf16 roundings per layer, carried along the residual stream: the same stack with its sums in another order
    # (PyTorch ops between the linears, another decode or prefill kernel) ends 1.2 to 1.9 percent away after 4 to 8 layers
    return {"rel": 2.5e-2, "max": 2.5e-1}
