"""What a user of this framework has it do, as measurable cases: action chunks of the whole pi0 model through
``NativePi0`` (device-resident and host tensors, both operand formats, the smallest to the largest observation) and the
stand-alone operators of which such a model is made.

A case is a dict of plain values; ``kind`` says which entry point it goes through:

* ``pi0``        ``NativePi0.forward`` on CUDA tensors, or ``NativePi0.sample_actions`` on pinned host tensors
* ``linear``     ``ResidentNVFP4``: NVFP4 projection with a fused epilogue
* ``dense``      ``ResidentDense``: BF16 or FP8 projection
* ``attention``  ``ResidentAttention``: multi-query (Gemma) and multi-head (SigLIP) attention with KV splits
* ``norm``       ``ResidentNorm``: LayerNorm / RMSNorm into the format of the projection behind it
"""
import math
import sys
from collections import OrderedDict
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "pizero-megakernel_b200"))
from native_pi0.attention import ResidentAttention                      # noqa: E402
from native_pi0.dense import ResidentDense                              # noqa: E402
from native_pi0.model import NativePi0                                  # noqa: E402
from native_pi0.normalization import ResidentNorm                       # noqa: E402
from native_pi0.primitives import ResidentNVFP4                         # noqa: E402
from native_pi0.quantization import PackedNVFP4                         # noqa: E402
from native_pi0.weights import Pi0Config, StateDictModel, random_state_dict  # noqa: E402

WORKERS = 148
# (N, K) of the model's projections: SigLIP q|k|v, out, fc1, fc2; Gemma-2B q|k|v, o, gate/up, down; action expert the same
PROJECTIONS = ((3456, 1152), (1152, 1280), (4352, 1152), (1152, 4352), (2560, 2048), (2048, 2048), (32768, 2048), (2048, 16384),
               (2560, 1024), (1024, 2048), (8192, 1024), (1024, 4096))


# ------------------------------------------------------------------------------------------------------------- cases
def pi0(name, views, prompt, chunk, steps, precision="nvfp4", host=False):
    return _named(name, kind="pi0", views=views, prompt=prompt, chunk=chunk, steps=steps, precision=precision, host=host)


def linear(name, rows, n, k, out, act="none", block_n=128, residual=False):
    return _named(name, kind="linear", rows=rows, n=n, k=k, out=out, act=act, block_n=block_n, residual=residual)


def dense(name, rows, n, k, dtype, out="bf16", bias=False, residual=False):
    return _named(name, kind="dense", rows=rows, n=n, k=k, dtype=dtype, out=out, bias=bias, residual=residual)


def attention(name, batch, queries, keys, heads, kv_heads, head_dim, splits=1, prefix=-1):
    return _named(name, kind="attention", batch=batch, queries=queries, keys=keys, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                  splits=splits, prefix=prefix)


def norm(name, rows, width, norm_kind, out):
    return _named(name, kind="norm", rows=rows, width=width, norm=norm_kind, out=out)


def _named(name, **case):
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # the benchmark's configuration: three cameras, no prompt, 50 actions, ten Euler steps, inputs on the device
        pi0("chunk of 50, 3 views", 3, 0, 50, 10),
        # a serving process: pinned host tensors in, host actions out, a 16-token prompt, 63 actions
        pi0("served chunk of 63", 3, 16, 63, 10, host=True),
        # the smallest observation: one camera, a short odd prompt, ten actions, five Euler steps
        pi0("chunk of 10, 1 view", 1, 9, 10, 5),
        # the largest: a full-length prompt and a long chunk (more than 64 expert rows, ragged prefix bands)
        pi0("chunk of 100, prompt 48", 3, 48, 100, 10),
        # the accuracy-first operand format of the same model
        pi0("chunk of 50 in bf16", 3, 0, 50, 10, precision="bf16"),
        # Gemma-2B gate/up with GeGLU for a 768-row prefix: the largest projection of the model
        linear("gate/up of 768 rows", 768, 32768, 2048, "fp4", "geglu"),
        # the action expert's q|k|v: few rows, latency
        linear("expert qkv of 51 rows", 51, 2560, 1024, "bf16", block_n=64),
        # a BF16 projection of ragged size
        dense("bf16 333 x 1000 x 1152", 333, 1000, 1152, "bf16", bias=True),
        # the Gemma-2B down projection on FP8 operands
        dense("fp8 down of 768 rows", 768, 2048, 16384, "fp8"),
        # prefix attention over three views and a 16-token prompt: more tiles than SMs
        attention("prefix attention 784", 1, 784, 784, 8, 1, 256, splits=4),
        # the action expert's queries over the cached prefix
        attention("expert attention 51 x 819", 1, 51, 819, 8, 1, 256, splits=13, prefix=768),
        # a norm in front of the expert's projections: the smallest call
        norm("rms norm 51 x 1024", 51, 1024, "rms", "fp4"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("pi0", "pi0", "linear", "linear", "dense", "attention", "attention", "norm"))
    if kind == "pi0":
        views, steps, host = rng.randint(1, 3), rng.choice((4, 5, 8, 10, 10)), rng.random() < 0.4
        if rng.random() < 0.25:
            return pi0(None, views, 0, rng.randint(8, 50), steps, "bf16", host)
        return pi0(None, views, rng.randint(0, 48), rng.randint(8, 100), steps, "nvfp4", host)
    if kind == "linear":
        rows = _log(rng, 1, 820)
        n, k = rng.choice(PROJECTIONS)
        out, act = rng.choice((("bf16", "none"), ("bf16", "none"), ("fp4", "gelu"), ("fp4", "geglu"), ("fp4", "none"), ("f32", "none")))
        if act == "geglu" and n % 256:
            act = "gelu"
        return linear(None, rows, n, k, out, act, 64 if rows <= 128 else 128, out == "bf16" and rng.random() < 0.5)
    if kind == "dense":
        dtype = rng.choice(("bf16", "bf16", "fp8"))
        return dense(None, _log(rng, 1, 820), _log(rng, 100, 4400), _log(rng, 500, 4400) // 8 * 8, dtype,
                     "f32" if rng.random() < 0.2 else "bf16", rng.random() < 0.5, rng.random() < 0.3)
    if kind == "attention":
        where = rng.choice(("vision", "prefix", "expert"))
        if where == "vision":
            return attention(None, rng.randint(1, 3), rng.randint(196, 256), rng.randint(196, 256), 16, 16, 72)
        if where == "prefix":
            rows = rng.randint(256, 820)
            return attention(None, 1, rows, rows, 8, 1, 256, splits=-(-rows // 256))
        queries, prefix = rng.randint(9, 101), rng.randint(256, 820)
        return attention(None, 1, queries, prefix + queries, 8, 1, 256, splits=min(13, (prefix + queries) // 32), prefix=prefix)
    return norm(None, _log(rng, 1, 820), rng.randint(16, 128) * 16, rng.choice(("rms", "layer")), rng.choice(("fp4", "fp4", "bf16", "fp8")))


# ----------------------------------------------------------------------------------------------------------- prepare
_checkpoint = []                 # one set of weights per process, as a serving process loads one checkpoint
_packed = {}                     # ... packed once per operand format, shared by the engines of all shapes
_engines = OrderedDict()         # the engines of the shapes seen last


def _model():
    """pi0 at full depth and width with random weights.  Matrices are N(0, 0.02) as in the benchmark; the ones that
    write to the residual stream are divided by the depth of their tower, because in a trained network every layer
    changes the stream by a few percent.  (Undivided, each layer replaces it, and the rounding of a single 4-bit code
    grows to a tenth of the result.)"""
    if not _checkpoint:
        config = Pi0Config()
        weights = random_state_dict(config, seed=0, device="cuda")
        for name, value in weights.items():
            if name.endswith((".out_proj.weight", ".fc2.weight")):
                value.div_(config.vision_layers)
            elif name.endswith((".o_proj.weight", ".down_proj.weight")):
                value.div_(config.expert_layers if "gemma_expert" in name else config.prefix_layers)
        _checkpoint.append(StateDictModel(config, weights))
    return _checkpoint[0]


def _engine(case):
    key = tuple(case[k] for k in ("views", "prompt", "chunk", "steps", "precision"))
    if key not in _engines:
        _engines[key] = NativePi0(_model(), num_views=case["views"], prompt_len=case["prompt"], chunk_size=case["chunk"],
                                  flow_steps=case["steps"], precision=case["precision"], weight_store=_packed.setdefault(case["precision"], {}))
    _engines.move_to_end(key)
    while len(_engines) > 3:
        _engines.popitem(last=False)
    return _engines[key]


def _codes(generator, rows, k, global_scale):
    """An NVFP4 matrix of uniform E2M1 codes and block scales between 0.25 and 1.5, times ``global_scale``."""
    return PackedNVFP4(generator.integers(0, 256, size=(rows, k // 2), dtype=np.uint8),
                       generator.integers(40, 61, size=(rows, k // 16), dtype=np.uint8), np.float32(global_scale), (rows, k))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")      # noqa: E731
    if case["kind"] == "pi0":
        engine = _engine(case)
        inputs = (torch.rand(case["views"], 224, 224, 3, generator=g, device="cuda") * 2 - 1, randn(1, engine.config.action_dim),
                  randn(1, case["chunk"], engine.config.action_dim),
                  torch.randint(0, engine.config.vocab, (1, case["prompt"]), generator=g, device="cuda"))
        if case["host"]:
            inputs = tuple(t.cpu().pin_memory() for t in inputs)
        return engine.sample_actions if case["host"] else engine.forward, inputs, None
    if case["kind"] == "linear":
        rng = np.random.default_rng(seed)
        padded = -(-case["rows"] // 128) * 128
        residual = randn(padded, case["n"]) if case["residual"] else None
        op = ResidentNVFP4(None, _codes(rng, padded, case["k"], 1.0), _codes(rng, case["n"], case["k"], 0.01), workers=WORKERS,
                           output_dtype={"f32": torch.float32, "bf16": torch.bfloat16, "fp4": torch.uint8}[case["out"]],
                           output_gelu=case["act"] == "gelu", output_geglu=case["act"] == "geglu", residual=residual,
                           block_n=case["block_n"], rows=case["rows"], tiled_weight=case["k"] % 256 == 0)
        return op.forward, (), op
    if case["kind"] == "dense":
        dtype = {"bf16": torch.bfloat16, "fp8": torch.float8_e4m3fn}[case["dtype"]]
        op = ResidentDense(None, randn(case["rows"], case["k"]).to(dtype), randn(case["n"], case["k"]).to(dtype),
                           alpha=0.02, bias=randn(case["n"]) if case["bias"] else None,
                           residual=randn(case["rows"], case["n"]) if case["residual"] and case["out"] == "bf16" else None,
                           output_dtype=torch.float32 if case["out"] == "f32" else torch.bfloat16, workers=WORKERS)
        return op.forward, (), op
    if case["kind"] == "attention":
        hd = case["head_dim"]
        stored = 128 if hd == 72 else hd                    # SigLIP's heads lie 128 elements apart, zeros behind them
        heads = lambda rows, count: torch.nn.functional.pad(randn(case["batch"], rows, count, hd), (0, stored - hd)).bfloat16()    # noqa: E731
        q, k, v = heads(case["queries"], case["heads"]), heads(case["keys"], case["kv_heads"]), heads(case["keys"], case["kv_heads"])
        tiles = case["batch"] * -(-case["queries"] // 128) * case["heads"] * case["splits"]
        op = ResidentAttention(None, q, k, v, workers=WORKERS, prefix=None if case["prefix"] < 0 else case["prefix"], splits=case["splits"],
                               fused_merge=case["splits"] > 1 and tiles <= WORKERS, head_dim=hd)
        return op.forward, (), op
    layer = case["norm"] == "layer"
    op = ResidentNorm(None, randn(case["rows"], case["width"]).bfloat16(), kind=case["norm"], precision=case["out"],
                      gamma=1 + 0.1 * randn(case["width"]), beta=0.1 * randn(case["width"]) if layer else None, workers=WORKERS, row_alignment=128)
    return op.forward, (), op


# --------------------------------------------------------------------------------------------------------------- run
def run(state):
    call, inputs, op = state
    out = call(*inputs)
    scales = getattr(op, "output_scales", None)
    return out if scales is None else (out, scales)         # NVFP4: packed codes and block scales


# -------------------------------------------------------------------------------------------------------------- work
def _pi0_work(case):
    c, weight = Pi0Config(), 9 / 16 if case["precision"] == "nvfp4" else 2          # bytes per weight: 4 bits and a scale byte per 16
    vision_rows, prefix_rows, expert_rows = case["views"] * 256, case["views"] * 256 + case["prompt"], case["chunk"] + 1
    kv = 2 * c.head_dim
    vision = c.vision_layers * (4 * c.vision_width ** 2 + 2 * c.vision_width * c.vision_mlp) + c.vision_width * c.width
    gemma = lambda width, mlp: 2 * width * c.heads * c.head_dim + width * kv + 3 * width * mlp          # noqa: E731
    prefix = (c.prefix_layers - 1) * gemma(c.width, c.mlp) + c.width * kv           # the last layer only fills its cache
    expert = c.expert_layers * gemma(c.expert_width, c.expert_mlp)
    heads = 2 * c.expert_width ** 2 + 2 * c.expert_width * c.action_dim             # time MLP and action projections, FP32
    attend = lambda q, k, count, dim: 4 * q * k * count * dim                       # noqa: E731
    flops = 2 * (vision_rows * (vision + 588 * c.vision_width) + prefix_rows * prefix + case["steps"] * expert_rows * (expert + heads))
    flops += c.vision_layers * case["views"] * attend(256, 256, c.vision_heads, c.vision_width // c.vision_heads)
    flops += (c.prefix_layers - 1) * attend(prefix_rows, prefix_rows, c.heads, c.head_dim)
    flops += case["steps"] * c.expert_layers * attend(expert_rows, prefix_rows + expert_rows, c.heads, c.head_dim)
    read = weight * (vision + prefix + expert) + 4 * (heads + 588 * c.vision_width)
    return read + case["views"] * 224 * 224 * 3 * 4 + 2 * case["chunk"] * c.action_dim * 4, flops


def work(case):
    size = {"f32": 4, "bf16": 2, "fp8": 1, "fp4": 9 / 16}
    if case["kind"] == "pi0":
        read, flops = _pi0_work(case)
    elif case["kind"] in ("linear", "dense"):
        rows, n, k = case["rows"], case["n"], case["k"]
        operand = size["fp4"] if case["kind"] == "linear" else size[case["dtype"]]
        columns = n // 2 if case.get("act") == "geglu" else n
        read = operand * (rows + n) * k + size[case["out"]] * rows * columns + (2 * rows * n if case["residual"] else 0)
        flops = 2 * rows * n * k
    elif case["kind"] == "attention":
        q = case["batch"] * case["queries"] * case["heads"] * case["head_dim"]
        kv = case["batch"] * case["keys"] * case["kv_heads"] * case["head_dim"]
        read, flops = 2 * (2 * q + 2 * kv), 4 * q * case["keys"]
    else:
        values = case["rows"] * case["width"]
        read, flops = values * (2 + size[case["out"]]), 8 * values
    return {"bytes": read, "flops": flops}


# --------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case):
    if case["kind"] == "pi0":
        # a sum in another order now and then moves an activation to the next 4-bit code, which eighteen layers and ten
        # steps carry to 1.5 to 2 % of the actions; in BF16 the same differences stay at 0.2 %
        return {"rel": 0.03, "max": 0.15} if case["precision"] == "nvfp4" else {"rel": 0.01, "max": 0.05}
    if case.get("out") == "f32":
        return {"rel": 2e-5, "max": 1e-3}
    if case.get("out") == "fp4":
        return {"rel": 0.0, "differ": 0.005}                # codes next to the middle between two values
    if case.get("out") == "fp8":
        return {"rel": 0.02, "max": 0.13, "differ": 0.005}
    return {"rel": 0.01, "max": 0.05}
