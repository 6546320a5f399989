"""What a user of this package has it do, as cases that can be timed one by one.

A case is a dict of plain values; ``kind`` says which public entry points a pass goes through:

* ``layer``       one attention layer over the scale schedule of one generated image batch, as the attention hook runs it:
                  a new ``LayerKV`` (``kv_caching(True)``), then one ``step`` per scale -- quantize and append K and V, attend
                  the scale's queries over everything cached.  ``route`` "step" takes q and k already L2-normalised in fp32 and
                  v in bf16; "normalised" takes the raw bf16 QKV activation through ``step_normalised``, which is what
                  ``hooks.install`` puts into a module.
* ``drop_in``     the same schedule through the reference's own call, ``use_var_q`` for K and for V (fp32 caches out), without a
                  capacity hint: what the unedited attention hooks call.
* ``round_trip``  quantize + pack one K and one V tensor and dequantise them again (``quant``, ``dequant_current``).
* ``attend``      attention of Lq queries over a cache that is already there (``attend_cached``).

Batch sizes are images; classifier-free guidance doubles them.  Inputs are synthetic: activations ~N(0, 1) with a few large
channels, as the K / V of these models show, unit-length q and k rows where the model normalises them.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("var-q_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from VAR_Q.attention import attend_cached  # noqa: E402
from VAR_Q.hooks import LayerKV  # noqa: E402
from VAR_Q.quant import VAR_Q  # noqa: E402

# patch sides of the scale schedules: 256 px and 512 px VAR, the 1024 px Infinity schedule and its shorter prefixes
SCHEDULES = {
    "256px": (1, 2, 3, 4, 5, 6, 8, 10, 13, 16),
    "512px": (1, 2, 3, 4, 6, 9, 13, 18, 24, 32),
    "1024px": (1, 2, 4, 6, 8, 12, 16, 20, 24, 32, 40, 48, 64),
    "640px": (1, 2, 4, 6, 8, 12, 16, 20, 24, 32, 40),
    "320px": (1, 2, 4, 6, 8, 12, 16, 20),
}
# per K / V settings: bits, method, options
SETTINGS = {
    "int8_dim": (8, "G_SCALE_HEAD_DIM", {}),                                     # the shipped configurations of both models
    "int4_dim_asym": (4, "G_SCALE_HEAD_DIM", {"symmetric": False}),
    "int8_head": (8, "G_TOKEN_HEAD", {}),
    "int4_head": (4, "G_TOKEN_HEAD", {}),
    "int2_head": (2, "G_TOKEN_HEAD", {}),
    "int4_head_asym": (4, "G_TOKEN_HEAD", {"symmetric": False}),
    "int8_group32": (8, "G_TOKEN_HEAD", {"symmetric": False, "group_size": 32}),
    "int4_group32": (4, "G_TOKEN_HEAD", {"symmetric": False, "group_size": 32}),
    "int2_group32": (2, "G_TOKEN_HEAD", {"symmetric": False, "group_size": 32}),
    "int8_token": (8, "G_TOKEN", {}),
}
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
Q_GAIN = 4.0            # exp of the models' initial per-head query scale


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one image at a time, the interactive use: ten tiny steps per layer, latency and launches
        dict(name="layer 256px, 1 image", kind="layer", route="step", schedule="256px", h_div_w=1.0, images=1, heads=16, head_dim=64,
             fmt="BLHc", k="int8_head", v="int8_head"),
        # the VAR-d16 job of the benchmark: batch 32, INT8 per head
        dict(name="layer 256px, 32 images", kind="layer", route="step", schedule="256px", h_div_w=1.0, images=32, heads=16, head_dim=64,
             fmt="BLHc", k="int8_head", v="int8_head"),
        # the shipped VAR configuration (INT8 per dim, batch_size 50) through the installed hook: raw bf16 QKV in
        dict(name="layer 256px, 50 images, shipped", kind="layer", route="normalised", schedule="256px", h_div_w=1.0, images=50, heads=16,
             head_dim=64, fmt="BLHc", k="int8_dim", v="int8_dim"),
        # the VAR-d30 job of the benchmark: 30 heads, K per dim and V per head in asymmetric INT4
        dict(name="layer 512px, 64 images", kind="layer", route="step", schedule="512px", h_div_w=1.0, images=64, heads=30, head_dim=64,
             fmt="BLHc", k="int4_dim_asym", v="int4_head_asym"),
        # Infinity, one prompt: the user waits for this one
        dict(name="layer 1024px, 1 image", kind="layer", route="step", schedule="1024px", h_div_w=1.0, images=1, heads=16, head_dim=128,
             fmt="BHLc", k="int4_group32", v="int2_group32"),
        # the Infinity-2B job of the benchmark, its headline workload
        dict(name="layer 1024px, 8 images", kind="layer", route="step", schedule="1024px", h_div_w=1.0, images=8, heads=16, head_dim=128,
             fmt="BHLc", k="int4_group32", v="int2_group32"),
        # Infinity with the shipped settings at another aspect ratio: step lengths that are no squares and no multiples of anything
        dict(name="layer 640px 3:2, 3 images, shipped", kind="layer", route="normalised", schedule="640px", h_div_w=1.5, images=3, heads=16,
             head_dim=128, fmt="BHLc", k="int8_dim", v="int8_dim"),
        # the reference's hook unedited: fp32 caches come back at every scale, the cache grows without a hint
        dict(name="drop-in 256px, 8 images", kind="drop_in", schedule="256px", h_div_w=1.0, images=8, heads=16, head_dim=64,
             fmt="BLHc", k="int8_dim", v="int8_dim"),
        # quantize + pack + dequantise K and V of a whole 256px history: per-head asymmetric INT4
        dict(name="round trip 16x680, int4", kind="round_trip", batch=16, tokens=680, heads=16, head_dim=64, fmt="BHLc",
             k="int4_head_asym", v="int4_head_asym", dtype="fp32"),
        # the isolated attention sweep of the benchmark: a single query per (sample, head), bound by the packed cache ...
        dict(name="attend 1 query, 10521 tokens", kind="attend", batch=64, heads=16, head_dim=128, lq=1, lk=10521, fmt="BHLc",
             k="int4_head", v="int4_head", q_dtype="bf16"),
        # ... and some hundred queries, group-wise INT2
        dict(name="attend 256 queries, 10521 tokens", kind="attend", batch=64, heads=16, head_dim=64, lq=256, lk=10521, fmt="BHLc",
             k="int2_group32", v="int2_group32", q_dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges, no dearer than the dearest listed one."""
    top = [work(c) for c in listed()]
    most_bytes, most_flops = max(w["bytes"] for w in top), max(w["flops"] for w in top)
    while True:
        kind = rng.choice(("layer", "layer", "layer", "layer", "layer", "drop_in", "round_trip", "attend", "attend"))
        head_dim = rng.choice((64, 128))
        case = {"kind": kind, "heads": rng.choice((16, 16, 20, 24, 30)), "head_dim": head_dim}
        if kind in ("layer", "drop_in"):
            case["schedule"] = rng.choice(("256px", "512px") if head_dim == 64 else ("320px", "640px", "1024px"))
            case["h_div_w"] = rng.choice((1.0, 1.0, 1.0, 0.5, 0.75, 1.25, 1.5, 2.0)) if head_dim == 128 else 1.0
            case["images"] = _log_int(rng, 1, 64 if kind == "layer" else 32)
            case["fmt"] = "BLHc" if head_dim == 64 else "BHLc"
            case["k"], case["v"] = rng.choice((
                ("int8_dim", "int8_dim"), ("int8_head", "int8_head"), ("int4_dim_asym", "int4_head_asym"), ("int4_group32", "int2_group32"),
                ("int4_head", "int4_head"), ("int8_token", "int8_token"), ("int8_group32", "int4_group32")))
            if kind == "layer":
                case["route"] = rng.choice(("step", "normalised"))
        elif kind == "round_trip":
            case["batch"], case["tokens"] = _log_int(rng, 1, 128), _log_int(rng, 16, 4096)
            case["fmt"] = rng.choice(("BLHc", "BHLc"))
            case["dtype"] = rng.choice(("fp32", "bf16", "fp16"))
            case["k"] = rng.choice(("int8_dim", "int8_head", "int4_dim_asym", "int4_head_asym", "int4_group32", "int8_token"))
            case["v"] = rng.choice(("int8_dim", "int8_head", "int4_head_asym", "int2_group32"))
        else:
            case["batch"], case["lq"], case["lk"] = _log_int(rng, 1, 64), _log_int(rng, 1, 4096), _log_int(rng, 256, 10521)
            case["fmt"] = "BHLc"
            case["k"] = case["v"] = rng.choice(("int8_head", "int4_head", "int2_head", "int8_group32", "int4_group32", "int2_group32"))
            case["q_dtype"] = rng.choice(("bf16", "bf16", "fp16", "fp32"))
        w = work(case)
        if w["bytes"] <= most_bytes and w["flops"] <= most_flops:
            return case


# ------------------------------------------------------------------------------------------------ inputs
def _step_lengths(case):
    r = math.sqrt(case["h_div_w"])
    return [max(1, round(p * r)) * max(1, round(p / r)) for p in SCHEDULES[case["schedule"]]]


def _shape(fmt, b, l, h, d):
    return (b, l, h, d) if fmt == "BLHc" else (b, h, l, d)


def _activation(shape, gen, gain=6.0):
    """fp32 ~N(0, 1) with the first four channels ``gain`` times larger."""
    x = torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda")
    x[..., :4] *= gain
    return x


def _unit_rows(x):
    return x / torch.linalg.vector_norm(x, dim=-1, keepdim=True).clamp_min_(1e-12)


def _kwargs(name):
    bits, method, options = SETTINGS[name]
    return dict(quant_bits=bits, quant_method=method, **options)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, fmt, H, D = case["kind"], case["fmt"], case["heads"], case["head_dim"]
    state = dict(case)
    if kind in ("layer", "drop_in"):
        b = 2 * case["images"]
        steps = []
        for l in _step_lengths(case):
            if kind == "layer" and case["route"] == "normalised":
                # the fused QKV activation of the layer; q, k, v are views of it
                qkv = _activation((b, l, 3, H, D), gen).to(torch.bfloat16)
                q, k, v = qkv.unbind(dim=2)
                if fmt == "BHLc":
                    q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
                steps.append((q, k, v))
                continue
            k = _unit_rows(_activation(_shape(fmt, b, l, H, D), gen))
            v = _activation(_shape(fmt, b, l, H, D), gen).to(torch.bfloat16)
            if fmt == "BLHc":           # v stays a third of the fused activation, as the hook receives it
                qkv = torch.empty((b, l, 3, H, D), dtype=torch.bfloat16, device="cuda")
                qkv[:, :, 2] = v
                v = qkv[:, :, 2]
            q = _unit_rows(_activation(_shape(fmt, b, l, H, D), gen)).mul_(Q_GAIN) if kind == "layer" else None
            steps.append((q, k, v))
        state["steps"] = steps
        state["tokens"] = sum(_step_lengths(case))
        state["scale_mul"] = torch.full((1, 1, H, 1), Q_GAIN, device="cuda")
        state["k_kwargs"], state["v_kwargs"] = _kwargs(case["k"]), _kwargs(case["v"])
    elif kind == "round_trip":
        b, l, dtype = case["batch"], case["tokens"], DTYPES[case["dtype"]]
        state["k_item"], state["v_item"] = (_activation(_shape(fmt, b, l, H, D), gen, gain=20.0).to(dtype) for _ in range(2))
        state["k_quant"] = VAR_Q(qkv_format=fmt, max_tokens=l, **_kwargs(case["k"]))
        state["v_quant"] = VAR_Q(qkv_format=fmt, max_tokens=l, **_kwargs(case["v"]))
    else:
        b, lq, lk = case["batch"], case["lq"], case["lk"]
        kq, vq = (VAR_Q(qkv_format=fmt, max_tokens=lk, **_kwargs(case[n])) for n in ("k", "v"))
        kq.append(_activation(_shape(fmt, b, lk, H, D), gen, gain=20.0))
        vq.append(torch.randn(_shape(fmt, b, lk, H, D), generator=gen, device="cuda").to(torch.bfloat16))
        state["k_quant"], state["v_quant"] = kq, vq
        state["q"] = torch.randn(_shape(fmt, b, lq, H, D), generator=gen, device="cuda").to(DTYPES[case["q_dtype"]])
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind, fmt = state["kind"], state["fmt"]
    if kind == "layer":
        kv = LayerKV(qkv_format=fmt, k_kwargs=state["k_kwargs"], v_kwargs=state["v_kwargs"], max_tokens=state["tokens"])
        if state["route"] == "normalised":
            outs = [kv.step_normalised(q, k, v, state["scale_mul"], 1.0, out_dtype=torch.bfloat16) for q, k, v in state["steps"]]
        else:
            outs = [kv.step(q, k, v, 1.0, out_dtype=torch.bfloat16) for q, k, v in state["steps"]]
        return {"out": outs, "k_codes": kv.k_quant.cached_item, "v_codes": kv.v_quant.cached_item,
                "k_scale": kv.k_quant.scale, "v_scale": kv.v_quant.scale}
    if kind == "drop_in":
        kq, vq = (VAR_Q(qkv_format=fmt, **state[n]) for n in ("k_kwargs", "v_kwargs"))
        return [(kq.use_var_q(k), vq.use_var_q(v)) for _, k, v in state["steps"]]
    if kind == "round_trip":
        out = {}
        for n in ("k", "v"):
            quantizer = state[n + "_quant"]
            quantizer.quant(state[n + "_item"])
            out[n] = [quantizer.dequant_current(), quantizer.quantized_item, quantizer.scale, quantizer.zero_point]
        return out
    return attend_cached(state["q"], state["k_quant"], state["v_quant"], 1.0 / math.sqrt(state["head_dim"]))


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _packed_bytes(name, b, l, h, d):
    """Codes and parameters of l tokens in one appended step."""
    bits, method, options = SETTINGS[name]
    per_group = 4 if options.get("symmetric", True) else 8
    groups = {"G_SCALE_HEAD_DIM": h * d, "G_TOKEN": l}.get(method, l * h * (d // options.get("group_size", d)))
    return b * l * h * d * bits // 8 + groups * per_group


def work(case):
    kind, H, D = case["kind"], case["heads"], case["head_dim"]
    nbytes = flops = 0
    if kind in ("layer", "drop_in"):
        b, cached = 2 * case["images"], 0
        raw = kind == "layer" and case["route"] == "normalised"
        for l in _step_lengths(case):
            cached += l
            n = b * l * H * D
            nbytes += n * (2 if raw else 4) + n * 2 + sum(_packed_bytes(case[t], b, l, H, D) for t in ("k", "v"))     # fresh k, v; codes out
            if kind == "layer":
                # q in, attention out, and the older part of the packed cache once more
                nbytes += n * (2 if raw else 4) + n * 2 + sum(_packed_bytes(case[t], b, cached - l, H, D) for t in ("k", "v"))
                flops += 4 * b * H * l * cached * D
            else:
                nbytes += 2 * b * cached * H * D * 4 + sum(_packed_bytes(case[t], b, cached - l, H, D) for t in ("k", "v"))
    elif kind == "round_trip":
        b, l = case["batch"], case["tokens"]
        n = b * l * H * D
        nbytes = 2 * n * (4 if case["dtype"] == "fp32" else 2) + 2 * n * 4 + sum(_packed_bytes(case[t], b, l, H, D) for t in ("k", "v"))
    else:
        b, lq, lk = case["batch"], case["lq"], case["lk"]
        es = 4 if case["q_dtype"] == "fp32" else 2
        nbytes = 2 * b * lq * H * D * es + sum(_packed_bytes(case[t], b, lk, H, D) for t in ("k", "v"))
        flops = 4 * b * H * lq * lk * D
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] in ("drop_in", "round_trip"):
        return "exact"              # codes, parameters and their fp32 products are defined bit for bit
    if case["kind"] == "layer":
        # bf16 results over fp16 tensor-core operands.  Codes are exact, unless the layer normalises k itself: a row length that
        # rounds the other way can move a value across a rounding boundary
        tol = {"rel": 5e-3}
        if case["route"] == "normalised":
            tol["differ"] = 1e-4
        return tol
    return {"rel": 1e-3 if case["q_dtype"] == "fp32" else 5e-3 if case["q_dtype"] == "bf16" else 2e-3}
