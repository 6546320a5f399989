"""The fp32 kernel of the first scales (parameters that vary along head_dim) at the edges of its 16 queries and 32 keys.

Against float64 over the dequantised cache.  The dequantised values are exact in both, scores and sums are fp32.  A chain of n rounded additions errs by
about sqrt(n) 2^-24 of its sum: the kernel's longest are 32 (four partial sums of a score over 128 dims), 16 (the keys of a chunk, even and odd) and 8
(chunks), 3.4e-7, 2.4e-7 and 1.7e-7.  A score's error counts in full in its weight, times the score (up to 4 for unit keys and queries of length 4, scale
0.7: 2.8): 9.5e-7 + 4e-7 in all, below 2e-6.
"""
import pytest
import torch

from VAR_Q import _cabi
from VAR_Q.attention import attend_cached
from VAR_Q.hooks import LayerKV
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"
DIM = dict(quant_method="G_SCALE_HEAD_DIM")
SETTINGS = {
    "int8": (dict(quant_bits=8, **DIM), dict(quant_bits=8, **DIM)),
    "int4_asym_int2": (dict(quant_bits=4, symmetric=False, **DIM), dict(quant_bits=2, symmetric=False, **DIM)),
    "int2_head8": (dict(quant_bits=2, symmetric=False, **DIM), dict(quant_bits=8, quant_method="G_TOKEN_HEAD")),
    "groups_of_8": (dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=8),) * 2,
}


def _cache(kw, steps, fmt, B, H, D, gen, unit):
    qz = VAR_Q(qkv_format=fmt, max_tokens=sum(steps), **kw)
    for n in steps:
        x = torch.randn((B, n, H, D) if fmt == "BLHc" else (B, H, n, D), generator=gen, device=DEV)
        qz.append(x / x.norm(dim=-1, keepdim=True) if unit else x.to(torch.bfloat16))
    return qz


def _reference(q, kq, vq, scale, fmt):
    q, k, v = (t.double() for t in (q, kq.dequant_all(), vq.dequant_all()))
    if fmt == "BLHc":
        q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    return (torch.softmax(q @ k.transpose(-1, -2) * scale, -1) @ v).transpose(1, 2)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("settings", sorted(SETTINGS))
@pytest.mark.parametrize("lq,steps", [(1, (1,)), (4, (1, 4)), (5, (31,)), (9, (7, 25)), (16, (33,)), (13, (1, 30, 2, 31)), (16, (100, 28, 128)), (3, (17, 50))])
def test_edges(D, settings, lq, steps):
    fmt = "BLHc" if lq % 2 else "BHLc"
    B, H = 3, 2
    gen = torch.Generator(device=DEV).manual_seed(lq + sum(steps))
    kq, vq = (_cache(kw, steps, fmt, B, H, D, gen, i == 0) for i, kw in enumerate(SETTINGS[settings]))
    q = torch.randn((B, lq, H, D) if fmt == "BLHc" else (B, H, lq, D), generator=gen, device=DEV)
    q = q / q.norm(dim=-1, keepdim=True) * 4.0
    for q_dtype in (torch.float32, torch.bfloat16):
        x = q.to(q_dtype)
        ref = _reference(x, kq, vq, 0.7, fmt)
        outs = []
        for path in ("early", None):
            _cabi.force_attn_path(path)
            try:
                outs.append(attend_cached(x, kq, vq, 0.7, out_dtype=torch.float32).double())
            finally:
                _cabi.force_attn_path(None)
        for out in outs:
            assert ((out - ref).norm() / ref.norm()).item() <= 2e-6


@pytest.mark.parametrize("D", [64, 128])
def test_normalised_queries_and_strided_rows(D):
    """What the installed hook runs: queries normalised on load, views of a fused activation that starts off a 16-byte boundary."""
    B, H, mul = 2, 3, torch.tensor([0.5, 2.0, 4.0], device=DEV).view(1, 1, 3, 1)
    gen = torch.Generator(device=DEV).manual_seed(D)
    kw = dict(quant_bits=8, **DIM)
    kv = LayerKV(qkv_format="BLHc", k_kwargs=kw, v_kwargs=kw, max_tokens=80)
    for n in (1, 4, 9, 16):
        flat = torch.randn(B * n * 3 * H * D + 2, generator=gen, device=DEV).to(torch.bfloat16)[2:]
        q, k, v = flat.view(B, n, 3, H, D).unbind(2)
        out = kv.step_normalised(q, k, v, mul, 1.0, out_dtype=torch.float32).double()
        qn = q.double() / q.double().norm(dim=-1, keepdim=True).clamp_min(1e-12) * mul.double()
        ref = _reference(qn, kv.k_quant, kv.v_quant, 1.0, "BLHc")
        assert ((out - ref).norm() / ref.norm()).item() <= 2e-6


@pytest.mark.parametrize("kw", [dict(quant_bits=8, quant_method="G_TOKEN_HEAD"), dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False),
                                dict(quant_bits=2, quant_method="G_TOKEN")], ids=["int8_head", "int4_head_asym", "int2_token"])
@pytest.mark.parametrize("heads", [512, 544])
@pytest.mark.parametrize("lq,lk,fp32", [(9, 14, True), (12, 32, True), (13, 32, False), (12, 33, True), (16, 30, False), (25, 55, False), (33, 60, False)])
def test_choice_with_one_scale_per_key(kw, heads, lq, lk, fp32):
    """Both sides of the lines of the automatic choice: fp32-like accuracy wherever the decode or the early kernel takes the call (on 512 pairs
    decode takes 13 and 16 queries too), fp16 weights elsewhere."""
    B, H = heads // 16, 16
    gen = torch.Generator(device=DEV).manual_seed(lq * lk)
    kq, vq = (_cache(kw, (lk,), "BLHc", B, H, 64, gen, i == 0) for i in range(2))
    q = torch.randn((B, lq, H, 64), generator=gen, device=DEV)
    q = q / q.norm(dim=-1, keepdim=True) * 4.0
    out = attend_cached(q, kq, vq, 0.7, out_dtype=torch.float32).double()
    ref = _reference(q, kq, vq, 0.7, "BLHc")
    limit = 2e-6 if fp32 or (lq <= 16 and heads <= 512) else 1e-3
    assert ((out - ref).norm() / ref.norm()).item() <= limit
