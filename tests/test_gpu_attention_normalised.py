"""Attention on queries normalised inside the kernel (``varq_attn_fwd_qnorm``, ``LayerKV.step_normalised``), each kernel forced and the
automatic choice, against float64 attention over the dequantised cache.

Bars, relative L2.  Kernels with fp32 weights (small, stream, decode): 2e-6 -- a logit of magnitude s <= 8 sums head_dim products in fp32, an
error of about sqrt(head_dim) * 2^-24 * s = 4e-6 at worst and a tenth of that on average, and the weighted sum over keys adds less; weights
rounded to fp16 would be 2e-4.  Tensor-core kernel: 1e-3, fp16 weights and V."""
import pytest
import torch

from VAR_Q import _cabi
from VAR_Q.hooks import LayerKV
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"
FP32_BAR, FP16_BAR = 2e-6, 1e-3
SETTINGS = {
    "dim8": dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM"),
    "dim4_asym": dict(quant_bits=4, quant_method="G_SCALE_HEAD_DIM", symmetric=False),
    "group32": dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=32),
    "head8": dict(quant_bits=8, quant_method="G_TOKEN_HEAD"),
    "head2_asym": dict(quant_bits=2, quant_method="G_TOKEN_HEAD", symmetric=False),
}


@pytest.fixture(autouse=True)
def _auto_path_afterwards():
    yield
    _cabi.force_attn_path(None)


def exact(q, mul, kd, vd, scale):
    """float64 attention, BHLc in, [B, L, H, c] out"""
    q, kd, vd = q.double(), kd.double(), vd.double()
    q = q / q.norm(dim=-1, keepdim=True).clamp_min(1e-12)
    if mul is not None:
        q = q * mul.double().view(1, -1, 1, 1)
    return (torch.softmax(q @ kd.transpose(-1, -2) * scale, -1) @ vd).transpose(1, 2)


def rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("fmt", ["BLHc", "BHLc"])
@pytest.mark.parametrize("k_name,v_name", [("dim8", "dim8"), ("dim4_asym", "head2_asym"), ("group32", "group32"), ("head8", "head8")])
def test_few_normalised_queries_keep_fp32_weights(D, fmt, k_name, v_name):
    """The first scales of a schedule, and up to four queries over any history."""
    B, H = 3, 5
    kv = LayerKV(qkv_format=fmt, k_kwargs=SETTINGS[k_name], v_kwargs=SETTINGS[v_name])
    mul = torch.linspace(1.0, 5.0, H, device=DEV)
    gen = torch.Generator(device=DEV).manual_seed(D)
    for n in (1, 4, 9, 16, 100, 16, 200, 4, 3):
        qkv = torch.randn((B, n, 3, H, D), generator=gen, device=DEV)
        qkv[..., :4] *= 6.0
        q, k, v = qkv.to(torch.bfloat16).unbind(dim=2)
        if fmt == "BHLc":
            q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
        out = kv.step_normalised(q, k, v, mul, 1.0, out_dtype=torch.float32)
        kd, vd = kv.k_quant.dequant_all(), kv.v_quant.dequant_all()
        if fmt == "BLHc":
            q, kd, vd = (t.permute(0, 2, 1, 3) for t in (q, kd, vd))
        few = n <= 4 or (n <= 16 and kv.n_tokens <= 256)
        err = rel(out, exact(q, mul, kd, vd, 1.0))
        assert err <= (FP32_BAR if few else FP16_BAR), f"{n} queries over {kv.n_tokens} tokens: rel-L2 {err:.2e}"
    assert _cabi.device_status() == 0


def attend_qnorm(path, q, kq, vq, scale, mul, eps=1e-12):
    B, H, lq, D = q.shape
    lib, lk = _cabi.lib(), kq.n_tokens
    out = torch.full((B, lq, H, D), float("nan"), device=DEV)
    (kc, kp), (vc, vp) = kq.cache_descriptors(), vq.cache_descriptors()
    need = lib.varq_attn_workspace_bytes(B, H, lq, lk, D, kq.store_bits, vq.store_bits)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    od = _cabi.tensor_desc(out.data_ptr(), _cabi.F32, lq * H * D, H * D, D)
    _cabi.force_attn_path(path)
    _cabi.check(lib.varq_attn_fwd_qnorm(kq._item_desc(q), kc, vc, kp, vp, B, H, lq, lk, D, kq.store_bits, vq.store_bits, float(scale),
                                        mul.data_ptr() if mul is not None else None, eps, od, ws.data_ptr(), need, _cabi.stream_ptr(q.device)))
    torch.cuda.synchronize()
    assert _cabi.device_status() == 0
    return out


# one key, a full warp step, a second query tile of the tensor-core kernel, split key ranges of every kernel
@pytest.mark.parametrize("path,lq,lk", [(p, lq, lk) for p in ("small", "stream", "decode") for lq, lk in ((1, 1), (3, 65), (5, 300), (16, 1500))] +
                         [("tc", lq, lk) for lq, lk in ((1, 1), (33, 65), (129, 200), (300, 130), (20, 1500))])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("k_name,v_name", [("dim8", "dim4_asym"), ("group32", "head8"), ("head8", "head2_asym")])
@pytest.mark.parametrize("dtype,with_mul", [(torch.bfloat16, True), (torch.float32, False), (torch.float16, True)])
def test_each_kernel_normalises_the_queries_it_loads(path, lq, lk, D, k_name, v_name, dtype, with_mul):
    B, H = 2, 3
    gen = torch.Generator(device=DEV).manual_seed(lq + lk)
    kq, vq = VAR_Q(qkv_format="BHLc", **SETTINGS[k_name]), VAR_Q(qkv_format="BHLc", **SETTINGS[v_name])
    for n in (lk - lk // 3, lk // 3):
        if n:
            kq.append(torch.nn.functional.normalize(torch.randn((B, H, n, D), generator=gen, device=DEV), dim=-1))
            vq.append(torch.randn((B, H, n, D), generator=gen, device=DEV))
    # a third of a fused activation: strided rows; magnitudes that only matter if a row is not normalised
    q = (torch.randn((B, lq, 3, H, D), generator=gen, device=DEV) * torch.logspace(-2, 2, lq, device=DEV).view(1, lq, 1, 1, 1)).to(dtype)
    q = q.unbind(dim=2)[1].permute(0, 2, 1, 3)
    mul = torch.linspace(2.0, 6.0, H, device=DEV) if with_mul else None
    err = rel(attend_qnorm(path, q, kq, vq, 1.0, mul), exact(q, mul, kq.dequant_all(), vq.dequant_all(), 1.0))
    # (where a kernel does not take the grouping or the call, the next one in line does)
    bar = FP16_BAR if path == "tc" else FP32_BAR
    assert err <= bar, f"rel-L2 {err:.2e}"


@pytest.mark.parametrize("path", ["small", "stream", "decode", "tc"])
def test_a_query_of_zeros_attends_to_all_keys_alike(path):
    kq, vq = VAR_Q(qkv_format="BHLc", **SETTINGS["head8"]), VAR_Q(qkv_format="BHLc", **SETTINGS["head8"])
    x = torch.randn((1, 2, 70, 64), generator=torch.Generator(device=DEV).manual_seed(3), device=DEV)
    kq.append(x); vq.append(x.flip(2).contiguous())
    out = attend_qnorm(path, torch.zeros((1, 2, 3, 64), device=DEV), kq, vq, 1.0, None)
    assert torch.allclose(out, vq.dequant_all().mean(dim=2).view(1, 1, 2, 64).expand_as(out), atol=1e-3)
