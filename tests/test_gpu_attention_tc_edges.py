"""The tensor-core kernel, forced, at the edges of its tiles: one, two and three key tiles per row (head_dim 128 gives even and odd tiles to
different threads), a second query tile, split key ranges, a reference maximum that moves.
Tolerance: max-abs 2e-3, relative L2 1e-3 (fp32 oracle)."""
import pytest
import torch

from oracle import varq_oracle as O
from test_gpu_attention_normalised import attend_qnorm, exact, rel
from VAR_Q import _cabi
from VAR_Q.attention import attend_cached
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _auto_path_afterwards():
    yield
    _cabi.force_attn_path(None)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("q_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kb,vb,options", [(8, 8, {}), (4, 2, dict(symmetric=False)), (4, 4, dict(group_size=32))])
@pytest.mark.parametrize("lq,lk,gain", [(1, 1, 1.0), (128, 64, 1.0), (129, 65, 1.0), (200, 128, 300.0), (33, 129, 300.0), (20, 1500, 1.0)])
def test_against_the_oracle(D, q_dtype, kb, vb, options, lq, lk, gain):
    fmt, B, H = "BHLc", 1, 2
    kq, vq = (VAR_Q(b, fmt, "G_TOKEN_HEAD", **options) for b in (kb, vb))
    kr, vr = (O.OracleVARQ(b, fmt, "G_TOKEN_HEAD", **options) for b in (kb, vb))
    k = O.synthetic_kv((B, H, lk, D), fmt, 3 + lk, n_outlier=0)
    k = k / k.norm(dim=-1, keepdim=True) * torch.linspace(0.2, 1.0, lk).view(1, 1, lk, 1)        # later keys weigh more
    v = O.synthetic_kv((B, H, lk, D), fmt, 5 + lk, n_outlier=0)
    kq.append(k.to(DEV)); vq.append(v.to(DEV))
    kd, vd = kr.use_var_q(k), vr.use_var_q(v)
    q = torch.randn((B, H, lq, D), generator=torch.Generator().manual_seed(lq + lk))
    q = (q / q.norm(dim=-1, keepdim=True) * gain).to(q_dtype)
    _cabi.force_attn_path("tc")
    out = attend_cached(q.to(DEV), kq, vq, 1.0, out_dtype=torch.float32).cpu()
    ref = O.attention(q.float(), kd, vd, fmt, 1.0).transpose(1, 2)
    err, rel = (out - ref).abs().max().item(), ((out - ref).norm() / ref.norm()).item()
    assert err <= 2e-3 and rel <= 1e-3, f"max-abs {err:.3e}, rel-L2 {rel:.3e}"
    assert _cabi.device_status() == 0


@pytest.mark.parametrize("B,H,lq,lk", [(2, 16, 169, 424), (4, 16, 256, 680), (5, 16, 256, 680), (1, 16, 169, 424), (2, 16, 256, 1024), (2, 16, 256, 1025), (1, 12, 400, 300)])
def test_query_tiles_per_cta(B, H, lq, lk):
    """Both sides of the line between one and two query tiles per CTA (few CTAs, short caches), with and without key splits."""
    g = torch.Generator(device="cuda").manual_seed(lq + lk)
    kq, vq = (VAR_Q(qkv_format="BHLc", quant_bits=8, quant_method="G_TOKEN_HEAD", max_tokens=lk) for _ in range(2))
    for qz in (kq, vq):
        qz.append(torch.randn((B, H, lk, 64), generator=g, device="cuda"))
    q = torch.randn((B, H, lq, 64), generator=g, device="cuda")
    out = attend_cached(q, kq, vq, 0.125, out_dtype=torch.float32).transpose(1, 2).double()
    ref = torch.softmax(q.double() @ kq.dequant_all().double().transpose(-1, -2) * 0.125, -1) @ vq.dequant_all().double()
    assert ((out - ref).norm() / ref.norm()).item() <= 1e-3        # fp16 weights


@pytest.mark.parametrize("kw", [dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=32), dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM")],
                         ids=["group32", "dim8"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,lq,lk", [(2, 16, 169, 424), (4, 16, 256, 680), (5, 16, 256, 680), (1, 16, 169, 424), (2, 16, 256, 1025)])
def test_query_tiles_per_cta_with_dequantised_k(B, H, lq, lk, dtype, kw):
    """The same line for caches whose K and V every query tile of a CTA of its own has to convert again."""
    g = torch.Generator(device="cuda").manual_seed(lq + lk)
    kq, vq = (VAR_Q(qkv_format="BHLc", max_tokens=lk, **kw) for _ in range(2))
    for qz in (kq, vq):
        for n in (lk // 3, lk - lk // 3):
            qz.append(torch.randn((B, H, n, 64), generator=g, device="cuda"))
    q = torch.randn((B, H, lq, 64), generator=g, device="cuda").to(dtype)
    out = attend_cached(q, kq, vq, 0.125, out_dtype=torch.float32).transpose(1, 2).double()
    ref = torch.softmax(q.double() @ kq.dequant_all().double().transpose(-1, -2) * 0.125, -1) @ vq.dequant_all().double()
    assert ((out - ref).norm() / ref.norm()).item() <= 1e-3        # fp16 weights and V


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,lq,lk", [(2, 18, 256, 1100), (2, 19, 200, 1100), (2, 37, 129, 1024), (2, 37, 129, 1300), (5, 15, 200, 1300)])
def test_query_tiles_per_cta_over_longer_caches(B, H, lq, lk, dtype):
    """36 CTAs of two tiles (their key range is split), 38 and 74 (single tiles), 75 (two again)."""
    test_query_tiles_per_cta_with_dequantised_k(B, H, lq, lk, dtype, dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM"))
    test_query_tiles_per_cta(B, H, lq, lk)


@pytest.mark.parametrize("normalised", [False, True])
@pytest.mark.parametrize("dtype,shift,pad", [(torch.float32, 1, 1), (torch.bfloat16, 1, 0), (torch.bfloat16, 0, 3), (torch.float16, 3, 1)])
@pytest.mark.parametrize("kw", [dict(quant_bits=8, quant_method="G_TOKEN_HEAD"), dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=32),
                                dict(quant_bits=2, quant_method="G_SCALE_HEAD_DIM", symmetric=False)], ids=["head8", "group32", "dim2"])
@pytest.mark.parametrize("D,lq", [(64, 45), (64, 150), (128, 45), (128, 150)])
def test_query_rows_off_a_16_byte_boundary(D, lq, kw, dtype, shift, pad, normalised):
    """Rows that start anywhere and lie any distance apart, in every kind of kernel that reads them in pieces of 16 bytes."""
    B, H, lk = 2, 3, 150
    g = torch.Generator(device=DEV).manual_seed(lq + shift)
    kq, vq = (VAR_Q(qkv_format="BHLc", max_tokens=lk, **kw) for _ in range(2))
    for n in (50, 100):
        kq.append(torch.nn.functional.normalize(torch.randn((B, H, n, D), generator=g, device=DEV), dim=-1))
        vq.append(torch.randn((B, H, n, D), generator=g, device=DEV))
    row = H * D + pad
    flat = torch.randn(B * lq * row + 8, generator=g, device=DEV).to(dtype)[shift:]
    q = flat.as_strided((B, H, lq, D), (lq * row, D, row, 1))
    mul = torch.linspace(2.0, 4.0, H, device=DEV)
    if normalised:
        out, ref = attend_qnorm("tc", q, kq, vq, 1.0, mul), exact(q, mul, kq.dequant_all(), vq.dequant_all(), 1.0)
    else:
        _cabi.force_attn_path("tc")
        out = attend_cached(q, kq, vq, 0.2, out_dtype=torch.float32)
        ref = (torch.softmax(q.double() @ kq.dequant_all().double().transpose(-1, -2) * 0.2, -1) @ vq.dequant_all().double()).transpose(1, 2)
    assert rel(out, ref) <= 1e-3        # fp16 weights
