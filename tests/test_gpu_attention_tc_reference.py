"""Tensor-core attention where the softmax reference of a row has to move in the middle of its keys.

A row keeps its reference until a tile's weights outgrow fp16; the accumulators are then rescaled.  Here rows of one of the two query tiles,
of single warps or of every second row meet far larger scores every few tiles, V scales span orders of magnitude, and K zero-points lie
outside the exact operand's range.  Against float64 over the dequantised cache; tolerance 1e-3 relative L2 (fp16 weights give 2-3e-4).
"""
import pytest
import torch

from VAR_Q import _cabi
from VAR_Q.attention import attend_cached
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"
HEAD8 = dict(quant_bits=8, quant_method="G_TOKEN_HEAD")
HEAD4 = dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False)
GROUP4 = dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=32)
GROUP16 = dict(quant_bits=2, quant_method="G_TOKEN_HEAD", symmetric=False, group_size=16)
DIM8 = dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM")


@pytest.fixture(autouse=True)
def _tensor_core_path():
    _cabi.force_attn_path("tc")
    yield
    _cabi.force_attn_path(None)
    torch.cuda.synchronize()
    assert _cabi.device_status() == 0


def _check(q, kq, vq, scale, tag):
    out = attend_cached(q, kq, vq, scale, out_dtype=torch.float32).transpose(1, 2).double()
    kd, vd = kq.dequant_all().double(), vq.dequant_all().double()
    ref = torch.softmax(q.double() @ kd.transpose(-1, -2) * scale, -1) @ vd
    err = ((out - ref).norm(dim=-1) / ref.norm(dim=-1).clamp_min(1e-30)).max().item()
    rel = ((out - ref).norm() / ref.norm()).item()
    assert rel <= 1e-3 and err <= 5e-3, f"{tag}: rel-L2 {rel:.2e}, worst row {err:.2e}"


@pytest.mark.parametrize("rows", ["second_tile", "one_warp", "alternate", "all"])
@pytest.mark.parametrize("D,lq,k_kw,v_kw,q_dtype", [
    (64, 256, HEAD8, HEAD4, torch.float32), (64, 256, GROUP4, GROUP4, torch.bfloat16), (64, 200, DIM8, HEAD8, torch.float32),
    (64, 100, HEAD4, HEAD8, torch.bfloat16), (64, 256, GROUP16, GROUP16, torch.float32), (128, 256, HEAD8, HEAD8, torch.bfloat16),
    (128, 160, GROUP4, GROUP4, torch.float32), (128, 130, DIM8, HEAD4, torch.bfloat16)])
def test_reference_moves(D, lq, k_kw, v_kw, q_dtype, rows):
    B, H, lk = 2, 40, 1500
    g = torch.Generator(device=DEV).manual_seed(D + lq)
    k, v = (torch.randn((B, H, lk, D), generator=g, device=DEV) for _ in range(2))
    q = torch.randn((B, H, lq, D), generator=g, device=DEV)
    who = torch.zeros(lq, device=DEV)
    who[{"second_tile": slice(128, None), "one_warp": slice(32, 64), "alternate": slice(0, None, 2), "all": slice(None)}[rows]] = 1.0
    # the marked rows look along the first dimension, where every third tile holds a key that is larger than all before it
    q[..., 0] = who * 6.0
    for n, tile in enumerate(range(2, lk // 64, 3)):
        k[:, :, tile * 64 + 7 * n % 64, 0] = 4.0 + 4.0 * n
    kq, vq = VAR_Q(qkv_format="BHLc", max_tokens=lk, **k_kw), VAR_Q(qkv_format="BHLc", max_tokens=lk, **v_kw)
    kq.append(k)
    vq.append(v)
    _check(q.to(q_dtype), kq, vq, 1.0, f"{D} {lq} {rows}")


@pytest.mark.parametrize("D,lq,q_dtype", [(64, 256, torch.float32), (64, 40, torch.bfloat16), (128, 256, torch.bfloat16), (128, 256, torch.float32)])
def test_scales_of_a_tile_far_apart(D, lq, q_dtype):
    """V rows between 0.03 and 10 side by side (a weight has to stay inside fp16 next to the largest product of weight and V scale), and K rows
    far from zero (a zero-point outside +-512)."""
    B, H, lk = 1, 40, 333
    g = torch.Generator(device=DEV).manual_seed(lq)
    k, v = (torch.randn((B, H, lk, D), generator=g, device=DEV) for _ in range(2))
    v *= (10.0 ** (torch.rand((1, 1, lk, 1), generator=g, device=DEV) * 2.5 - 1.5))
    k[:, :, 5::17] = k[:, :, 5::17] * 1e-3 + 0.5
    q = torch.randn((B, H, lq, D), generator=g, device=DEV)
    kq, vq = VAR_Q(qkv_format="BHLc", max_tokens=lk, **HEAD4), VAR_Q(qkv_format="BHLc", max_tokens=lk, **HEAD8)
    kq.append(k)
    vq.append(v)
    _check(q.to(q_dtype), kq, vq, 0.3, f"{D} {lq}")


@pytest.mark.parametrize("D,lq,q_dtype", [(64, 256, torch.float32), (64, 40, torch.bfloat16), (128, 256, torch.float32), (128, 256, torch.bfloat16)])
@pytest.mark.parametrize("grows", [False, True])
def test_heavy_keys_with_small_v_scales(D, lq, q_dtype, grows):
    """The first key of most tiles is far lighter than the others and its V 10^5 times larger: the sum of the weights passes the limit of its tile,
    the reference stays.  Some tiles are even, and in some rows larger keys follow later."""
    B, H, lk = 1, 40, 64 * 9 + 11
    g = torch.Generator(device=DEV).manual_seed(lq + D)
    u = torch.nn.functional.normalize(torch.randn((B, H, 1, D), generator=g, device=DEV), dim=-1)
    k = torch.randn((B, H, lk, D), generator=g, device=DEV) / D ** 0.5 + 3 * u
    v = torch.randn((B, H, lk, D), generator=g, device=DEV) * 1e-2
    k[:, :, ::64] -= 6 * u
    v[:, :, ::64] *= 1e5
    k[:, :, 128:256:64] += 6 * u
    v[:, :, 128:256:64] *= 1e-5
    if grows:
        k[:, :, 300::150] *= 3.0
    q = 5 * u + torch.randn((B, H, lq, D), generator=g, device=DEV)
    q[:, :, 1::3] *= 0.2
    kq, vq = VAR_Q(qkv_format="BHLc", max_tokens=lk, **HEAD8), VAR_Q(qkv_format="BHLc", max_tokens=lk, **HEAD8)
    kq.append(k)
    vq.append(v)
    _check(q.to(q_dtype), kq, vq, 1.0, f"{D} {lq}")
