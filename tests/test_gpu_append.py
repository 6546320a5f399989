"""The append kernels (rows, planes in one cluster, planes in two passes, per-token planes; K alone and normalised) at the edges of
their ranges, against the CPU oracle.  Bar: bit-exact codes, scales, zero-points and dequantised values."""
import pytest
import torch

from oracle import varq_oracle as O
from VAR_Q.hooks import LayerKV, normalise_qk
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


def same_bits(a, b):
    a, b = a.detach().cpu().contiguous(), b.detach().cpu().contiguous()
    return a.shape == b.shape and a.dtype == b.dtype and torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a,
                                                                     b.view(torch.int32) if b.dtype == torch.float32 else b)


# batch 1 / 33 / 65: one row per thread, a ragged last batch lane, 512 threads; 2 x 900 rows: planes in two passes; 1 and 3 tokens: one CTA
@pytest.mark.parametrize("B,H,steps", [(1, 3, (1, 3)), (33, 2, (2, 5)), (65, 1, (4,)), (2, 3, (40, 900))])
@pytest.mark.parametrize("D,fmt", [(64, "BLHc"), (128, "BHLc"), (32, "BLHc")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits,mode,options", [
    (8, "G_SCALE_HEAD_DIM", {}), (4, "G_SCALE_HEAD_DIM", dict(symmetric=False)), (4, "G_SCALE", {}), (8, "G_TOKEN", dict(symmetric=False)),
    (2, "G_TOKEN_HEAD", {}), (8, "G_TOKEN_HEAD", dict(symmetric=False)), (4, "G_TOKEN_HEAD", dict(group_size=32))])
def test_codes_and_parameters_match_the_oracle(B, H, steps, D, fmt, dtype, bits, mode, options):
    dut, ref = VAR_Q(bits, fmt, mode, **options), O.OracleVARQ(bits, fmt, mode, **options)
    for si, n in enumerate(steps):
        x = O.synthetic_kv((B, n, H, D) if fmt == "BLHc" else (B, H, n, D), fmt, 7 * si + B, n_outlier=2).to(dtype)
        deq, want = dut.use_var_q(x.to(DEV)), ref.use_var_q(x)
        assert same_bits(dut.cached_item, ref.cached_item) and same_bits(dut.cached_scale, ref.cached_scale)
        assert ref.cached_zp is None or same_bits(dut.cached_zero_point, ref.cached_zp)
        assert same_bits(deq, want)


@pytest.mark.parametrize("D,fmt", [(64, "BLHc"), (128, "BHLc")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits,mode,options", [(8, "G_SCALE_HEAD_DIM", {}), (4, "G_TOKEN_HEAD", {}), (4, "G_TOKEN_HEAD", dict(group_size=32, symmetric=False)),
                                               (8, "G_TOKEN", {})])
def test_rows_normalised_on_the_way_in_get_the_codes_of_normalised_rows(D, fmt, dtype, bits, mode, options):
    """The row length is summed in the order of the normalising kernel: the same bits, hence the same codes."""
    B, H, kw = 3, 5, dict(quant_bits=bits, quant_method=mode, **options)
    kv, kq, vq = LayerKV(qkv_format=fmt, k_kwargs=kw, v_kwargs=kw), VAR_Q(qkv_format=fmt, **kw), VAR_Q(qkv_format=fmt, **kw)
    gen = torch.Generator().manual_seed(D + bits)
    for n in (1, 25, 600):
        q, k, v = torch.randn((B, n, 3, H, D), generator=gen).mul_(3).to(dtype).to(DEV).unbind(dim=2)
        if fmt == "BHLc":
            q, k, v = (t.permute(0, 2, 1, 3) for t in (q, k, v))
        kv.step_normalised(q, k, v, None, 1.0)
        kq.append(normalise_qk(q, k, v, kq, vq)[1]); vq.append(v)
        for dut, ref in ((kv.k_quant, kq), (kv.v_quant, vq)):
            assert same_bits(dut.cached_item, ref.cached_item) and same_bits(dut.cached_scale, ref.cached_scale)
            assert ref.cached_zero_point is None or same_bits(dut.cached_zero_point, ref.cached_zero_point)
