"""Which kernel the automatic choice takes: its result is compared bit for bit with that of the kernel pinned, on both sides of the lines between
kernels, and has to differ from that of the kernel on the other side (another order of sums, or fp16 weights instead of fp32)."""
import pytest
import torch

from VAR_Q import _cabi
from VAR_Q.attention import attend_cached
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"
HEAD8 = dict(quant_bits=8, quant_method="G_TOKEN_HEAD")
HEAD4 = dict(quant_bits=4, quant_method="G_TOKEN_HEAD", symmetric=False)
TOKEN2 = dict(quant_bits=2, quant_method="G_TOKEN")


@pytest.fixture(autouse=True)
def _auto_path_afterwards():
    yield
    _cabi.force_attn_path(None)


def _pair(kw, heads, lk, gen, D=64):
    out = []
    for unit in (True, False):
        x = torch.randn((1, heads, lk, D), generator=gen, device=DEV)
        qz = VAR_Q(qkv_format="BHLc", max_tokens=lk, **kw)
        qz.append(x / x.norm(dim=-1, keepdim=True) if unit else x)
        out.append(qz)
    return out


def _run(path, q, kq, vq):
    _cabi.force_attn_path(path)
    return attend_cached(q, kq, vq, 0.7, out_dtype=torch.float32)


def _check(kw, heads, lq, lk, dtype, taken, others, limit=1e-3):
    gen = torch.Generator(device=DEV).manual_seed(heads + lq + lk)
    kq, vq = _pair(kw, heads, lk, gen)
    q = (torch.nn.functional.normalize(torch.randn((1, heads, lq, 64), generator=gen, device=DEV), dim=-1) * 4.0).to(dtype)
    auto = _run(None, q, kq, vq)
    assert torch.equal(auto, _run(taken, q, kq, vq)), f"not the result of {taken}"
    for path in others:
        assert not torch.equal(auto, _run(path, q, kq, vq)), f"{taken} and {path} cannot be told apart"
    ref = torch.softmax(q.double() @ kq.dequant_all().double().transpose(-1, -2) * 0.7, -1) @ vq.dequant_all().double()
    assert ((auto.double() - ref.transpose(1, 2)).norm() / ref.norm()).item() <= limit


# CTAs per SM and their waves decide, so heads are given per SM: 2.0 to 2.1 around the line, 3.4 a well filled wave of four (16-bit queries), 4.2 and 8.1 badly filled ones
@pytest.mark.parametrize("kw", [HEAD8, HEAD4, TOKEN2], ids=["int8", "int4", "int2"])
@pytest.mark.parametrize("per_sm,lq,lk,dtype,mid", [
    (2.0, 33, 40, torch.bfloat16, False), (2.1, 33, 40, torch.bfloat16, True), (2.1, 48, 96, torch.float16, True), (2.1, 49, 96, torch.bfloat16, False),
    (3.4, 64, 96, torch.bfloat16, True), (3.4, 65, 96, torch.bfloat16, False), (3.4, 64, 97, torch.bfloat16, None), (3.4, 36, 208, torch.float16, None),
    (3.4, 36, 209, torch.bfloat16, False), (4.2, 48, 64, torch.bfloat16, True), (4.2, 64, 64, torch.bfloat16, False),
    (2.1, 33, 40, torch.float32, True), (2.9, 64, 91, torch.float32, True), (2.9, 64, 97, torch.float32, False),
    (3.4, 33, 40, torch.float32, False), (4.3, 40, 64, torch.float32, True), (4.3, 41, 64, torch.float32, False), (4.3, 33, 65, torch.float32, False),
    (2.0, 17, 30, torch.bfloat16, False), (2.1, 17, 30, torch.bfloat16, True), (2.1, 32, 200, torch.float32, True)])
def test_warp_level_or_tcgen05(kw, per_sm, lq, lk, dtype, mid):
    heads = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    if mid is None:
        mid = kw is not HEAD8           # narrow codes only
    _check(kw, heads, lq, lk, dtype, *(("mid", ["tc"]) if mid else ("tc", ["mid"])))


# (sample, head) pairs per SM, or as such: 3 and 5 per SM and 512 are the lines
@pytest.mark.parametrize("kw", [HEAD8, HEAD4, TOKEN2], ids=["int8", "int4", "int2"])
@pytest.mark.parametrize("per_sm,pairs,lq,lk,dtype,taken", [
    (3.0, 0, 9, 14, torch.float32, "decode"), (3.1, 0, 9, 14, torch.float32, "early"), (3.1, 0, 16, 16, torch.bfloat16, "early"), (3.1, 0, 12, 17, torch.bfloat16, "decode"),
    (5.0, 0, 12, 30, torch.float32, "decode"), (5.1, 0, 12, 32, torch.bfloat16, "early"), (5.1, 0, 16, 32, torch.float32, "early"), (5.1, 0, 13, 32, torch.bfloat16, "mid"),
    (5.1, 0, 12, 33, torch.float32, "decode"), (0, 512, 13, 30, torch.float32, "decode"), (0, 513, 13, 30, torch.float32, "mid"), (0, 513, 13, 33, torch.bfloat16, "decode")])
def test_nine_to_sixteen_queries(kw, per_sm, pairs, lq, lk, dtype, taken):
    heads = pairs or int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    _check(kw, heads, lq, lk, dtype, taken, {"decode", "early", "mid"} - {taken}, 1e-3 if taken == "mid" else 2e-6)


@pytest.mark.parametrize("lq,lk,taken,other", [(4, 300, "small", "tc"), (16, 256, "early", "small"), (17, 256, "tc", "early"), (16, 257, "tc", "early")])
def test_parameters_along_head_dim(lq, lk, taken, other):
    kw = dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM")
    _check(kw, 96, lq, lk, torch.float32, taken, {other}, 1e-3 if taken == "tc" else 2e-6)
