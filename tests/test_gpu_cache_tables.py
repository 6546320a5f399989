"""The token <-> step tables of a cache whose parameters are kept per appended step: what is stored after every kind of append, and
attention that is given only part of them."""
import ctypes

import pytest
import torch

from VAR_Q import _cabi
from VAR_Q.hooks import LayerKV
from VAR_Q.quant import VAR_Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [32, 64])
def test_first_tokens_of_the_steps_whatever_appended_them(D):
    """At head_dim 32 no append kernel normalises K: the native call has allocated the tables when it hands over to the separate
    producer kernel, and nothing in them may be left as the allocator gave it."""
    kw = dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM")
    kv = LayerKV(qkv_format="BLHc", k_kwargs=kw, v_kwargs=kw, max_tokens=64)
    junk = [torch.full((128,), -1, dtype=torch.int32, device=DEV) for _ in range(8192)]        # recycled memory is not zero: every small block
    del junk
    steps = (1, 4, 9)
    for n in steps:
        q, k, v = torch.randn((2, n, 3, 3, D), device=DEV).unbind(dim=2)
        kv.step_normalised(q, k, v, None, 1.0)
    for c in (kv.k_quant, kv.v_quant):
        assert c.state_dict()["row_begin"].tolist() == [0, 1, 5, 14]
        assert c.state_dict()["row_of_token"].tolist() == [0] + [1] * 4 + [2] * 9


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("steps", [(3, 60, 200), (9,) * 45])
def test_attention_without_the_table_of_first_tokens_or_the_number_of_steps(D, steps):
    """`row_begin` is not read (the same bits without it); without `n_rows` the steps are taken as the keys name them."""
    B, H, lq, lk, scale = 1, 2, 40, sum(steps), 0.1
    kw = dict(quant_bits=4, quant_method="G_SCALE_HEAD_DIM", symmetric=False)
    kq, vq = VAR_Q(qkv_format="BHLc", **kw), VAR_Q(qkv_format="BHLc", **kw)
    gen = torch.Generator(device=DEV).manual_seed(D)
    for n in steps:
        kq.append(torch.randn((B, H, n, D), generator=gen, device=DEV)); vq.append(torch.randn((B, H, n, D), generator=gen, device=DEV))
    q = torch.randn((B, H, lq, D), generator=gen, device=DEV)
    lib, outs = _cabi.lib(), []
    need = lib.varq_attn_workspace_bytes(B, H, lq, lk, D, 4, 4)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    for begin, rows in ((True, len(steps)), (False, len(steps)), (False, 0), (True, lk + 1)):
        (kc, kp), (vc, vp) = kq.cache_descriptors(), vq.cache_descriptors()
        for p in (kp, vp):
            p.n_rows = rows
            if not begin:
                p.row_begin = ctypes.c_void_p(None)
        out = torch.empty((B, lq, H, D), device=DEV)
        od = _cabi.tensor_desc(out.data_ptr(), _cabi.F32, lq * H * D, H * D, D)
        _cabi.check(lib.varq_attn_fwd(kq._item_desc(q), kc, vc, kp, vp, B, H, lq, lk, D, 4, 4, scale, od, ws.data_ptr(), need, _cabi.stream_ptr(q.device)))
        outs.append(out)
    kd, vd = kq.dequant_all().double(), vq.dequant_all().double()
    ref = (torch.softmax(q.double() @ kd.transpose(-1, -2) * scale, -1) @ vd).transpose(1, 2)
    assert _cabi.device_status() == 0
    assert torch.equal(outs[0], outs[1])
    for out in outs:
        assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3        # weights and V in fp16
