"""The token <-> step tables of a cache whose parameters are kept per appended step: what is stored after every kind of append."""
import pytest
import torch

from VAR_Q.hooks import LayerKV

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
