"""The warp-level tensor-core kernel for a few queries over a long cache, forced, against the oracle.
Tolerance: max-abs 2e-3, relative L2 1e-3 (fp32 oracle)."""
import pytest
import torch

from oracle import varq_oracle as O
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
@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 4), (2, 2), (4, 2), (2, 8), (8, 4)])
@pytest.mark.parametrize("lq,lk,mode,symmetric,q_dtype", [
    (1, 1, "G_TOKEN_HEAD", True, torch.float32), (4, 15, "G_TOKEN_HEAD", False, torch.float32), (3, 300, "G_TOKEN", False, torch.bfloat16),
    (5, 1000, "G_TOKEN_HEAD", False, torch.float32), (8, 2049, "G_TOKEN", True, torch.float16), (9, 529, "G_TOKEN_HEAD", True, torch.float32)])
def test_against_the_oracle(D, kb, vb, lq, lk, mode, symmetric, q_dtype):
    fmt, B, H = "BHLc", 2, 3
    kq, vq = (VAR_Q(b, fmt, mode, symmetric=symmetric) for b in (kb, vb))
    kr, vr = (O.OracleVARQ(b, fmt, mode, symmetric=symmetric) for b in (kb, vb))
    for si, n in enumerate((lk - lk // 3, lk // 3)):
        if n == 0:
            continue
        k = O.synthetic_kv((B, H, n, D), fmt, 31 + si, n_outlier=4)
        v = O.synthetic_kv((B, H, n, D), fmt, 41 + si, n_outlier=0)
        kq.append(k.to(DEV)); vq.append(v.to(DEV))
        kd, vd = kr.use_var_q(k), vr.use_var_q(v)
    q = torch.randn((B, H, lq, D), generator=torch.Generator().manual_seed(lq + lk)).to(q_dtype)
    _cabi.force_attn_path("decode")
    out = attend_cached(q.to(DEV), kq, vq, 1.0 / D ** 0.5, out_dtype=torch.float32).cpu()
    ref = O.attention(q.float(), kd, vd, fmt, 1.0 / D ** 0.5).transpose(1, 2)
    err, rel = (out - ref).abs().max().item(), ((out - ref).norm() / ref.norm()).item()
    assert err <= 2e-3 and rel <= 1e-4, f"max-abs {err:.3e}, rel-L2 {rel:.3e}"       # fp32-like accuracy: fp16 hi + lo operands
