"""Scratch of captured calls: a CUDA graph replays the addresses it was captured with, so what its kernels write must belong to the graph and
to nobody else, whatever runs between capture and replay."""
import pytest
import torch

from VAR_Q import _cabi, attention, quant
from VAR_Q.attention import attend_cached
from VAR_Q.quant import VAR_Q, _host

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("python_path", [False, True])
def test_a_replay_writes_no_memory_that_others_were_given(python_path, monkeypatch):
    """Few heads and a long cache: attention with split key ranges, whose partial rows go through scratch; and a step large enough for the
    two-pass quantizer, whose statistics do."""
    if python_path:
        monkeypatch.setattr(attention, "_host", None)
        monkeypatch.setattr(quant, "_host", None)
    gen = torch.Generator(device=DEV).manual_seed(1)
    kw = dict(quant_bits=8, quant_method="G_SCALE_HEAD_DIM")

    def cache(tokens):
        kq, vq = VAR_Q(qkv_format="BHLc", max_tokens=tokens, **kw), VAR_Q(qkv_format="BHLc", max_tokens=tokens, **kw)
        for c in (kq, vq):
            c.append(torch.randn((1, 2, tokens, 64), generator=gen, device=DEV))
        return kq, vq
    kq, vq = cache(3000)
    q, x = torch.randn((1, 2, 20, 64), generator=gen, device=DEV), torch.randn((8, 3, 2000, 64), generator=gen, device=DEV)

    def work():
        step = VAR_Q(qkv_format="BHLc", max_tokens=2000, **kw)
        step.append(x)
        return attend_cached(q, kq, vq, 0.125), step.cached_item, step.scale
    want = [t.clone() for t in work()]
    assert _cabi.lib().varq_attn_workspace_bytes(1, 2, 20, 3000, 64, 8, 8) > 256, "this call splits its key range"

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        work()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = work()
    # other streams by the dozen, larger calls on the stream of the capture, and then memory of every size that was given back
    kq2, vq2 = cache(9000)
    q2 = torch.randn((1, 2, 500, 64), generator=gen, device=DEV)
    for s in [torch.cuda.Stream() for _ in range(24)] + [side]:
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            work()
            attend_cached(q2, kq2, vq2, 0.125)
    torch.cuda.synchronize()
    held = []
    for s in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(s):
            for shift in range(9, 24):
                held += [torch.full((1 << shift,), 77, dtype=torch.uint8, device=DEV) for _ in range(4)]
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(bool((t == 77).all()) for t in held), "the replay wrote into memory of another tensor"
    assert _cabi.device_status() == 0 and _host is not None
