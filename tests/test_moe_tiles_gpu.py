"""Experts of a few tokens on the weight-streaming kernel, and the rows per tile that the averages choose."""
import pytest
import torch

from uniserve_v1_b200.ops import functional as F
from uniserve_v1_b200.ops import native as N
from uniserve_v1_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,top,H,I", [(1, 8, 8, 2048, 768), (1, 64, 4, 256, 256), (2, 16, 8, 512, 256),
                                          (17, 4, 2, 256, 512), (16, 1, 1, 768, 256), (5, 6, 3, 1024, 768)])
def test_streamed_experts(T, E, top, H, I, monkeypatch):
    """Against the formula and the tensor-memory kernels; one tile holds up to 16 rows of an expert."""
    g = torch.Generator(device="cuda").manual_seed(T * 7 + E)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w13, w2 = rnd(T, H), rnd(E, 2 * I, H) * H ** -0.5, rnd(E, H, I) * I ** -0.5
    ids, w = F.topk_softmax(torch.randn(T, E, generator=g, device="cuda"), top, True)
    ws = F.MoeWorkspace.create(T, top, E, H, I, "cuda", block_n=16)
    calls = []
    call = N.call
    monkeypatch.setattr(N, "call", lambda name, *a, **k: (calls.append(name), call(name, *a, **k))[1])
    monkeypatch.setattr(F, "MOE_STREAM_WEIGHTS", 1 << 40)
    out = F.moe_experts(x, ids, w, w13, w2, ws=ws)
    assert calls.count("us_linear_decode_grouped") == 2
    monkeypatch.setattr(F, "MOE_STREAM_WEIGHTS", 0)
    other = F.moe_experts(x, ids, w, w13, w2, ws=ws)
    assert calls.count("us_linear_decode_grouped") == 2
    torch.cuda.synchronize()
    N.raise_on_device_error()
    want = R.moe_experts(x.float(), ids, w, w13.float(), w2.float())
    # bf16 between the products and at the end (2^-8 each), FP32 sums of at most 2048 products
    assert float((out.float() - want).norm() / want.norm()) < 2 ** -7
    assert float((out.float() - other.float()).norm() / want.norm()) < 2 ** -7


@pytest.mark.parametrize("T,E,top,rows", [(1, 128, 8, 16), (63, 128, 8, 16), (64, 128, 8, 32), (500, 128, 8, 32),
                                           (1535, 128, 8, 32), (1536, 128, 8, 256), (96, 1, 1, 256), (95, 1, 1, 32)])
def test_rows_per_tile(T, E, top, rows):
    ws = F.MoeWorkspace.create(T, top, E, 64, 64, "cuda")
    assert ws.block_n == rows and ws.max_tiles * rows >= T * top
    # at most a partial tile per expert
    assert ws.max_tiles >= min(T * top, E) + T * top // rows
