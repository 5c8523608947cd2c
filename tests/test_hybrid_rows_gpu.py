"""Rows between the hybrid decoder's products against the same formulas in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _near(got, want, steps=1.0):
    """Within ``steps`` roundings to bf16 (2^-8 of the value each) and FP32 sums of values of order one."""
    err = (got.double() - want).abs()
    assert bool((err <= steps * 2.0 ** -8 * want.abs() + 2e-5).all()), float(err.max())


@pytest.mark.parametrize("T,H,top", [(1, 8, 1), (3, 64, 0), (5, 2048, 4), (2, 2056, 2), (7, 4104, 8), (2, 8192, 1)])
def test_add_norm(T, H, top):
    from uniserve_v1_b200.ops import hybrid_rows as HR
    g = torch.Generator(device="cuda").manual_seed(H + top)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    wide = rnd(T, H + 8)
    x, add, w, gw = wide[:, 8:], rnd(T, H), torch.rand(H, generator=g, device="cuda") + 0.5, rnd(1, H)
    out = HR.Output(rows=add)
    total = add.double()
    size = total.abs()
    if top:
        routed, wts = rnd(T * top, H), torch.rand(T, top, generator=g, device="cuda")
        perm = torch.randperm(T * top, generator=g, device="cuda").int().view(T, top)
        perm[0, 0] = -1                                       # a route that has no row here
        shared, logit = rnd(T, H), torch.randn(T, generator=g, device="cuda")
        out = HR.Output(rows=None, routed=routed, perm=perm, weights=wts, shared=shared, shared_gate=logit)
        picked = routed.double()[perm.clamp(min=0).long()] * wts.double()[:, :, None] * (perm >= 0)[:, :, None]
        scaled = shared.double() * torch.sigmoid(logit.double())[:, None]
        total, size = picked.sum(1) + scaled, picked.sum(1).abs() + scaled.abs()
    new, y, dots = HR.add_norm(x, out, w, 1e-6, gw)
    # up to four roundings on the way (2^-8 each), none of a value above the parts' sizes together
    bound = 4 * 2.0 ** -8 * (size + x.double().abs()) + 2e-5
    assert bool(((new.double() - x.double() - total).abs() <= bound).all())
    f = new.double()
    want = f * torch.rsqrt((f * f).mean(1, keepdim=True) + 1e-6) * w.double()
    _near(y, want)
    dot = (y.double() * gw.double()).sum(1)
    assert torch.allclose(dots.double(), dot, rtol=1e-5, atol=1e-4 * H ** 0.5)
    same, y2, none = HR.add_norm(x, None, w, 1e-6)
    f = x.double()
    assert same is x and none is None
    _near(y2, f * torch.rsqrt((f * f).mean(1, keepdim=True) + 1e-6) * w.double())


@pytest.mark.parametrize("T,Hq,Hk,D,rot,pos0", [(1, 1, 1, 8, 8, 0), (3, 4, 2, 32, 8, 5), (4, 32, 4, 128, 32, 4000),
                                                 (2, 16, 2, 256, 64, 17), (2, 3, 1, 136, 136, 1), (2, 2, 1, 64, 0, 3)])
def test_heads_and_gate(T, Hq, Hk, D, rot, pos0):
    from uniserve_v1_b200.ops import hybrid_rows as HR
    g = torch.Generator(device="cuda").manual_seed(D + rot)
    proj = torch.randn(T, (2 * Hq + 2 * Hk) * D, generator=g, device="cuda").bfloat16()
    qw, kw = (torch.rand(D, generator=g, device="cuda") + 0.5 for _ in range(2))
    freq = 10000.0 ** (-torch.arange(0, rot, 2, device="cuda").float() / max(rot, 1))
    q, k, v = HR.heads(proj, qw, kw, freq, pos0, Hq, Hk, D, rot, 1e-6)
    pairs = proj[:, :2 * Hq * D].view(T, Hq, 2 * D)
    kv = proj[:, 2 * Hq * D:].view(T, 2 * Hk, D)
    angle = ((pos0 + torch.arange(T, device="cuda")).float()[:, None] * freq).double()   # an FP32 product, as the model's

    def want(x, w):
        f = x.double()
        f = f * torch.rsqrt((f * f).mean(-1, keepdim=True) + 1e-6) * w.double()
        a, b, h = f[..., :rot // 2], f[..., rot // 2:rot], angle[:, None]
        return torch.cat([a * h.cos() - b * h.sin(), b * h.cos() + a * h.sin(), f[..., rot:]], -1)
    _near(q, want(pairs[..., :D], qw))
    _near(k, want(kv[:, :Hk], kw))
    assert torch.equal(v, kv[:, Hk:])
    att = torch.randn(T, Hq * D, generator=g, device="cuda").bfloat16()
    _near(HR.gate(att, proj, Hq, D), att.double() * torch.sigmoid(pairs[..., D:].reshape(T, Hq * D).double()))


@pytest.mark.parametrize("start,stride", [(0, 64), (1, 64), (4, 64), (0, 72)])
def test_embeddings_anywhere(start, stride):
    """Prompt rows of a caller that start on any element, or stand apart, are served like aligned ones."""
    from uniserve_v1_b200.models.qwen3_5 import Qwen35MoeModel
    cfg = Qwen35MoeModel.tiny_config()
    model = Qwen35MoeModel(cfg, "cuda", torch.bfloat16).init_random()
    T, H = 7, cfg.hidden_size
    buf = torch.zeros(start + T * stride, dtype=torch.bfloat16, device="cuda")
    rows = buf[start:].view(T, stride)[:, :H]
    rows.copy_(torch.randn(T, H, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda"))
    ids = torch.zeros(T, dtype=torch.long)
    got = model.forward(ids, model.new_state(), embeds=rows)
    want = model.forward(ids, model.new_state(), embeds=rows.clone(memory_format=torch.contiguous_format))
    # the same sums with other places of rounding to bf16, 2^-9 each, some ten a layer
    assert float((got - want).norm() / want.norm()) < 2.0 ** -5
