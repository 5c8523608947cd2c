"""The delta rules sixteen tokens at a time, and token by token where there are few, against the recurrence in 64 bits, at
the edges of chunks, tiles and widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["chunks", "tokens"])
def route(request, monkeypatch):
    """Both kernels, whatever the sizes."""
    from uniserve_v1_b200.ops import vector_delta as VD
    monkeypatch.setattr(VD, "few_tokens", lambda *a: request.param == "tokens")
    return request.param


def _inputs(lens, H, Hk, D, V, rate, per_channel):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T = sum(lens)
    q, k = (torch.nn.functional.normalize(rnd(T, Hk, D) + 0.3, dim=-1) for _ in range(2))
    shape = (T, H, D) if per_channel else (T, H)
    decay = torch.exp(-rate * torch.rand(*shape, generator=g, device="cuda"))
    return q * D ** -0.5, k, rnd(T, H, V), decay, torch.rand(T, H, generator=g, device="cuda"), rnd(len(lens) + 1, H, D, V)


def _recurrence(q, k, v, g, beta, S, lens, fresh):
    q, k, v, g, beta, S = (t.double() for t in (q, k, v, g, beta, S))
    rep = v.shape[1] // q.shape[1]
    q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
    g = g if g.dim() == 3 else g[:, :, None]
    out, at = torch.zeros_like(v), 0
    for s, n in enumerate(lens):
        if fresh[s]:
            S[s] = 0
        for t in range(at, at + n):
            S[s] *= g[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S[s], k[t]))
            S[s] += k[t][:, :, None] * u[:, None]
            out[t] = torch.einsum("hdv,hd->hv", S[s], q[t])
        at += n
    return out, S


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("lens,H,Hk,D,V,rate", [
    ([1], 2, 1, 128, 128, 0.5), ([15, 16, 17], 4, 2, 128, 128, 0.3), ([33, 1, 31], 2, 2, 64, 64, 0.05),
    ([200], 6, 3, 128, 128, 4.0), ([18, 5], 2, 1, 40, 36, 0.3), ([34], 2, 1, 256, 256, 0.1),
    ([23, 49], 2, 1, 30, 33, 0.1), ([17], 1, 1, 132, 4, 30.0), ([600], 2, 1, 128, 32, 0.001)])
def test_chunks_follow_the_recurrence(lens, H, Hk, D, V, rate, per_channel, route):
    from uniserve_v1_b200.ops import vector_delta as VD
    q, k, v, g, beta, S = _inputs(lens, H, Hk, D, V, rate, per_channel)
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], **i32)
    fresh = [i % 2 == 1 for i in range(len(lens))]
    pos = torch.cat([torch.arange(n, **i32) + (0 if f else 7) for n, f in zip(lens, fresh)])
    slots = torch.arange(len(lens), **i32)
    want, state = _recurrence(q, k, v, g, beta, S, lens, fresh)
    m = VD.SeqMeta(cu, slots, pos, False)
    got = VD.vector_delta_rule(q, k, v, g, S, m, beta=beta)
    torch.cuda.synchronize()
    # a token rounds every number of a state a few times (2^-25 each on average); over the 600 tokens that the slowest
    # decay here remembers, a random sum of some 60 of them
    for a, b in ((got, want), (S, state)):
        assert float((a.double() - b).norm() / b.norm()) < 5e-7
    assert torch.equal(S[-1].double(), state[-1])              # a slot that no sequence has


def _recurrence_fp32(q, k, v, g, beta, S):
    """Token by token in FP32, one sequence: what the rounding of each operation leaves."""
    rep = v.shape[1] // q.shape[1]
    q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
    g = g if g.dim() == 3 else g[:, :, None]
    out = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out, S


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("T,D,V,rate", [(16, 128, 128, 0.05), (200, 64, 64, 0.001), (500, 128, 128, 0.05),
                                         (500, 128, 128, 1.0), (300, 256, 64, 0.3), (200, 40, 36, 1.0)])
def test_no_further_off_than_fp32(T, D, V, rate, per_channel, route):
    """Operands in parts on the tensor cores against the same recurrence in FP32: as close to 64 bits (a sixth more is
    left for which values the two round differently)."""
    from uniserve_v1_b200.ops import vector_delta as VD
    q, k, v, g, beta, S = _inputs([T], 4, 2, D, V, rate, per_channel)
    S = S[:1].contiguous()
    want, state = _recurrence(q, k, v, g, beta, S.clone(), [T], [False])
    plain, plain_state = _recurrence_fp32(q, k, v, g, beta, S[0])
    i32 = dict(dtype=torch.int32, device="cuda")
    m = VD.SeqMeta(torch.tensor([0, T], **i32), torch.zeros(1, **i32), torch.arange(T, **i32) + 7, False)
    got = VD.vector_delta_rule(q, k, v, g, S, m, beta=beta)
    off = lambda a, b: float((a.double() - b).norm() / b.norm())
    assert off(got, want) < 1.17 * off(plain, want)
    assert off(S[0], state[0]) < 1.17 * off(plain_state, state[0])


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("where", ["v", "k", "q", "g"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_not_finite_stays_with_later_tokens(where, bad, per_channel, route):
    """A token that is not finite in the middle of a chunk: tokens before it, and for a value the other columns, are what
    they are without it."""
    from uniserve_v1_b200.ops import vector_delta as VD
    T, at, head, D, V = 40, 21, 1, 64, 40
    i32 = dict(dtype=torch.int32, device="cuda")
    m = VD.SeqMeta(torch.tensor([0, T], **i32), torch.zeros(1, **i32), torch.arange(T, **i32) + 7, False)
    outs = []
    for spoiled in (False, True):
        q, k, v, g, beta, S = _inputs([T], 2, 2, D, V, 0.3, per_channel)
        if spoiled:
            x = dict(q=q, k=k, v=v, g=g)[where]
            x[(at, head) if x.dim() == 2 else (at, head, 5)] = bad
        S = S[:1].contiguous()
        outs.append((VD.vector_delta_rule(q, k, v, g, S, m, beta=beta), S))
    (clean, S0), (got, S1) = outs
    # the sums of a tile without its later tokens are taken in another order: FP32 sums of 16 products
    near = lambda a, b: torch.allclose(a, b, rtol=0, atol=16 * 2.0 ** -24 * float(clean.abs().max()))
    assert near(got[:at], clean[:at]) and torch.equal(got[:, 0], clean[:, 0])
    if where == "v":
        others = [c for c in range(V) if c != 5]
        assert near(got[:, head, others], clean[:, head, others])
        assert not bool(torch.isfinite(got[at:, head, 5]).any()) and not bool(torch.isfinite(S1[0, head, :, 5]).any())
        assert bool(torch.isfinite(S1[0, head][:, others]).all())
    elif where == "q":
        assert near(got[at + 1:], clean[at + 1:]) and torch.equal(S1, S0)
        assert not bool(torch.isfinite(got[at, head]).any())
    else:
        assert not bool(torch.isfinite(got[at:, head]).any())


@pytest.mark.parametrize("lens,H,D,per_channel,names", [
    ([48], 32, 128, False, ["us_token_delta_rule"]), ([49], 32, 128, False, ["us_head_delta_rule"]),
    ([1] * 7, 4, 64, True, ["us_token_delta_rule"]), ([65], 4, 64, True, ["us_channel_delta_rule"]),
    ([1] * 63 + [200], 2, 128, True, ["us_channel_delta_rule"]), ([80] * 3, 128, 64, True, ["us_token_delta_rule"])])
def test_route(lens, H, D, per_channel, names, monkeypatch):
    """Which kernel runs, with the lengths on the host and, from the number of rows alone, without."""
    from uniserve_v1_b200.ops import native as N
    from uniserve_v1_b200.ops import vector_delta as VD
    q, k, v, g, beta, S = _inputs(lens, H, H, D, D, 0.3, per_channel)
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], **i32)
    pos = torch.cat([torch.arange(n, **i32) + 7 for n in lens])
    m = VD.SeqMeta(cu, torch.arange(len(lens), **i32), pos, False, [7] * len(lens), lens)
    called, call = [], N.call
    monkeypatch.setattr(N, "call", lambda name, *a, **kw: (called.append(name), call(name, *a, **kw))[1])
    S0 = S.clone()
    out = VD.vector_delta_rule(q, k, v, g, S, m, beta=beta)
    assert called == names
    bare = VD.SeqMeta(cu, m.slots, pos, False)
    again = VD.vector_delta_rule(q, k, v, g, S0, bare, beta=beta)
    # two kernels, each within the bound above of 64 bits
    assert float((out - again).norm() / out.norm()) < 1e-6 and float((S - S0).norm() / S.norm()) < 1e-6
