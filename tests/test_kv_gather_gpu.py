"""Cached rows gathered and new rows placed behind them in one launch."""
import pytest
import torch

from uniserve_v1_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,news,page,Hkv,D", [([37, 20], [3, 9], 16, 2, 128), ([0, 5, 0], [1, 8, 2], 4, 1, 64),
                                                   ([16], [1], 16, 4, 128), ([9, 1], [0, 17], 8, 3, 8)])
def test_new_rows_stand_behind_the_cached_ones(lens, news, page, Hkv, D):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    B, most = len(lens), max((n + page - 1) // page for n in lens) + 1
    pages = torch.randperm(B * most, generator=g, device="cuda").int().view(B, most)
    kc, vc = rnd(B * most, page, Hkv, D), rnd(B * most, page, Hkv, D)
    qkv = rnd(sum(news), (5 + 2 * Hkv) * D).view(sum(news), 5 + 2 * Hkv, D)
    k, v = qkv[:, 5:5 + Hkv], qkv[:, 5 + Hkv:]
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([sum(lens[:i]) for i in range(B + 1)], **i32)
    at = [sum(lens[:i]) + sum(news[:i]) for i in range(B + 1)]
    dst = torch.tensor([a + n + j for a, n, m in zip(at, lens, news) for j in range(m)], device="cuda")
    out = tuple(torch.full((at[-1], Hkv, D), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    F.kv_gather(kc, vc, pages, cu, sum(lens), out=out, out_cu=torch.tensor(at, **i32), new=(k, v, dst))
    for got, cache, new in ((out[0], kc, k), (out[1], vc, v)):
        done = 0
        for s, (n, m) in enumerate(zip(lens, news)):
            rows = cache[pages[s].long()].reshape(-1, Hkv, D)[:n]
            assert torch.equal(got[at[s]:at[s + 1]], torch.cat([rows, new[done:done + m]]))
            done += m
