"""The packed columns of a prompt batch against a token by token loop."""
import ctypes
import random
from array import array

import pytest

from uniserve_v1_b200.ops import native as N


def _plan(start, length, slots, pages, page):
    """As the library takes them, and what it has to make of them."""
    ids = list(range(7, 7 + sum(length)))
    flat = array("i", start + length + [len(p) for p in pages] + slots + [x for p in pages for x in p])
    pos = [p for a, n in zip(start, length) for p in range(a, a + n)]
    where = [pg[p // page] * page + p % page for pg, a, n in zip(pages, start, length) for p in range(a, a + n)]
    cu_q, cu_k = [0], [0]
    for a, n in zip(start, length):
        cu_q.append(cu_q[-1] + n)
        cu_k.append(cu_k[-1] + a + n)
    return ids, flat, pos, where, cu_q, cu_k


def _run(plan, ids, B, rows, page, most, at, size):
    out, ids = array("i", [-9] * size), array("i", ids)
    rc = N.host().us_batch_rows(*(ctypes.c_void_p(x.buffer_info()[0]) for x in (plan, ids)), B, rows, page, most, at,
                                ctypes.c_void_p(out.buffer_info()[0]))
    return rc, out.tolist()


@pytest.mark.parametrize("B,page,pad,table", [(1, 1, 0, True), (1, 16, 3, False), (5, 16, 0, True), (9, 4, 17, True),
                                              (0, 16, 4, True)])
def test_columns(B, page, pad, table):
    r = random.Random(B * 31 + page)
    start = [r.randrange(0, 40) for _ in range(B)]
    length = [r.randrange(0 if b else 1, 35) for b in range(B)]
    pages = [[r.randrange(1, 999) for _ in range((a + n + page - 1) // page + r.randrange(2))]
             for a, n in zip(start, length)]
    slots, most = list(range(B)), max((len(p) for p in pages), default=0) + 1
    ids, plan, pos, where, cu_q, cu_k = _plan(start, length, slots, pages, page)
    rows = len(ids) + pad
    at = 3 * rows + 2 * (B + 1) + B + 1 + 2
    rc, out = _run(plan, ids, B, rows, page, most if table else 0, at, at + B * most)
    assert rc == 0
    assert out[:rows] == ids + [0] * pad
    assert out[rows:2 * rows] == pos + [0] * pad
    assert out[2 * rows:3 * rows] == where + [-1] * pad
    assert out[3 * rows:at - 2] == cu_q + cu_k + slots + [len(ids)]
    want = [x for p in pages for x in p + [0] * (most - len(p))] if table else [-9] * (B * most)
    assert out[at:] == want and out[at - 2:at] == [-9, -9]


@pytest.mark.parametrize("held,most,bad", [(1, 8, 2), (3, 2, 2)])
def test_pages_that_do_not_hold_the_tokens(held, most, bad):
    """The second request has a page too few, or more than a row of the table takes."""
    start, length, pages = [0, 16], [16, 9], [[4], [5] * held]
    plan = array("i", start + length + [len(p) for p in pages] + [0, 1] + [x for p in pages for x in p])
    rc, _ = _run(plan, list(range(25)), 2, 25, 16, most, 90, 200)
    assert rc == bad


@pytest.mark.parametrize("pages,why", [([1, 2, 3], "3 pages, a row of the page table takes 2"),
                                        ([1], "its pages do not hold its tokens")])
def test_refusal_names_its_reason(pages, why):
    from types import SimpleNamespace

    import torch

    from uniserve_v1_b200.engine.runner import CausalLmRunner
    runner = SimpleNamespace(device=torch.device("cpu"), attends_pages=True, max_pages=2, page_size=4)
    request = SimpleNamespace(token_slice=lambda a, b: [7] * (b - a), pages=pages, slot=0, request_id="r")
    with pytest.raises(IndexError, match=f"request r: {why}"):
        CausalLmRunner._prefill_rows(runner, [SimpleNamespace(start=0, length=6, request=request)])
