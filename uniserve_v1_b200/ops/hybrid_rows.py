"""Rows between the products of the hybrid decoder on a GPU (bf16 stream, FP32 norm weights); see
``csrc/hybrid_rows.cu``.  Other types and devices take the model's PyTorch formulas."""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from . import native as N

P, I, L, F = N.P, N.I, N.L, N.F
N.register_signatures({
    "us_hybrid_rows": (I, [P, L, P, L, P, P, P, I, P, P, P, P, P, P, P, I, I, F, P]),
    "us_hybrid_heads": (I, [P, L, P, P, P, P, P, P, I, I, I, I, I, I, F, P]),
    "us_hybrid_gate": (I, [P, P, L, P, I, I, I, P]),
})


@dataclass
class Output:
    """A sublayer's output: its rows, or expert rows in permuted order with every token's places and weights, and
    the shared expert's rows with the logits of their gate."""
    rows: Optional[torch.Tensor] = None
    routed: Optional[torch.Tensor] = None
    perm: Optional[torch.Tensor] = None
    weights: Optional[torch.Tensor] = None
    shared: Optional[torch.Tensor] = None
    shared_gate: Optional[torch.Tensor] = None


def rows_serve(x, w) -> bool:
    """Whether ``add_norm`` takes a model of these: rows in sixteen-byte columns that start on sixteen bytes, a row of
    which a CTA holds."""
    return x.is_cuda and x.dtype == torch.bfloat16 and w.dtype == torch.float32 and x.dim() == 2 and \
        x.shape[1] % 8 == 0 and x.shape[1] <= 8192 and x.is_contiguous() and x.data_ptr() % 16 == 0


def heads_serve(x, D: int) -> bool:
    return x.is_cuda and x.dtype == torch.bfloat16 and D % 8 == 0 and D <= 256


def add_norm(x, out: Optional[Output], w, eps, gate_w=None):
    """x [T, H] plus a sublayer's output, rounded once (x itself without one); its norm times ``w``; the dots of the
    norm with ``gate_w`` [1, H]: (x', y, dots or None)."""
    T, H = x.shape
    o = out or Output()
    new = torch.empty(T, H, dtype=x.dtype, device=x.device) if out is not None else None
    y = torch.empty(T, H, dtype=x.dtype, device=x.device)
    gate = torch.empty(T, dtype=torch.float32, device=x.device) if gate_w is not None else None
    assert x.stride(1) == 1 and (o.rows is None or o.rows.stride(1) == 1)
    for t in (o.routed, o.perm, o.weights, o.shared, o.shared_gate, gate_w):
        assert t is None or t.is_contiguous()
    N.call("us_hybrid_rows", N.ptr(x), x.stride(0), N.ptr(o.rows), o.rows.stride(0) if o.rows is not None else 0,
           N.ptr(o.routed), N.ptr(o.perm), N.ptr(o.weights), o.perm.shape[1] if o.perm is not None else 0,
           N.ptr(o.shared), N.ptr(o.shared_gate), N.ptr(w), N.ptr(gate_w), N.ptr(new), N.ptr(y), N.ptr(gate), T, H,
           eps, N.stream())
    return x if new is None else new, y, gate


def heads(proj, qw, kw, inv_freq, pos0: int, Hq: int, Hk: int, D: int, rot: int, eps: float):
    """Normed, turned queries [T, Hq, D] and keys [T, Hk, D] and the values of ``proj`` [T, (2 Hq + 2 Hk) D]: Hq pairs
    of query and gate, keys, values.  Row t stands at position pos0 + t."""
    T = proj.shape[0]
    assert proj.stride(1) == 1 and proj.shape[1] == (2 * Hq + 2 * Hk) * D
    assert qw.dtype == kw.dtype == inv_freq.dtype == torch.float32
    q, k, v = (torch.empty(T, h, D, dtype=proj.dtype, device=proj.device) for h in (Hq, Hk, Hk))
    N.call("us_hybrid_heads", N.ptr(proj), proj.stride(0), N.ptr(qw), N.ptr(kw), N.ptr(inv_freq), N.ptr(q), N.ptr(k),
           N.ptr(v), T, pos0, Hq, Hk, D, rot, eps, N.stream())
    return q, k, v


def gate(att, proj, Hq: int, D: int):
    """att [T, Hq * D] times the sigmoid of the gates that stand behind every query of ``proj``."""
    assert att.is_contiguous() and att.dtype == proj.dtype
    out = torch.empty_like(att)
    N.call("us_hybrid_gate", N.ptr(att), N.ptr(proj), proj.stride(0), N.ptr(out), att.shape[0], Hq, D, N.stream())
    return out
