"""What the speed of this framework is measured on: forward passes of every served family through the calls
that its engines make (``CausalLmRunner.batch_logits`` for the paged decoders, ``Qwen35MoeModel.forward`` for the
hybrid one, ``H3Transformer.embed_rows`` / ``forward`` for the video transformer).

Layer sizes are those of the families' named configurations and of ``bench.py``; a case keeps a few layers (one of each
kind that the family has) and the benchmark's vocabulary of 32,000, so that the output matrix keeps about the share of
a pass that it has in a whole model.  Weights are random, of unit gain; routers are drawn wider, since trained ones are
decided: the last expert chosen then weighs little, and a token whose choice hangs on rounding moves the outputs by
less than the data types do.  Lengths within a batch are ragged.

* ``prompt``: whole prompts, or what follows ``context`` cached tokens of each request, as one packed batch; logits
  of every request's last token, cache pages and recurrent states.
* ``decode``: the next token of every request from ``context`` tokens; logits, and recurrent states.
* ``step``: one evaluation of the video transformer on a clip; the velocities of all video and audio rows."""
import math

import numpy as np
import torch

from uniserve_v1_b200.engine.runner import CausalLmRunner
from uniserve_v1_b200.engine.scheduler import Batch, Chunk
from uniserve_v1_b200.engine.types import Request, SamplingParams
from uniserve_v1_b200.models.minimax_h3 import H3Block, H3Config, H3Transformer, build_layout
from uniserve_v1_b200.models.nepevik import NepevikConfig, NepevikModel
from uniserve_v1_b200.models.nopuzen import NopuzenConfig, NopuzenModel
from uniserve_v1_b200.models.qwen3_5 import Qwen35Config, Qwen35MoeModel
from uniserve_v1_b200.models.qwen3_moe import Qwen3MoeConfig, Qwen3MoeModel
from uniserve_v1_b200.models.tadinex import GLU_ALPHA, TadinexConfig, TadinexModel
from uniserve_v1_b200.models.zonopel import ZonopelConfig, ZonopelModel

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
VOCAB, PAGE = 32000, 16
ROUTER, DOWN = 6.0, 0.5  # gain of the routers' logits, and of what a routed expert adds to the stream
LAYERED = {"nepevik": (NepevikConfig, NepevikModel), "zonopel": (ZonopelConfig, ZonopelModel),
           "tadinex": (TadinexConfig, TadinexModel), "nopuzen": (NopuzenConfig, NopuzenModel)}
CHUNK = 8192            # rows that an engine hands over at a time (``max_num_batched_tokens`` of the benchmark)


def listed():
    return [
        # one user of a chat service: every launch of a step is in the way of the next token
        _text("chat-decode-1", "qwen3-moe", "decode", 1, 700),
        # the serving benchmark's step: 64 concurrent requests of 1024 tokens and what they have written so far
        _text("chat-decode-64", "qwen3-moe", "decode", 64, 1100),
        # block-scaled FP8 experts at the width of the largest served shape, 256 concurrent requests of 2048 tokens
        _text("chat-decode-256-fp8", "qwen3-moe-235b", "decode", 256, 2200, fp8=True),
        # what the scheduler hands over when requests arrive: eight prompts at once
        _text("chat-prompts", "qwen3-moe", "prompt", 8, 0, 8152),
        # the next turn of three conversations: short messages behind a cached history
        _text("chat-next-turn", "qwen3-moe", "prompt", 3, 1531, 211),
        # a document read by the hybrid decoder
        _text("hybrid-prompt", "qwen3.5", "prompt", 1, 0, 4093),
        _text("nepevik-prompts", "nepevik", "prompt", 2, 0, 8101),
        _text("zonopel-prompts", "zonopel", "prompt", 8, 0, 8152),
        _text("tadinex-prompt", "tadinex", "prompt", 1, 0, 4093),
        _text("tadinex-decode-64", "tadinex", "decode", 64, 300),
        _text("nopuzen-prompts", "nopuzen", "prompt", 4, 0, 8152),
        # one block of a denoising step of the five-second clip
        _video("video-step", 37, 48, 84, 1000),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["qwen3-moe", "qwen3-moe", "qwen3.5", "nepevik", "zonopel", "tadinex", "nopuzen", "h3"])
    if model == "h3":
        return _video("", 5 * rng.randint(0, 6) + 2, 2 * log(8, 24), 2 * log(8, 42), log(32, 1000), nameless=True)
    if model == "qwen3.5":
        return _text("", model, "prompt", 1, 0, log(65, 4093), nameless=True)
    n = log(1, 64)
    if rng.random() < 0.4:
        context = log(64, 2200) if model == "qwen3-moe" else log(64, 16000 // n if n > 8 else 2000)
        return _text("", model, "decode", n, context, nameless=True)
    n = min(n, 16)
    context = log(100, 2000) if model == "qwen3-moe" and rng.random() < 0.5 else 0
    return _text("", model, "prompt", n, context, max(n, log(33, 8152)), nameless=True)


def _text(name, model, phase, requests, context, tokens=0, fp8=False, nameless=False):
    c = {"name": name, "model": model, "phase": phase, "requests": requests, "context": context,
         "tokens": tokens or requests, "fp8": fp8}
    if nameless:
        del c["name"]
    return c


def _video(name, frames, height, width, text, nameless=False):
    c = {"name": name, "model": "h3", "phase": "step", "frames": frames, "height": height, "width": width, "text": text}
    if nameless:
        del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ shapes --
def _config(case):
    m = case["model"]
    if m == "qwen3-moe":
        return Qwen3MoeConfig(vocab_size=VOCAB, num_hidden_layers=4, eos_token_id=VOCAB - 1)
    if m == "qwen3-moe-235b":
        c = Qwen3MoeConfig.qwen3_235b_a22b()
        c.vocab_size, c.num_hidden_layers, c.eos_token_id = VOCAB, 2, VOCAB - 1
        return c
    if m == "qwen3.5":
        return Qwen35Config(vocab_size=VOCAB, hidden_size=2048, num_hidden_layers=4, num_attention_heads=32,
                            num_key_value_heads=4, head_dim=128, linear_num_key_heads=16, linear_num_value_heads=32,
                            num_experts=64, num_experts_per_tok=4, moe_intermediate_size=768,
                            shared_expert_intermediate_size=1024, eos_token_id=VOCAB - 1,
                            layer_types=["linear_attention"] * 3 + ["full_attention"])
    if m == "h3":
        return H3Config(num_layers=1, refiner_layers=0)
    c = LAYERED[m][0].bench(4)
    c.vocab_size = VOCAB
    return c


def _spread(n, total):
    """``n`` unlike lengths, at least 1, of ``total`` tokens in all."""
    w = [0.4 + 1.2 * ((i * 0.618034 + 0.3) % 1.0) for i in range(n)]
    out = [max(1, int((total - n) * x / sum(w)) + 1) for x in w]
    out[0] += max(0, total - sum(out))
    return out


def _contexts(case):
    n, c = case["requests"], case["context"]
    return [0] * n if not c else [c] if n == 1 else _spread(n, n * c)


def _counts(case):
    """Tokens of this pass per request."""
    return [1] * case["requests"] if case["phase"] == "decode" else _spread(case["requests"], case["tokens"])


def _recurrent(case):
    return case["model"] in ("nepevik", "zonopel", "tadinex")


def _tokens(case, seed):
    """Per request all its tokens, those of the context first."""
    r = np.random.RandomState((seed * 7919 + 17) % (1 << 31))
    return [r.randint(0, VOCAB - 1, a + b).tolist() for a, b in zip(_contexts(case), _counts(case))]


# ----------------------------------------------------------------------------------------------- weights --
class _Draw:
    """A checkpoint's tensors drawn at random on the GPU; also the loader that the models read it through."""

    def __init__(self, seed):
        self.g, self.t = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1), {}

    def get(self, n):
        return self.t[n]

    def has(self, n):
        return n in self.t

    def names(self):
        return list(self.t)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def lin(self, n, *shape, gain=1.0):
        self.t[n] = (self.randn(*shape).mul_(gain * shape[-1] ** -0.5)).to(BF16)

    def around(self, n, width, mean=1.0, std=0.1, dtype=BF16):
        self.t[n] = (self.randn(width) * std + mean).to(dtype)


def _weights(case, seed):
    d, c = _Draw(seed), _config(case)
    {"qwen3-moe": _qwen_weights, "qwen3-moe-235b": _qwen_weights, "qwen3.5": _hybrid_weights, "nepevik": _nepevik_weights,
     "zonopel": _zonopel_weights, "tadinex": _tadinex_weights, "nopuzen": _nopuzen_weights, "h3": _h3_weights}[case["model"]](d, c)
    return d


def _qwen_weights(d, c):
    H, D, I, E = c.hidden_size, c.head_dim, c.moe_intermediate_size, c.num_experts
    d.lin("model.embed_tokens.weight", VOCAB, H, gain=H ** 0.5)
    d.lin("lm_head.weight", VOCAB, H)
    d.around("model.norm.weight", H)
    for i in range(c.num_hidden_layers):
        p = f"model.layers.{i}."
        d.around(p + "input_layernorm.weight", H)
        d.around(p + "post_attention_layernorm.weight", H)
        for n, k in (("q", c.num_attention_heads), ("k", c.num_key_value_heads), ("v", c.num_key_value_heads)):
            d.lin(p + f"self_attn.{n}_proj.weight", k * D, H)
        d.lin(p + "self_attn.o_proj.weight", H, c.num_attention_heads * D)
        d.around(p + "self_attn.q_norm.weight", D)
        d.around(p + "self_attn.k_norm.weight", D)
        d.lin(p + "mlp.gate.weight", E, H, gain=ROUTER)
        d.lin(p + "mlp.experts.gate_up_proj", E, 2 * I, H)
        d.lin(p + "mlp.experts.down_proj", E, H, I, gain=DOWN)


def _hybrid_weights(d, c):
    H, D, I, E, S = (c.hidden_size, c.head_dim, c.moe_intermediate_size, c.num_experts,
                     c.shared_expert_intermediate_size)
    kd, vd, Hv = (c.linear_num_key_heads * c.linear_key_head_dim, c.linear_num_value_heads * c.linear_value_head_dim,
                  c.linear_num_value_heads)
    d.lin("model.embed_tokens.weight", VOCAB, H, gain=H ** 0.5)
    d.lin("lm_head.weight", VOCAB, H)
    d.around("model.norm.weight", H, 0.0)
    for i, kind in enumerate(c.layer_types):
        p = f"model.layers.{i}."
        d.around(p + "input_layernorm.weight", H, 0.0)
        d.around(p + "post_attention_layernorm.weight", H, 0.0)
        if kind == "full_attention":
            a = p + "self_attn."
            d.lin(a + "q_proj.weight", c.num_attention_heads * 2 * D, H)
            d.lin(a + "k_proj.weight", c.num_key_value_heads * D, H)
            d.lin(a + "v_proj.weight", c.num_key_value_heads * D, H)
            d.lin(a + "o_proj.weight", H, c.num_attention_heads * D)
            d.around(a + "q_norm.weight", D, 0.0)
            d.around(a + "k_norm.weight", D, 0.0)
        else:
            a = p + "linear_attn."
            for n, k in (("qkv", 2 * kd + vd), ("z", vd), ("b", Hv), ("a", Hv)):
                d.lin(a + f"in_proj_{n}.weight", k, H)
            d.lin(a + "conv1d.weight", 2 * kd + vd, 1, c.linear_conv_kernel_dim)
            d.around(a + "dt_bias", Hv, -3.0, 1.0)
            d.around(a + "A_log", Hv, 0.0, 0.5)
            d.around(a + "norm.weight", c.linear_value_head_dim)
            d.lin(a + "out_proj.weight", H, vd)
        m = p + "mlp."
        d.lin(m + "gate.weight", E, H, gain=ROUTER)
        d.lin(m + "experts.gate_up_proj", E, 2 * I, H)
        d.lin(m + "experts.down_proj", E, H, I, gain=DOWN)
        d.lin(m + "shared_expert.up_proj.weight", S, H)
        d.lin(m + "shared_expert.gate_proj.weight", S, H)
        d.lin(m + "shared_expert.down_proj.weight", H, S)
        d.lin(m + "shared_expert_gate.weight", 1, H)


def _experts(d, m, n, ff, W, gated):
    """Expert by expert, as checkpoints name them (views of one draw)."""
    for part, shape in (("up", (n, ff, W)), ("down", (n, W, ff))) + ((("gate", (n, ff, W)),) if gated else ()):
        d.lin("stack", *shape, gain=DOWN if part == "down" else 1.0)
        for j, t in enumerate(d.t.pop("stack")):
            d.t[m + f"e{j}.{part}"] = t


def _nepevik_weights(d, c):
    W = c.hidden_size
    d.lin("embed", VOCAB, W, gain=W ** 0.5)
    d.lin("head", VOCAB, W)
    d.t["final.norm"] = torch.tensor(1.0, dtype=BF16, device="cuda")
    for i, L in enumerate(c.layers):
        s, p = L.mixer, f"l{i}.mix."
        H, Hk, D, V = s.heads, s.kv_heads, s.dim, s.vdim
        if s.kind == "channel_delta":
            for n, ch in (("q", Hk * D), ("k", Hk * D), ("v", H * V)):
                d.lin(p + n, ch, W)
                d.lin(p + n + ".conv", ch, s.conv)
            d.lin(p + "b", H, W)
            d.lin(p + "a1", D, W)
            d.lin(p + "a2", H * D, D)
            d.lin(p + "g1", D, W)
            d.lin(p + "g2", H * V, D)
            d.around(p + "A_log", H, 0.0, 0.5)
            d.around(p + "dt_bias", H * D, -3.0, 1.0)
            d.around(p + "norm", V)
        elif s.kind == "general_delta":
            for n in "rkvga":
                d.lin(p + n, H * D, W)
            d.lin(p + "w1", D, W)
            d.lin(p + "w2", H * D, D)
            d.around(p + "a.b", H * D, 0.0, 0.5)
            d.around(p + "w0", H * D, -3.0, 1.0)
            d.around(p + "norm", H * D)
        else:
            d.lin(p + "q", H * D, W)
            d.lin(p + "k", Hk * D, W)
            d.lin(p + "v", Hk * V, W)
            d.around(p + "q.norm", H * D)
            d.around(p + "k.norm", Hk * D)
            d.t[p + "talk"] = (torch.eye(H, device="cuda") * 0.8 + d.randn(H, H) * 0.3 * H ** -0.5).to(BF16)
        d.lin(p + "o", W, H * V)
        for n in ("norm1", "norm2"):
            d.t[f"l{i}.{n}"] = torch.tensor(0.75, dtype=BF16, device="cuda")
        m, e = f"l{i}.mlp.", L.mlp
        _experts(d, m, e.experts, e.ff, W, False)
        d.t[m + "table"] = torch.rand(VOCAB, e.experts, generator=d.g, device="cuda").argsort(1)[:, :e.top].to(
            torch.int32).contiguous()
        d.lin(m + "shared.up", e.shared_ff, W)
        d.lin(m + "shared.down", W, e.shared_ff)
        d.lin(m + "shared.sg", 1, W)


def _latent_weights(d, p, s, W, gate=False):
    d.lin(p + "dq", s.q_rank, W)
    d.around(p + "dq.norm", s.q_rank)
    d.lin(p + "uq", s.heads * (s.dim + s.rot_dim), s.q_rank)
    d.lin(p + "dkv", s.kv_rank + s.rot_dim, W)
    d.around(p + "dkv.norm", s.kv_rank)
    d.lin(p + "uk", s.heads * s.dim, s.kv_rank)
    d.lin(p + "uv", s.heads * s.vdim, s.kv_rank)
    d.lin(p + "o", W, s.heads * s.vdim)
    if gate:
        d.lin(p + "g", s.heads * s.vdim, W)


def _zonopel_weights(d, c):
    W = c.hidden_size
    d.lin("embed", VOCAB, W, gain=W ** 0.5)
    d.lin("bigram", c.bigram.buckets + 1, W, gain=W ** 0.5)
    d.lin("head", VOCAB, W)
    d.around("embed.norm", W)
    d.around("final.norm", W)
    for i, L in enumerate(c.layers):
        if L.weights_of is not None:
            continue
        p, s, m = f"l{i}.mix.", L.mixer, f"l{i}.mlp."
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            d.around(f"l{i}.{n}", W)
        d.around(f"l{i}.shift", W, 0.3, 0.2)
        if L.kind == "mamba2":
            d.lin(p + "in", s.inner + s.channels + s.heads, W)
            d.lin(p + "conv", s.channels, s.taps)
            d.around(p + "conv.b", s.channels, 0.0)
            d.around(p + "dt_bias", s.heads, -3.0, 1.0)
            d.around(p + "A_log", s.heads, 0.0, 1.0)
            d.around(p + "D", s.heads, 1.0, 0.2)
            d.around(p + "norm", s.inner)
            d.lin(p + "o", W, s.inner)
        else:
            _latent_weights(d, p, s, W)
        d.lin(m + "up", L.ff, W)
        d.lin(m + "down", W, L.ff)
        d.around(m + "act", 4, 0.4, 0.2)


def _tadinex_weights(d, c):
    W = c.hidden_size
    d.lin("embed", VOCAB, W, gain=W ** 0.5)
    d.lin("head", VOCAB, W)
    d.around("final.norm", W, 0.0)
    for i, L in enumerate(c.layers):
        p, s, m, e = f"l{i}.mix.", L.mixer, f"l{i}.mlp.", L.moe
        d.around(f"l{i}.norm1", W, 0.0)
        d.around(f"l{i}.norm2", W, 0.0)
        if L.kind == "delta":
            H, nq, nv = s.heads, s.kv_heads * s.dim, s.heads * s.vdim
            for n, ch in (("q", nq), ("k", nq), ("v", nv)):
                d.lin(p + n, ch, W)
                d.lin(p + n + ".conv", ch, s.conv)
            d.lin(p + "b", H, W)
            d.lin(p + "a", H, W)
            d.lin(p + "g", nv, W)
            d.around(p + "A_log", H, 0.0, 0.5)
            d.around(p + "dt_bias", H, -3.0, 1.0)
            d.around(p + "norm", s.vdim)
            d.lin(p + "o", W, nv)
        else:
            a, b = s.left, s.right
            d.lin(p + "left.q", a.heads * a.dim, W)
            d.lin(p + "left.k", a.kv_heads * a.dim, W)
            d.around(p + "left.q.norm", a.dim)
            d.around(p + "left.k.norm", a.dim)
            d.around(p + "left.sink", a.heads, 0.0, 1.0)
            d.lin(p + "left.o", W, a.heads * a.vdim)
            for n, k in (("q", b.state), ("k", b.state), ("v", b.vdim), ("g", b.vdim)):
                d.lin(p + "right." + n, b.heads * k, W)
            d.around(p + "right.norm", b.inner)
            d.lin(p + "right.o", W, b.inner)
        d.lin(m + "router", e.experts + e.identity, W, gain=ROUTER)
        d.around(m + "correction", e.experts + e.identity, 0.0, 0.002)
        _experts(d, m, e.experts, e.ff, W, True)
        for n, shape in (("up", (e.shared_ff, W)), ("gate", (e.shared_ff, W)), ("down", (W, e.shared_ff))):
            d.lin(m + "shared." + n, *shape)


def _nopuzen_weights(d, c):
    W = c.hidden_size

    def norm(n):
        d.around(n, W)
        d.around(n + ".b", W, 0.0)
    d.lin("embed", VOCAB, W)
    norm("final.norm")
    for i, L in enumerate(c.layers):
        p, s, m, e = f"l{i}.mix.", L.mixer, f"l{i}.mlp.", L.moe
        norm(f"l{i}.norm1")
        norm(f"l{i}.norm2")
        if L.kind == "attention":
            for n, k in (("q", s.heads * s.dim), ("k", s.kv_heads * s.dim), ("v", s.kv_heads * s.vdim)):
                d.lin(p + n, k, W)
                d.around(p + n + ".b", k, 0.0)
            d.around(p + "q.norm", s.dim)
            d.around(p + "k.norm", s.dim)
            d.around(p + "temp", s.heads)
            d.around(p + "pb", s.heads, -6.0, 0.5)
            d.lin(p + "g", s.heads, W)
            d.lin(p + "o", W, s.heads * s.vdim)
            d.around(p + "o.b", W, 0.0)
        else:
            _latent_weights(d, p, s, W, True)
        if L.ff:
            d.lin(m + "up", L.ff, W)
            d.lin(m + "down", W, L.ff)
            d.around(m + "act", 2, -1.0, 0.3)
        else:
            d.lin(m + "router", e.experts, W, gain=ROUTER / 3)      # reads the stream itself, which is about 3 wide
            _experts(d, m, e.experts, e.ff, W, False)
            d.lin(m + "shared.up", e.shared_ff, W)
            d.lin(m + "shared.down", W, e.shared_ff)
            d.lin(m + "shared.sg", 1, W)


def _h3_weights(d, c):
    H, inner, Fn = c.hidden_size, c.num_heads * c.head_dim, c.ffn_size
    for n, shape in (("qkv", (3 * inner, H)), ("to_out", (H, inner)), ("ff1", (2 * Fn, H)), ("ff2", (H, Fn))):
        d.lin(n, *shape)
    d.around("q_norm", c.head_dim)
    d.around("k_norm", c.head_dim)
    for n, shape in (("proj_in", (H, c.patch_width)), ("audio_proj_in", (H, c.audio_channels)),
                     ("proj_out", (c.patch_width, H)), ("audio_proj_out", (c.audio_channels, H))):
        d.t[n] = d.randn(*shape) * shape[1] ** -0.5
    d.t["table"], d.t["table_out"] = d.randn(12 * 6, H) * 0.3, d.randn(12 * 2, H) * 0.3


# ----------------------------------------------------------------------------------------------- prepare --
def _video_inputs(case, seed, c):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2)
    n_audio = c.audio_rows(17 * ((case["frames"] - 2) // 5) + 5)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")
    return (randn(c.latent_channels, case["frames"], case["height"], case["width"]), randn(n_audio, c.audio_channels),
            randn(case["text"], c.hidden_size).to(BF16))


def _pages_of(case, seed, lengths):
    """Page ids per request, in no order (page 0 is the padding page); and how many pages there are."""
    need = [(n + PAGE) // PAGE for n in lengths]
    order = (np.random.RandomState((seed * 31 + 5) % (1 << 31)).permutation(sum(need)) + 1).tolist()
    ends = np.cumsum(need).tolist()
    return [order[b - a:b] for a, b in zip(need, ends)], sum(need) + 1


def prepare(case, seed):
    c, d = _config(case), _weights(case, seed)
    if case["model"] == "h3":
        m = H3Transformer(c, "cuda")
        for n in ("proj_in", "audio_proj_in", "proj_out", "audio_proj_out"):
            setattr(m, n, d.t[n])
        m.blocks = [H3Block(*(d.t[n] for n in ("qkv", "q_norm", "k_norm", "to_out", "ff1", "ff2")))]
        m.tables, m.tables_out = [[d.t["table"]]], [d.t["table_out"]]
        video, audio, text = _video_inputs(case, seed, c)
        layout = build_layout(c, case["frames"], case["height"], case["width"], audio.shape[0], case["text"], device="cuda")
        return {"kind": "video", "model": m, "layout": layout, "video": video, "audio": audio, "text": text}
    rows = _tokens(case, seed)
    if case["model"] == "qwen3.5":
        m = Qwen35MoeModel(c, "cuda").load_state(d)
        return {"kind": "hybrid", "model": m, "ids": torch.tensor(rows[0], device="cuda")}
    if case["model"].startswith("qwen3-moe"):
        m = Qwen3MoeModel(c, "cuda", expert_quant="fp8_block" if case["fp8"] else None).load_state(d)
    else:
        m = LAYERED[case["model"]][1](c, "cuda").load_state(d)
    del d
    longest = max(len(t) for t in rows)
    pages, n_pages = _pages_of(case, seed, [len(t) for t in rows])
    runner = CausalLmRunner(m, n_pages, PAGE, max_num_seqs=len(rows), max_model_len=(longest + 128) // PAGE * PAGE)
    sp = SamplingParams(temperature=0.0)
    reqs = [Request(f"r{i}", t, sp, pages=p, slot=i) for i, (t, p) in enumerate(zip(rows, pages))]
    contexts, counts = _contexts(case), _counts(case)
    if any(contexts):
        if case["model"].startswith("qwen3-moe"):
            _fill(runner.kv_caches, seed)
        else:                               # recurrent states and latents come from the context itself
            todo = [Chunk(r, 0, n, False) for r, n in zip(reqs, contexts)]
            while todo:
                part = [todo.pop()]
                while todo and sum(x.length for x in part) + todo[-1].length <= CHUNK:
                    part.append(todo.pop())
                runner.batch_logits(Batch("prefill", part), [[] for _ in part])
    batch = Batch("decode" if case["phase"] == "decode" else "prefill",
                  [Chunk(r, a, n, True) for r, a, n in zip(reqs, contexts, counts)])
    return {"kind": case["phase"], "runner": runner, "batch": batch, "want": [[n - 1] for n in counts]}


def _fill(planes, seed):
    """Cached keys (normed and turned: unit size) and values."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2)
    for k, v in planes:
        for t in (k, v):
            t.view(-1).copy_(torch.randn(t.numel(), generator=g, device="cuda", dtype=BF16))


def run(state):
    if state["kind"] == "video":
        m, layout = state["model"], state["layout"]
        h = m.embed_rows(layout, state["video"], state["audio"], state["text"])
        return dict(zip(("video", "audio"), m.forward(h, layout, 0)))
    if state["kind"] == "hybrid":
        states = state["model"].new_state()
        logits = state["model"].forward(state["ids"], states)
        return {"logits": logits, "states": [t for s in states for t in (s.k, s.v, s.conv, s.rule) if t is not None]}
    runner = state["runner"]
    logits = runner.batch_logits(state["batch"], state["want"])
    states = [t for s in runner.states or [] for t in s if t is not None]
    if state["kind"] == "decode":
        return {"logits": logits, "states": states}
    return {"logits": logits, "pages": [t for kv in runner.kv_caches for t in kv if t is not None], "states": states}


# -------------------------------------------------------------------------------------- what it comes to --
def _seen(case, window=0, keep=0):
    """Keys that the pass's rows look at, over all requests."""
    n = 0
    for a, b in zip(_contexts(case), _counts(case)):
        if not window:
            n += b * a + b * (b + 1) // 2
        else:
            n += sum(min(p + 1, window) + min(keep, max(0, p + 1 - window)) for p in range(a, a + b))
    return n


def _cached(case, window=0):
    return sum(min(a, window - 1) if window else a for a in _contexts(case))


def _mix(T, top, n, ff, W, mats, byte=2):
    """(multiply-adds, bytes of weights) of routed experts: those that T tokens touch."""
    hit = n * (1.0 - (1.0 - top / n) ** T)
    return T * top * mats * ff * W, hit * mats * ff * W * byte


def work(case):
    """Weights that a pass touches, cached keys that it reads, keys and states that it writes, tokens in, logits out."""
    c = _config(case)
    if case["model"] == "h3":
        layout = build_layout(c, case["frames"], case["height"], case["width"],
                              c.audio_rows(17 * ((case["frames"] - 2) // 5) + 5), case["text"])
        T, H, inner = layout.used, c.hidden_size, c.num_heads * c.head_dim
        w = H * (4 * inner + 3 * c.ffn_size)
        io = c.patch_width * H
        return {"bytes": 2 * w + 8 * layout.n_video * c.patch_width + 2 * case["text"] * H,
                "flops": 2 * (T * w + 2 * layout.n_video * io + 2 * T * T * inner)}
    T, n = sum(_counts(case)), case["requests"]
    W = c.hidden_size
    mac = (T if case["model"] == "qwen3.5" else n) * VOCAB * W
    byte = 2 * VOCAB * W + 4 * (mac // W) + 2 * T * W

    def dense(o, i, rows=T):
        nonlocal mac, byte
        mac, byte = mac + rows * o * i, byte + 2 * o * i

    def experts(top, num, ff, mats, b=2):
        nonlocal mac, byte
        x, y = _mix(T, top, num, ff, W, mats, b)
        mac, byte = mac + x, byte + y

    def attend(H, G, dk, dv, window=0, keep=0, latent=0):
        nonlocal mac, byte
        mac += H * (dk + dv) * _seen(case, window, keep)
        byte += 2 * (latent or G * (dk + dv)) * (_cached(case, window) + T)

    def state(H, D, V, ops):
        nonlocal mac, byte
        mac += ops * T * H * D * V
        byte += 4 * n * H * D * V * (2 if any(_contexts(case)) else 1)
    if case["model"].startswith("qwen3"):
        D, A, G = c.head_dim, c.num_attention_heads, c.num_key_value_heads
        for kind in getattr(c, "layer_types", None) or ["full_attention"] * c.num_hidden_layers:
            if kind == "full_attention":
                gated = case["model"] == "qwen3.5"
                dense(((2 if gated else 1) * A + 2 * G) * D, W)
                dense(W, A * D)
                attend(A, G, D, D)
            else:
                kd, vd = c.linear_num_key_heads * D, c.linear_num_value_heads * D
                dense(2 * kd + 2 * vd + 2 * c.linear_num_value_heads, W)
                dense(W, vd)
                state(c.linear_num_value_heads, D, D, 3)
            dense(c.num_experts, W)
            experts(c.num_experts_per_tok, c.num_experts, c.moe_intermediate_size, 3, 1 if case["fp8"] else 2)
            if case["model"] == "qwen3.5":
                dense(3 * c.shared_expert_intermediate_size, W)
        return {"bytes": byte, "flops": 2 * mac}
    for L in c.layers:
        s = L.mixer
        kind = getattr(L, "kind", None) or s.kind
        if kind in ("delta", "channel_delta"):
            nq, nv = s.kv_heads * s.dim, s.heads * s.vdim
            dense(2 * nq + 2 * nv + 2 * s.heads if kind == "delta" else 2 * nq + nv + s.heads + 2 * s.dim, W)
            if kind == "channel_delta":
                dense(s.heads * s.dim + nv, s.dim)
            dense(W, nv)
            state(s.heads, s.dim, s.vdim, 3)
        elif kind == "general_delta":
            dense(5 * s.heads * s.dim + s.dim, W)
            dense(s.heads * s.dim, s.dim)
            dense(W, s.heads * s.dim)
            state(s.heads, s.dim, s.dim, 3)
        elif kind == "mamba2":
            dense(s.inner + s.channels + s.heads, W)
            dense(W, s.inner)
            state(s.heads, s.state, s.vdim, 2)
        elif kind == "parallel":
            a, b = s.left, s.right
            dense((a.heads + a.kv_heads) * a.dim + 2 * b.heads * b.state + 2 * b.inner, W)
            dense(W, a.heads * a.vdim + b.inner)
            attend(a.heads, a.kv_heads, a.dim, a.vdim, a.window)
            state(b.heads, b.state, b.vdim, 2)
        elif kind == "latent_attention":
            dense(s.q_rank + s.kv_rank + s.rot_dim + (s.heads * s.vdim if case["model"] == "nopuzen" else 0), W)
            dense(s.heads * (s.dim + s.rot_dim), s.q_rank)
            dense(s.heads * (s.dim + s.vdim), s.kv_rank)
            dense(W, s.heads * s.vdim)
            attend(s.heads, 1, s.dim + s.rot_dim, s.vdim, s.window, 0, s.kv_rank + s.rot_dim)
        else:
            dense((s.heads + s.kv_heads) * s.dim + s.kv_heads * s.vdim, W)
            dense(W, s.heads * s.vdim)
            attend(s.heads, s.kv_heads, s.dim, s.vdim, s.window, getattr(s, "keep_first", 0))
            if case["model"] == "nepevik":          # the mixture of all heads' weights
                mac += s.heads * s.heads * _seen(case, s.window, s.keep_first)
        e = getattr(L, "moe", None) or getattr(L, "mlp", None)
        if e:
            if case["model"] != "nepevik":
                dense(e.experts, W)
            mats = 3 if case["model"] == "tadinex" else 2
            experts(e.top, e.experts, e.ff, mats)
            dense(mats * e.shared_ff, W)
        elif getattr(L, "ff", 0):
            dense(2 * L.ff, W)
    return {"bytes": byte, "flops": 2 * mac}


def tolerance(case):
    """bf16 operands through a few layers, against 64 bits: 0.0034 for the video block, 0.003 - 0.007 for decoders, up
    to 0.016 where a token whose last expert hangs on rounding takes another one, or where experts are FP8; single
    values of such a token's row move by more."""
    if case["model"] == "h3":
        return {"rel": 0.013, "max": 0.3}
    return {"rel": 0.03, "max": 0.99}


# ------------------------------------------------------------------------------------------- in 64 bits --
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _lin(x, w):
    return x @ w.to(F64).T


def _turn(x, pos, freq, mag=1.0, halves=True):
    """The channel pairs of x [T, heads, D] turned: the first with the middle one, or neighbours."""
    n = freq.shape[0]
    a = pos.to(F64)[:, None] * freq[None]
    co, si = (torch.cos(a) * mag)[:, None], (torch.sin(a) * mag)[:, None]
    one, two = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
    y = x.clone()
    y[..., one], y[..., two] = x[..., one] * co - x[..., two] * si, x[..., two] * co + x[..., one] * si
    return y


def _angles(dims, base, scaling=None):
    f, mag = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if scaling:
        factor, original, fast, slow = scaling

        def where(turns):
            return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(where(fast)), 0), min(math.ceil(where(slow)), dims - 1)
        r = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
        f, mag = [x / factor * y + x * (1.0 - y) for x, y in zip(f, r)], 0.1 * math.log(factor) + 1.0
    return torch.tensor(f, dtype=F64, device="cuda"), mag


def _see(a, b, N, start, window=0, keep=0):
    """Which of N keys the rows a .. b (the first row stands at position ``start``) look at."""
    j = torch.arange(N, device="cuda")[None]
    d = torch.arange(start + a, start + b, device="cuda")[:, None] - j
    return (d >= 0) & ((d < window) | (j < keep)) if window else d >= 0


def _softmax_attention(q, k, v, scale, start=0, window=0, sink=None, causal=True):
    """q [T, H, D], k [N, G, D], v [N, G, V] of one request -> [T, H, V]."""
    T, H, N = q.shape[0], q.shape[1], k.shape[0]
    per, out = H // k.shape[1], torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    step = max(1, (1 << 27) // N)
    for a in range(0, T, step):
        b = min(T, a + step)
        see = _see(a, b, N, start, window) if causal else None
        for h in range(H):
            s = (q[a:b, h] @ k[:, h // per].T).mul_(scale)
            if causal:
                s.masked_fill_(~see, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], 1)
            p = torch.softmax(s, -1)
            out[a:b, h] = p[:, :N] @ v[:, h // per]
    return out


def _sigmoid_attention(q, k, v, scale, temp, cap, shift):
    T, H, N = q.shape[0], q.shape[1], k.shape[0]
    per, out = H // k.shape[1], torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    see = _see(0, T, N, 0)
    for h in range(H):
        s = cap * torch.tanh((q[:, h] @ k[:, h // per].T) * (scale * temp[h] / cap))
        out[:, h] = (torch.sigmoid(s + shift[h]) * see) @ v[:, h // per]
    return out


def _mixed_attention(q, k, v, scale, window, keep, talk):
    T, H, N = q.shape[0], q.shape[1], k.shape[0]
    G, out = k.shape[1], torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    step = max(1, (1 << 26) // (N * H))
    for a in range(0, T, step):
        b = min(T, a + step)
        s = torch.einsum("tghd,ngd->ghtn", q[a:b].view(b - a, G, H // G, -1), k).reshape(H, b - a, N) * scale
        p = torch.softmax(s.masked_fill(~_see(a, b, N, 0, window, keep)[None], -math.inf), -1)
        p = (talk @ p.view(H, -1)).view(G, H // G, b - a, N)
        out[a:b] = torch.einsum("ghtn,ngv->tghv", p, v).reshape(b - a, H, -1)
    return out


def _packed(x, spans):
    """Rows [T, ...] as [requests, longest, ...] with zeros behind."""
    out = torch.zeros(len(spans), max(b - a for a, b in spans), *x.shape[1:], dtype=x.dtype, device=x.device)
    for i, (a, b) in enumerate(spans):
        out[i, :b - a] = x[a:b]
    return out


def _rows(y, spans):
    return torch.cat([y[i, :b - a] for i, (a, b) in enumerate(spans)])


def _scan(spans, D, V, step, *inputs):
    """``step(S, t, *rows)`` over time for all requests together; S [requests, heads, D, V] starts at zero."""
    packed = [_packed(x, spans) for x in inputs]
    n, T, H = packed[0].shape[:3]
    S, out = torch.zeros(n, H, D, V, dtype=F64, device="cuda"), torch.empty(n, T, H, V, dtype=F64, device="cuda")
    for t in range(T):
        S, out[:, t] = step(S, *(x[:, t] for x in packed))
    return _rows(out, spans)


def _delta_step(S, q, k, v, g, beta):
    """q, k [n, H, D], v [n, H, V], g [n, H, D or 1], beta [n, H, 1]."""
    S = S * g[..., None]
    u = beta * (v - (k[:, :, None] @ S)[:, :, 0])
    S = S + k[..., None] * u[:, :, None]
    return S, (q[:, :, None] @ S)[:, :, 0]


def _general_step(S, r, w, k, v, a):
    u = _unit(k)
    seen = u[:, :, None] @ S
    S = w[..., None] * S - (a * u)[..., None] * seen + k[..., None] * v[:, :, None]
    return S, (r[:, :, None] @ S)[:, :, 0]


def _decay_step(S, q, k, v, g):
    S = g[..., None] * S + k[..., None] * v[:, :, None]
    return S, (q[:, :, None] @ S)[:, :, 0]


def _unit(x):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _conv(x, taps, spans, bias=0.0):
    taps, K = taps.to(F64), taps.shape[-1]
    y = torch.empty_like(x)
    for a, b in spans:
        z = torch.cat([torch.zeros(K - 1, x.shape[1], dtype=F64, device="cuda"), x[a:b]])
        y[a:b] = sum(z[j:j + b - a] * taps[:, j] for j in range(K)) + bias
    return torch.nn.functional.silu(y)


def _routed(x, ids, wts, expert):
    out = torch.zeros_like(x)
    for e in torch.unique(ids).tolist():
        row, place = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, row, expert(e, x[row]) * wts[row, place][:, None])
    return out


def _heads(x, H):
    return x.view(x.shape[0], H, -1)


def _e4m3_blocks(w):
    """What E4M3 with one scale per 128 x 128 block keeps of w."""
    m, k = w.shape
    b = w.to(F32).view(m // 128, 128, k // 128, 128)
    scale = b.abs().amax((1, 3), keepdim=True) / 448.0
    return ((b * (1.0 / scale)).to(torch.float8_e4m3fn).to(F32) * scale).view(m, k)


def _exact_chat(case, seed, c, get):
    D, A, G, I, eps = c.head_dim, c.num_attention_heads, c.num_key_value_heads, c.moe_intermediate_size, c.rms_norm_eps
    rows, contexts, counts = _tokens(case, seed), _contexts(case), _counts(case)
    ids = torch.tensor([t for r, a in zip(rows, contexts) for t in r[a:]], device="cuda")
    pos = torch.tensor([p for a, n in zip(contexts, counts) for p in range(a, a + n)], device="cuda")
    ends = np.cumsum(counts).tolist()
    pages, n_pages = _pages_of(case, seed, [len(t) for t in rows])
    planes = [[torch.zeros(n_pages, PAGE, G, D, dtype=BF16, device="cuda") for _ in "kv"]
              for _ in range(c.num_hidden_layers)]
    if any(contexts):
        _fill(planes, seed)
    freq, _ = _angles(D, c.rope_theta)
    x = get("model.embed_tokens.weight")[ids].to(F64)
    for i in range(c.num_hidden_layers):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * get(p + "input_layernorm.weight").to(F64)
        q, k, v = (_heads(_lin(h, get(p + f"self_attn.{n}_proj.weight")), m) for n, m in (("q", A), ("k", G), ("v", G)))
        q = _turn(_rms(q, eps) * get(p + "self_attn.q_norm.weight").to(F64), pos, freq)
        k = _turn(_rms(k, eps) * get(p + "self_attn.k_norm.weight").to(F64), pos, freq)
        att = []
        for j, (b, n) in enumerate(zip(ends, counts)):
            old = [t[pages[j]].view(-1, G, D)[:contexts[j]].to(F64) for t in planes[i]]
            att.append(_softmax_attention(q[b - n:b], torch.cat([old[0], k[b - n:b]]), torch.cat([old[1], v[b - n:b]]),
                                          D ** -0.5, contexts[j]))
        x = x + _lin(torch.cat(att).flatten(1), get(p + "self_attn.o_proj.weight"))
        h = _rms(x, eps) * get(p + "post_attention_layernorm.weight").to(F64)
        top = torch.softmax(_lin(h, get(p + "mlp.gate.weight")), -1).topk(c.num_experts_per_tok, -1)
        up, down = get(p + "mlp.experts.gate_up_proj"), get(p + "mlp.experts.down_proj")

        def expert(e, y):
            a, b = (_e4m3_blocks(w) if case["fp8"] else w for w in (up[e], down[e]))
            z = _lin(y, a)
            return _lin(torch.nn.functional.silu(z[:, :I]) * z[:, I:], b)
        x = x + _routed(h, top.indices, top.values / top.values.sum(-1, keepdim=True), expert)
    x = x[torch.tensor([e - 1 for e in ends], device="cuda")]
    return _lin(_rms(x, eps) * get("model.norm.weight").to(F64), get("lm_head.weight"))


def _exact_hybrid(case, seed, c, get):
    eps, D, I = c.rms_norm_eps, c.head_dim, c.moe_intermediate_size
    Hk, Hv, A, G = c.linear_num_key_heads, c.linear_num_value_heads, c.num_attention_heads, c.num_key_value_heads
    ids = torch.tensor(_tokens(case, seed)[0], device="cuda")
    T, silu = len(ids), torch.nn.functional.silu
    spans, pos = [(0, T)], torch.arange(T, device="cuda")
    freq, _ = _angles(int(D * c.partial_rotary_factor), c.rope_theta)

    def norm(x, n):
        return _rms(x, eps) * (1.0 + get(n).to(F64))
    x = get("model.embed_tokens.weight")[ids].to(F64)
    for i, kind in enumerate(c.layer_types):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        if kind == "full_attention":
            a = p + "self_attn."
            qg = _heads(_lin(h, get(a + "q_proj.weight")), A)
            k, v = (_heads(_lin(h, get(a + n + "_proj.weight")), G) for n in "kv")
            o = _softmax_attention(_turn(norm(qg[..., :D], a + "q_norm.weight"), pos, freq),
                                   _turn(norm(k, a + "k_norm.weight"), pos, freq), v, D ** -0.5)
            y = _lin((o * torch.sigmoid(qg[..., D:])).flatten(1), get(a + "o_proj.weight"))
        else:
            a = p + "linear_attn."
            mixed = _conv(_lin(h, get(a + "in_proj_qkv.weight")), get(a + "conv1d.weight")[:, 0], spans)
            q, k, v = torch.split(mixed, [Hk * D, Hk * D, Hv * D], -1)
            q, k = (_unit(_heads(t, Hk)).repeat_interleave(Hv // Hk, 1) for t in (q, k))
            g = torch.exp(-torch.exp(get(a + "A_log").to(F64)) * torch.nn.functional.softplus(
                _lin(h, get(a + "in_proj_a.weight")) + get(a + "dt_bias").to(F64)))
            beta = torch.sigmoid(_lin(h, get(a + "in_proj_b.weight")))
            o = _scan(spans, D, D, _delta_step, q * D ** -0.5, k, _heads(v, Hv), g[..., None], beta[..., None])
            o = _rms(o, eps) * get(a + "norm.weight").to(F64) * silu(_heads(_lin(h, get(a + "in_proj_z.weight")), Hv))
            y = _lin(o.flatten(1), get(a + "out_proj.weight"))
        x = x + y
        h, m = norm(x, p + "post_attention_layernorm.weight"), p + "mlp."
        top = torch.softmax(_lin(h, get(m + "gate.weight")), -1).topk(c.num_experts_per_tok, -1)
        up, down = get(m + "experts.gate_up_proj"), get(m + "experts.down_proj")

        def expert(e, y):
            z = _lin(y, up[e])
            return _lin(silu(z[:, :I]) * z[:, I:], down[e])
        y = _routed(h, top.indices, top.values / top.values.sum(-1, keepdim=True), expert)
        s = silu(_lin(h, get(m + "shared_expert.gate_proj.weight"))) * _lin(h, get(m + "shared_expert.up_proj.weight"))
        x = x + y + _lin(s, get(m + "shared_expert.down_proj.weight")) * torch.sigmoid(
            _lin(h, get(m + "shared_expert_gate.weight")))
    return _lin(norm(x, "model.norm.weight"), get("lm_head.weight"))


def _per_request(f, spans, *tensors):
    return torch.cat([f(*(t[a:b] for t in tensors)) for a, b in spans])


def _positions(spans):
    return torch.cat([torch.arange(b - a, device="cuda") for a, b in spans])


def _nepevik(c, get, ids, spans):
    eps, x = c.eps, get("embed")[ids].to(F64)
    gelu, sig = torch.nn.functional.gelu, torch.sigmoid
    for i, L in enumerate(c.layers):
        s, p = L.mixer, f"l{i}.mix."
        H, Hk, D, V = s.heads, s.kv_heads, s.dim, s.vdim

        def lin(n, h=x, p=p):
            return _lin(h, get(p + n))
        if s.kind == "channel_delta":
            q, k, v = (_conv(lin(n), get(p + n + ".conv"), spans) for n in "qkv")
            q, k = (_unit(_heads(t, Hk)).repeat_interleave(H // Hk, 1) for t in (q, k))
            low = _heads(torch.nn.functional.softplus(lin("a2", lin("a1")) + get(p + "dt_bias").to(F64)), H)
            g = torch.exp(-torch.exp(get(p + "A_log").to(F64))[None, :, None] * low)
            o = _scan(spans, D, V, _delta_step, q * D ** -0.5, k, _heads(v, H), g, sig(lin("b"))[..., None])
            o = _rms(o, eps) * get(p + "norm").to(F64) * _heads(sig(lin("g2", lin("g1"))), H)
        elif s.kind == "general_delta":
            r, k, v = (_heads(lin(n), H) for n in "rkv")
            w = torch.exp(-math.exp(-0.5) * sig(lin("w2", torch.tanh(lin("w1"))) + get(p + "w0").to(F64)))
            a = sig(lin("a") + get(p + "a.b").to(F64))
            o = _rms(_scan(spans, D, D, _general_step, r, _heads(w, H), k, v, _heads(a, H)), eps).flatten(1)
            o = o * get(p + "norm").to(F64) * sig(lin("g"))
        else:
            q, k = (_heads(_rms(lin(n), eps) * get(p + n + ".norm").to(F64), m) for n, m in (("q", H), ("k", Hk)))
            o = _per_request(lambda q, k, v: _mixed_attention(q, k, v, s.scale, s.window, s.keep_first, get(p + "talk").to(F64)),
                             spans, q, k, _heads(lin("v"), Hk))
        x = x + _rms(lin("o", o.flatten(1)), eps) * get(f"l{i}.norm1").to(F64)
        m, e = f"l{i}.mlp.", L.mlp
        table = get(m + "table")[ids].long()
        y = _routed(x, table, torch.full(table.shape, 1.0 / e.top, dtype=F64, device="cuda"),
                    lambda j, h: _lin(gelu(_lin(h, get(m + f"e{j}.up"))), get(m + f"e{j}.down")))
        y = y + _lin(gelu(_lin(x, get(m + "shared.up"))), get(m + "shared.down")) * sig(_lin(x, get(m + "shared.sg")))
        x = x + _rms(y, eps) * get(f"l{i}.norm2").to(F64)
    return _rms(x, eps) * get("final.norm").to(F64), get("head")


def _latent(c, get, p, s, h, spans, freq, mag, halves, gate=None):
    H, D, R, K, pos = s.heads, s.dim, s.rot_dim, s.kv_rank, _positions(spans)
    q = _heads(_lin(_rms(_lin(h, get(p + "dq")), c.eps) * get(p + "dq.norm").to(F64), get(p + "uq")), H)
    kv = _lin(h, get(p + "dkv"))
    lat = _rms(kv[:, :K], c.eps) * get(p + "dkv.norm").to(F64)
    kr = _turn(kv[:, None, K:], pos, freq, mag, halves).expand(-1, H, R)
    q = torch.cat([q[..., :D], _turn(q[..., D:], pos, freq, mag, halves)], -1)
    k = torch.cat([_heads(_lin(lat, get(p + "uk")), H), kr], -1)
    o = _per_request(lambda q, k, v: _softmax_attention(q, k, v, s.scale, 0, s.window), spans, q, k,
                     _heads(_lin(lat, get(p + "uv")), H)).flatten(1)
    return _lin(o if gate is None else o * torch.sigmoid(_lin(h, get(gate))), get(p + "o"))


def _zonopel(c, get, ids, spans):
    eps, b = c.eps, c.bigram

    def norm(x, n):
        return _rms(x, eps) * get(n).to(F64)
    before = torch.cat([ids.new_zeros(1), ids[:-1]])
    row = (before * b.mul_prev + ids * b.mul_cur) % b.buckets
    starts = torch.tensor([a for a, _ in spans], device="cuda")
    row[starts] = b.buckets
    x = norm(get("embed")[ids].to(F64) * c.embed_scale + get("bigram")[row].to(F64), "embed.norm")
    for i, L in enumerate(c.layers):
        i = i if L.weights_of is None else L.weights_of
        p, s, l, m = f"l{i}.mix.", L.mixer, f"l{i}.", f"l{i}.mlp."
        h = norm(x, l + "norm1")
        back = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        back[starts] = 0.0
        h = h + (back - h) * get(l + "shift").to(F64)
        if L.kind == "mamba2":
            H, V, N, G = s.heads, s.vdim, s.state, s.groups
            z, xbc, dt = torch.split(_lin(h, get(p + "in")), [s.inner, s.channels, H], -1)
            xbc = _conv(xbc, get(p + "conv"), spans, get(p + "conv.b").to(F64))
            v, B, C = torch.split(xbc, [s.inner, G * N, G * N], -1)
            dt = torch.nn.functional.softplus(dt + get(p + "dt_bias").to(F64))
            B, C = (_heads(t, G).repeat_interleave(H // G, 1) for t in (B, C))
            g = torch.exp(-torch.exp(get(p + "A_log").to(F64)) * dt)
            y = _scan(spans, N, V, _decay_step, C, B * dt[..., None], _heads(v, H), g[..., None])
            y = (y + get(p + "D").to(F64)[:, None] * _heads(v, H)).flatten(1) * torch.nn.functional.silu(z)
            y = _lin(_rms(_heads(y, s.norm_groups), eps).flatten(1) * get(p + "norm").to(F64), get(p + "o"))
        else:
            y = _latent(c, get, p, s, h, spans, *_angles(L.rot_dims, L.rot_base), False)
        x = x + norm(y, l + "norm1b")
        u, act = _lin(norm(x, l + "norm2"), get(m + "up")), get(m + "act").to(F64)
        u = act[0] * _rms(u, eps) + act[1] * _rms(u * u, eps) + act[2] * _rms(u ** 3, eps) + act[3]
        x = x + norm(_lin(u, get(m + "down")), l + "norm2b")
    return norm(x, "final.norm"), get("head")


def _tadinex(c, get, ids, spans):
    eps, silu, pos = c.eps, torch.nn.functional.silu, _positions(spans)
    x = get("embed")[ids].to(F64) * c.embed_scale

    def norm(x, n):
        return _rms(x, eps) * (1.0 + get(n).to(F64))

    def expert(p, h, limit):
        g, u = _lin(h, get(p + "gate")).clamp(max=limit), _lin(h, get(p + "up")).clamp(-limit, limit)
        return _lin(g * torch.sigmoid(GLU_ALPHA * g) * (u + 1), get(p + "down"))
    for i, L in enumerate(c.layers):
        p, s, m, e = f"l{i}.mix.", L.mixer, f"l{i}.mlp.", L.moe
        h = norm(x, f"l{i}.norm1")

        def lin(n, h=h, p=p):
            return _lin(h, get(p + n))
        if L.kind == "delta":
            H, Hk, D, V = s.heads, s.kv_heads, s.dim, s.vdim
            q, k, v = (_conv(lin(n), get(p + n + ".conv"), spans) for n in "qkv")
            q, k = (_unit(_heads(t, Hk)).repeat_interleave(H // Hk, 1) for t in (q, k))
            g = torch.exp(-torch.exp(get(p + "A_log").to(F64)) * torch.nn.functional.softplus(
                lin("a") + get(p + "dt_bias").to(F64)))
            o = _scan(spans, D, V, _delta_step, q * D ** -0.5, k, _heads(v, H), g[..., None],
                      torch.sigmoid(lin("b"))[..., None])
            y = lin("o", (_rms(o, eps) * get(p + "norm").to(F64) * silu(_heads(lin("g"), H))).flatten(1))
        else:
            a, b = s.left, s.right
            freq, mag = _angles(s.rot_dims, s.rot_base, s.rot_scaling)
            q, v = _heads(lin("left.q"), a.heads), _heads(lin("left.k"), a.kv_heads)
            q, k = (_turn(_rms(t, eps) * get(p + n).to(F64), pos, freq, mag)
                    for t, n in ((q, "left.q.norm"), (v, "left.k.norm")))
            sink = get(p + "left.sink").to(F64)
            o = _per_request(lambda q, k, v: _softmax_attention(q, k, v, a.scale, 0, a.window, sink), spans, q, k, v)
            y = s.left_scale * lin("left.o", o.flatten(1))
            q, k, v = (_heads(silu(lin("right." + n)), b.heads) for n in "qkv")
            decay = torch.tensor(s.decay, dtype=F64, device="cuda")[None, :, None].expand(len(ids), -1, 1)
            o = _scan(spans, b.state, b.vdim, _decay_step, q, k, v, decay).flatten(1)
            o = _rms(o, eps) * get(p + "right.norm").to(F64) * torch.sigmoid(lin("right.g"))
            y = y + s.right_scale * lin("right.o", o)
        x = x + c.residual_mult * y
        h = norm(x, f"l{i}.norm2")
        z = torch.softmax(_lin(h, get(m + "router")), -1)
        top = (z + get(m + "correction").to(F64)).topk(e.top, -1).indices
        w = z.gather(1, top)
        y = _routed(h, top, w / w.sum(-1, keepdim=True),
                    lambda j, t: expert(m + f"e{j}.", t, e.limit) if j < e.experts else t)
        x = x + c.residual_mult * (y + expert(m + "shared.", h, e.shared_limit))
    return norm(x, "final.norm"), get("head")


def _nopuzen(c, get, ids, spans):
    eps, pos, sig, sp = c.eps, _positions(spans), torch.sigmoid, torch.nn.functional.softplus
    x = get("embed")[ids].to(F64)

    def norm(x, n):
        d = x - x.mean(-1, keepdim=True)
        return _rms(d, eps) * get(n).to(F64) + get(n + ".b").to(F64)

    def expert(p, h):
        return _lin(_lin(h, get(p + "up")).clamp(min=0) ** 2, get(p + "down"))
    for i, L in enumerate(c.layers):
        p, s, m, e = f"l{i}.mix.", L.mixer, f"l{i}.mlp.", L.moe
        freq, mag = _angles(L.rot.dims, L.rot.base, L.rot.scaling)
        if L.kind == "attention":
            q, k, v = (_heads(_lin(x, get(p + n)) + get(p + n + ".b").to(F64), h)
                       for n, h in (("q", s.heads), ("k", s.kv_heads), ("v", s.kv_heads)))
            q, k = (_turn(_rms(t, eps) * get(p + n).to(F64), pos, freq, mag, False)
                    for t, n in ((q, "q.norm"), (k, "k.norm")))
            temp, shift = get(p + "temp").to(F64), get(p + "pb").to(F64)
            o = _per_request(lambda q, k, v: _sigmoid_attention(q, k, v, s.scale, temp, L.softcap, shift), spans, q, k, v)
            o = o * sig(_lin(x, get(p + "g")))[:, :, None]
            y = _lin(o.flatten(1), get(p + "o")) + get(p + "o.b").to(F64)
        else:
            y = _latent(c, get, p, s, x, spans, freq, mag, True, p + "g")
        x = x + norm(y, f"l{i}.norm1")
        if L.ff:
            z, (a, b) = _lin(x, get(m + "up")), get(m + "act").to(F64)
            z = torch.where(z > 0, sp(a) * z * z + z / 2, (0.5 + sp(b)) * (torch.exp(z.clamp(max=0)) - 1 - z) + z / 2)
            y = _lin(z, get(m + "down"))
        else:
            z = torch.softmax(_lin(x, get(m + "router")), -1)
            count, keep = e.groups
            best = z.view(len(ids), count, -1).amax(-1).topk(keep, -1).indices
            open_ = torch.zeros(len(ids), count, dtype=torch.bool, device="cuda").scatter_(1, best, True)
            top = z.masked_fill(~open_.repeat_interleave(e.experts // count, 1), -1.0).topk(e.top, -1).indices
            y = _routed(x, top, z.gather(1, top) * e.scale, lambda j, t: expert(m + f"e{j}.", t))
            y = y + sig(_lin(x, get(m + "shared.sg"))) * expert(m + "shared.", x)
        x = x + norm(y, f"l{i}.norm2")
    return norm(x, "final.norm"), get("embed")


def _exact_video(case, seed, c, get):
    video, audio, text = _video_inputs(case, seed, c)
    C, Fr, H, W = video.shape
    N, D, I, eps = c.num_heads, c.head_dim, c.ffn_size, c.eps
    v = video.to(F64).view(C, Fr, H // 2, 2, W // 2, 2).permute(1, 2, 4, 0, 3, 5).reshape(-1, 4 * C)
    x = torch.cat([_lin(v, get("proj_in")), _lin(audio.to(F64), get("audio_proj_in")), text.to(F64)])
    n_video, n_audio, T = v.shape[0], audio.shape[0], x.shape[0]
    at = torch.zeros(3, T, dtype=F64, device="cuda")
    at[:, :n_video] = torch.stack(torch.meshgrid(*(torch.arange(n, dtype=F64, device="cuda") for n in (Fr, H // 2, W // 2)),
                                                 indexing="ij")).reshape(3, -1)
    at[0, n_video:n_video + n_audio] = torch.arange(n_audio, dtype=F64, device="cuda") * (Fr / n_audio)
    kind = torch.full((T,), 1, device="cuda")
    kind[:n_video], kind[n_video:n_video + n_audio] = 0, 3 + 2
    table, last = get("table").view(12, 6, -1).to(F64), get("table_out").view(12, 2, -1).to(F64)
    freq, _ = _angles(2 * c.rope_freqs_per_axis, c.rope_theta)
    n = 2 * c.rope_freqs_per_axis

    def turned(t):
        return torch.cat([_turn(t[..., a * n:(a + 1) * n], at[a], freq) for a in range(3)] + [t[..., 3 * n:]], -1)
    h = _rms(x, eps) * (1.0 + table[kind, 1]) + table[kind, 0]
    q, k, v = (_heads(t, N) for t in torch.chunk(_lin(h, get("qkv")), 3, 1))
    q, k = (turned(_rms(t, eps) * get(w).to(F64)) for t, w in ((q, "q_norm"), (k, "k_norm")))
    x = x + table[kind, 2] * _lin(_softmax_attention(q, k, v, D ** -0.5, causal=False).flatten(1), get("to_out"))
    del q, k, v
    h = _rms(x, eps) * (1.0 + table[kind, 4]) + table[kind, 3]
    z = _lin(h, get("ff1"))
    x = x + table[kind, 5] * _lin(z[:, :I] * torch.nn.functional.silu(z[:, I:]), get("ff2"))
    x = _rms(x, eps) * (1.0 + last[kind, 1]) + last[kind, 0]
    return {"video": _lin(x[:n_video], get("proj_out")), "audio": _lin(x[n_video:n_video + n_audio], get("audio_proj_out"))}


def exact(case, seed):
    c, get = _config(case), _weights(case, seed).get
    if case["model"] == "h3":
        return _exact_video(case, seed, c, get)
    out = {"states": None} if case["phase"] == "decode" or case["model"] == "qwen3.5" else {"pages": None, "states": None}
    if case["model"] == "qwen3.5":
        return {"logits": _exact_hybrid(case, seed, c, get), **out}
    if case["model"].startswith("qwen3-moe"):
        return {"logits": _exact_chat(case, seed, c, get).cpu(), **out}
    rows = _tokens(case, seed)
    ends = np.cumsum([len(t) for t in rows]).tolist()
    spans = [(b - len(t), b) for t, b in zip(rows, ends)]
    x, head = {"nepevik": _nepevik, "zonopel": _zonopel, "tadinex": _tadinex, "nopuzen": _nopuzen}[case["model"]](
        c, get, torch.tensor([t for r in rows for t in r], device="cuda"), spans)
    return {"logits": _lin(x[torch.tensor([b - 1 for b in ends], device="cuda")], head).cpu(), **out}
