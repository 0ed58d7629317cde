"""The work this framework is measured on, through its public entry points, on one GPU.

``listed()`` are twelve fixed cases, ``draw(rng)`` gives more of the same ranges. Every case is a dict
of plain values with a ``kind``:

* ``pattern``   ``ultraattn_b200.attention`` under a block pattern (causal, full, strided, global +
                local, star, streaming: the patterns of the campaign classes and of ``configs/``);
* ``flash``     ``flash_compat.flash_attn_func``: dense attention in flash-attention's calling
                convention, also with fewer queries than keys (decoding, chunked prefill);
* ``varlen``    ``api.varlen_attention``: a packed batch of documents of ragged lengths;
* ``window``    ``ops.window.sliding_window_attention``: token-exact bands, with or without sinks;
* ``llama``     ``models.llama.LlamaModel.train_step``: a whole optimizer step.

``train`` cases run forward and backward and return the output and all gradients, the others run
the forward under ``no_grad`` as a serving program does. Everything is bf16 with head dim 128, the
type and size of every configuration of this repository.
"""
from __future__ import annotations

import math
import random

import torch

import ultraattn_b200 as ua
from ultraattn_b200 import patterns as P
from ultraattn_b200.api import varlen_attention
from ultraattn_b200.models.llama import LlamaConfig, LlamaModel
from ultraattn_b200.ops.flash_compat import flash_attn_func
from ultraattn_b200.ops.window import sliding_window_attention

D = 128
# block patterns of the campaign (drivers/exp_configs.py): 32 blocks for the sparse ones
PATTERNS = {
    "causal": lambda: P.causal(1),
    "full": lambda: P.full(1),
    "strided": lambda: P.strided(32, 4, 2),
    "global_local": lambda: P.global_local(32, 1, 2),
    "star": lambda: P.star(32, 1),
    "streaming": lambda: P.streaming(32, 1, 2),
}


def listed() -> list:
    return [
        # the smallest training call: a unit-test or fine-tuning sized sequence, where launches and
        # host time count
        dict(name="short_train", kind="pattern", pattern="causal", train=True, batch=1, seq=512, heads=8, kv_heads=8),
        # serving: the prompt of one chat request, a length that fits no tile, grouped-query heads
        dict(name="short_prefill_gqa", kind="flash", causal=True, train=False, batch=1, seq_q=1000, seq_k=1000,
             heads=32, kv_heads=8),
        # serving: one decoding step of a batch, one new query per sequence behind its cached keys
        dict(name="decode_gqa", kind="flash", causal=True, train=False, batch=16, seq_q=1, seq_k=8123, heads=32,
             kv_heads=8),
        # serving: a chunk of a long prompt behind the keys of the chunks before it
        dict(name="chunk_prefill_gqa", kind="flash", causal=True, train=False, batch=1, seq_q=512, seq_k=32768,
             heads=32, kv_heads=8),
        # encoder-style training: a batch of full-attention sequences of an odd length
        dict(name="full_train_batch", kind="flash", causal=False, train=True, batch=4, seq_q=2000, seq_k=2000,
             heads=16, kv_heads=16),
        # the Llama-2-7B attention shape at an ordinary training length
        dict(name="causal_train_8k", kind="pattern", pattern="causal", train=True, batch=1, seq=8192, heads=32,
             kv_heads=32),
        # the headline pattern of the benchmark at a quarter of its length (the largest case)
        dict(name="strided_train_128k", kind="pattern", pattern="strided", train=True, batch=1, seq=131072, heads=32,
             kv_heads=32),
        # block-sparse prefill of a long prompt: sink block and local window
        dict(name="streaming_prefill_128k", kind="pattern", pattern="streaming", train=False, batch=1, seq=131072,
             heads=32, kv_heads=32),
        # packed pre-training batch: documents of very different lengths in one buffer
        dict(name="varlen_train_gqa", kind="varlen", causal=True, train=True, seq=16384, docs=12, doc_seed=3,
             heads=32, kv_heads=8),
        # Mistral-7B's attention shape: causal window of 4096 tokens, grouped-query heads
        dict(name="window_train_gqa", kind="window", train=True, batch=1, seq=16384, left=4095, sink=0, heads=32,
             kv_heads=8),
        # streaming inference: a window with attention sinks over a long prompt (drivers/bench_masks.py)
        dict(name="window_sink_prefill", kind="window", train=False, batch=1, seq=32768, left=1023, sink=4, heads=16,
             kv_heads=16),
        # a training step of two Llama-2-7B layers with embedding, loss head and optimizer
        dict(name="llama_step", kind="llama", layers=2, hidden=4096, heads=32, kv_heads=32, ffn=11008, vocab=32000,
             seq=8192),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng: random.Random) -> tuple:
    kv = rng.choice([2, 4, 8, 16, 32])
    return kv * rng.choice([g for g in (1, 2, 4, 8) if 8 <= kv * g <= 32 or (kv == 2 and g >= 4)]), kv


def draw(rng: random.Random) -> dict:
    """One more case. Sizes are spread over their logarithm, most of them multiples of nothing."""
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw(rng)
        if work(c)["flops"] <= most:
            return c


def _draw(rng: random.Random) -> dict:
    kind = rng.choice(["pattern", "pattern", "pattern", "flash", "flash", "decode", "chunk", "varlen", "window", "window",
                       "llama"])
    h, kv = _heads(rng)
    train = rng.random() < 0.6
    if kind == "pattern":
        name = rng.choice(sorted(PATTERNS))
        seq = 32 * _log(rng, 16, 4096) if name not in ("causal", "full") else _log(rng, 200, 32768)
        return dict(kind="pattern", pattern=name, train=train and name not in ("star", "streaming"), batch=1, seq=seq,
                    heads=h, kv_heads=kv)
    if kind == "flash":
        seq = _log(rng, 200, 16384)
        return dict(kind="flash", causal=rng.random() < 0.6, train=train, batch=rng.choice([1, 1, 2, 4]), seq_q=seq,
                    seq_k=seq, heads=h, kv_heads=kv)
    if kind == "decode":
        return dict(kind="flash", causal=True, train=False, batch=_log(rng, 1, 64), seq_q=1, seq_k=_log(rng, 512, 32768),
                    heads=h, kv_heads=kv)
    if kind == "chunk":
        sq = _log(rng, 16, 2048)
        return dict(kind="flash", causal=True, train=False, batch=1, seq_q=sq, seq_k=sq + _log(rng, 1024, 65536),
                    heads=h, kv_heads=kv)
    if kind == "varlen":
        return dict(kind="varlen", causal=rng.random() < 0.8, train=train, seq=_log(rng, 2048, 32768),
                    docs=_log(rng, 2, 32), doc_seed=rng.randrange(1 << 20), heads=h, kv_heads=kv)
    if kind == "window":
        seq = _log(rng, 2048, 65536)
        return dict(kind="window", train=train, batch=1, seq=seq, left=min(seq // 2, _log(rng, 256, 8192)) - 1,
                    sink=rng.choice([0, 0, 4]), heads=h, kv_heads=kv)
    hidden = rng.choice([2048, 4096])
    return dict(kind="llama", layers=rng.choice([1, 2]), hidden=hidden, heads=hidden // D,
                kv_heads=rng.choice([8, hidden // D]), ffn=rng.choice([5632, 11008, 14336]), vocab=32000,
                seq=8 * _log(rng, 128, 1024))      # the weight gradients need a multiple of 8 tokens


# ------------------------------------------------------------------------------------------------
def _doc_bounds(c: dict) -> list:
    """Start tokens of ``docs`` documents of random lengths (at least one token each) plus the end."""
    r = random.Random(c["doc_seed"])
    return [0] + sorted(r.sample(range(1, c["seq"]), c["docs"] - 1)) + [c["seq"]]


def prepare(case: dict, seed: int) -> dict:
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    c = case

    def rand(*shape, grad=False):
        # projections of normalised activations: standard normal
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.bfloat16).requires_grad_(grad)

    if c["kind"] == "llama":
        cfg = LlamaConfig(n_layers=c["layers"], hidden=c["hidden"], n_heads=c["heads"], n_kv_heads=c["kv_heads"],
                          head_dim=D, ffn=c["ffn"], vocab=c["vocab"])
        model = LlamaModel(cfg, device=dev, pattern=P.global_local(4, 1, 2), seed=seed)
        ids = torch.randint(0, c["vocab"], (c["seq"] + 1,), generator=g, device=dev)
        return dict(case=c, model=model, ids=ids[:-1].contiguous(), targets=ids[1:].contiguous(),
                    pos=torch.arange(c["seq"], device=dev))
    lead_q = (c["seq"],) if c["kind"] == "varlen" else (c["batch"], c.get("seq_q", c.get("seq")))
    lead_k = (c["seq"],) if c["kind"] == "varlen" else (c["batch"], c.get("seq_k", c.get("seq")))
    s = dict(case=c, q=rand(*lead_q, c["heads"], D, grad=c["train"]), k=rand(*lead_k, c["kv_heads"], D, grad=c["train"]),
             v=rand(*lead_k, c["kv_heads"], D, grad=c["train"]))
    if c["train"]:
        s["d_o"] = rand(*lead_q, c["heads"], D)
    if c["kind"] == "pattern":
        s["pattern"] = PATTERNS[c["pattern"]]()
    if c["kind"] == "varlen":
        s["cu"] = _doc_bounds(c)
    return s


def _attend(s: dict):
    c, q, k, v = s["case"], s["q"], s["k"], s["v"]
    if c["kind"] == "pattern":
        return ua.attention(q, k, v, s["pattern"])
    if c["kind"] == "flash":
        return flash_attn_func(q, k, v, causal=c["causal"])
    if c["kind"] == "varlen":
        return varlen_attention(q, k, v, s["cu"], causal=c["causal"])
    return sliding_window_attention(q, k, v, (c["left"], 0), causal=True, sink_tokens=c["sink"])


def run(state: dict):
    c = state["case"]
    if c["kind"] == "llama":
        m = state["model"]
        loss = m.train_step(state["ids"], state["targets"], state["pos"], n_total_tokens=c["seq"])
        # the updated weights and Adam's first moment (a tenth of the step's gradients, at the first step)
        return {"loss": loss, "weights": m.flat, "moment": m.m}
    if not c["train"]:
        with torch.no_grad():
            return {"o": _attend(state)}
    o = _attend(state)
    dq, dk, dv = torch.autograd.grad(o, (state["q"], state["k"], state["v"]), state["d_o"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


# ------------------------------------------------------------------------------------------------
def _pairs(c: dict) -> float:
    """Visible (query, key) pairs of one head, over the whole batch."""
    tri = lambda n: n * (n + 1) / 2
    if c["kind"] == "pattern":
        t = PATTERNS[c["pattern"]]().block_table_int
        blk = c["seq"] // t.shape[0]
        return c["batch"] * float((t == 1).sum() * blk * blk + (t == 2).sum() * tri(blk))
    if c["kind"] == "flash":
        sq, sk = c["seq_q"], c["seq_k"]
        return c["batch"] * float(sq * sk - (tri(sq - 1) if c["causal"] else 0))
    if c["kind"] == "varlen":
        b = _doc_bounds(c)
        return float(sum(tri(y - x) if c["causal"] else (y - x) ** 2 for x, y in zip(b[:-1], b[1:])))
    w, n = c["left"] + 1, c["seq"]
    band = tri(min(w, n)) + max(0, n - w) * w
    sinks = sum(max(0, n - w - j) for j in range(c["sink"]))        # queries that have sink key j outside their window
    return c["batch"] * float(band + sinks)


def work(case: dict) -> dict:
    c = case
    if c["kind"] == "llama":
        T, H, q, kv, F, V, L = c["seq"], c["hidden"], c["heads"] * D, c["kv_heads"] * D, c["ffn"], c["vocab"], c["layers"]
        linear = L * (H * (q + 2 * kv) + q * H + 3 * H * F) + V * H
        blk = T // 4
        t = P.global_local(4, 1, 2).block_table_int
        pairs = float((t == 1).sum() * blk * blk + (t == 2).sum() * blk * (blk + 1) / 2)
        params = linear + V * H + (2 * L + 1) * H
        # every product forward and twice backward, attention with its scores again in the backward;
        # per parameter: fp32 master and two moments in and out, the bf16 weight out
        return {"bytes": params * (12 + 14), "flops": 6.0 * T * linear + 3.5 * 4 * pairs * q * L}
    tok_q = c["seq"] if c["kind"] == "varlen" else c["batch"] * c.get("seq_q", c.get("seq"))
    tok_k = c["seq"] if c["kind"] == "varlen" else c["batch"] * c.get("seq_k", c.get("seq"))
    nq, nk = tok_q * c["heads"] * D * 2, tok_k * c["kv_heads"] * D * 2
    flops = 4.0 * _pairs(c) * c["heads"] * D
    if not c["train"]:
        return {"bytes": 2 * nq + 2 * nk, "flops": flops}
    # in: q, k, v, dO; out: o, dq, dk, dv. Five products in the backward for the forward's two
    return {"bytes": 4 * nq + 4 * nk, "flops": 3.5 * flops}


def tolerance(case: dict):
    """bf16 inputs and outputs, fp32 sums, probabilities and score gradients rounded to bf16 on their
    way into the tensor core: o is 2.5e-3 and the gradients are 3.5e-3 away from float64 at most, over
    all kinds at 512 to 3000 tokens; four times that. A training step repeats itself to 2.5e-3 (dQ and the
    norm weights are summed in arrival order)."""
    if case["kind"] == "llama":
        return {"rel": 2e-2}
    return {"rel": 1.4e-2} if case["train"] else {"rel": 1e-2}
