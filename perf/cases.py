"""Performance cases: the work that users of this framework have it do, through its public entry points.

A pass is what one attention layer runs: `create_mask` on the layer's bias where the layer has one, then
`flash_sparse_attn_func` (or the packed-sequence form), and for training the gradients of everything that is learned.
Every case is a dict of plain values:

  kind     "train"   forward and backward            "prefill"  forward of a prompt, no gradients
           "decode"  one query row per sequence      "packed"   forward and backward over packed sequences
  mask     "row"     one bias row per (batch, kv head), shared by all queries: the layout a model's bias producer gives
           "query"   a bias row of its own for every query          "none"  no bias, no dynamic mask
  batch, seqlen_q, seqlen_k, heads, kv_heads, head_dim, window (kept keys per row), dtype, causal,
  padded   left-padded caches (decode): 2-D padding mask, lengths falling evenly from the whole to about half
  deterministic      bit-identical gradients from run to run
  lengths  (packed only) the sequences' lengths, as text
"""
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "flash-dmattn_b200"))  # the package of the tree that is the working folder

from flash_sparse_attn import flash_sparse_attn_func, flash_sparse_attn_varlen_func  # noqa: E402
from flash_sparse_attn.utils.mask import create_mask  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# (query heads, kv heads): multi-query, grouped and plain multi-head layouts
_HEADS = ((2, 1), (8, 2), (8, 8), (12, 4), (16, 4), (16, 1), (32, 8))


def _case(kind, mask, batch, seqlen_q, seqlen_k, heads, head_dim, window, dtype="bf16", causal=True, padded=False,
          deterministic=False, lengths="", name=None):
    c = {} if name is None else {"name": name}
    c.update(kind=kind, mask=mask, batch=batch, seqlen_q=seqlen_q, seqlen_k=seqlen_k, heads=heads[0],
             kv_heads=heads[1], head_dim=head_dim, window=window, dtype=dtype, causal=causal, padded=padded,
             deterministic=deterministic)
    if kind == "packed":
        c["lengths"] = lengths
    return c


def listed():
    return [
        # The smallest training call in use (unit-scale models, tests, debugging): launches and host work count.
        _case("train", "row", 1, 256, 256, (2, 1), 64, 128, name="train_small"),
        # Pre-training of a small model at its usual context: head dim 64, a few sequences per GPU.
        _case("train", "row", 4, 2048, 2048, (16, 4), 64, 512, name="train_2k_d64"),
        # Fine-tuning on sequences of whatever length the data has, fp16 with loss scaling.
        _case("train", "row", 2, 3001, 3001, (12, 4), 128, 700, dtype="fp16", name="train_ragged_fp16"),
        # Long-context training, the headline workload.
        _case("train", "row", 1, 32768, 32768, (32, 8), 128, 2048, name="train_32k"),
        # One very long sequence, wide heads, a single kv head.
        _case("train", "row", 1, 65536, 65536, (16, 1), 256, 2048, name="train_65k_d256"),
        # Training with a bias per (query, key) pair, which also takes a gradient.
        _case("train", "query", 1, 8192, 8192, (32, 8), 128, 1024, name="train_per_query_8k"),
        # Layers without a dynamic mask, and sequences no longer than the window: plain causal attention.
        _case("train", "none", 1, 4096, 4096, (32, 8), 128, 0, name="train_plain_4k"),
        # Reproducible training runs: gradients that are the same bits every time.
        _case("train", "row", 1, 8192, 8192, (32, 8), 128, 2048, deterministic=True, name="train_deterministic_8k"),
        # Padding-free fine-tuning: several documents packed into one row.
        _case("packed", "none", 1, 8192, 8192, (16, 4), 128, 0, lengths="4096,1733,1290,700,373",
              name="train_packed_8k"),
        # Serving, prompt phase: a few prompts at once, no gradients.
        _case("prefill", "row", 4, 4096, 4096, (32, 8), 128, 1024, name="prefill_4k"),
        # Serving, token phase, one user: latency of a single step.
        _case("decode", "row", 1, 1, 4097, (32, 8), 128, 1024, causal=False, name="decode_one"),
        # Serving, token phase, many users with long caches: memory traffic counts.
        _case("decode", "row", 32, 1, 65536, (32, 8), 128, 4096, causal=False, name="decode_32x64k"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _length(rng, lo, hi):
    """A length between lo and hi, spread over its logarithm: half as drawn (odd ones among them), half in whole tiles."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.5 else max(lo, (n + 64) // 128 * 128)


def _window(rng, keys):
    return _log(rng, max(32, -(-keys // 32)), max(32, min(4096, keys)))


def draw(rng):
    """One more case of the ranges above: training lengths 128 to 32768 (with a bias per query or without a mask up to
    8192), prompts up to 32768, caches up to 65536, head dims 64 to 256. A window is at most 4096 keys and at least a
    32nd of the keys (decode: 128 keys or all)."""
    while True:
        kind, mask = rng.choice((("train", "row"), ("train", "row"), ("train", "row"), ("train", "query"), ("train", "none"),
                                 ("packed", "none"), ("prefill", "row"), ("prefill", "row"), ("decode", "row"),
                                 ("decode", "row")))
        heads = rng.choice(_HEADS)
        dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
        head_dim = rng.choice((64, 64, 128, 128, 128, 96, 256) if mask == "row" else (64, 128, 128))
        if kind == "packed":
            lens = [_length(rng, 64, 4096) for _ in range(rng.randint(2, 8))]
            total = sum(lens)
            c = _case(kind, mask, 1, total, total, heads, head_dim, 0, dtype, lengths=",".join(map(str, lens)))
        elif kind == "decode":
            sk = _length(rng, 512, 65536)
            c = _case(kind, mask, _log(rng, 1, 32), 1, sk, heads, head_dim, min(_log(rng, 128, 4096), sk), dtype,
                      causal=False, padded=rng.random() < 0.25)
        elif kind == "prefill":
            s = _length(rng, 128, 32768)
            batch = _log(rng, 1, 8)
            cached = _length(rng, 128, 16384) if rng.random() < 0.25 else 0  # a later part of a prompt that is fed in parts
            c = _case(kind, mask, batch, s, s + cached, heads, head_dim, _window(rng, s + cached), dtype)
        else:
            s = _length(rng, 128, 32768 if mask == "row" else 8192)
            c = _case(kind, mask, _log(rng, 1, 8), s, s, heads, head_dim, _window(rng, s) if mask != "none" else 0, dtype,
                      deterministic=rng.random() < 0.15)
        if c["batch"] * c["seqlen_q"] <= 32768 and _scores(c) <= 1.1e10 and c["batch"] * c["seqlen_k"] <= (1 << 21):
            return c


def _scores(c):
    """Scores a whole-tile implementation computes, over all heads, scaled to head dim 128 and to a backward pass: what a
    drawn case may cost at most."""
    keys = c["window"] if c["mask"] == "row" else c["seqlen_k"]
    rows = c["batch"] * c["seqlen_q"] * c["heads"]
    half = 0.5 if c["causal"] and c["mask"] != "row" else 1.0
    return rows * keys * half * max(1.0, c["head_dim"] / 128) * (8 if c["mask"] == "query" else 1)


def _valid_keys(c):
    """Valid keys per sequence: all of them, or for a padded batch falling evenly from all to about half."""
    n, b = c["seqlen_k"], c["batch"]
    return [n - i * n // (2 * b) for i in range(b)] if c["padded"] else [n] * b


def prepare(case, seed):
    """Activations, bias and output gradient ~ N(0,1), as after a normalisation layer; all from the seed."""
    c, dtype = case, _DTYPES[case["dtype"]]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    B, Sq, Sk, H, Hk, d = (c[n] for n in ("batch", "seqlen_q", "seqlen_k", "heads", "kv_heads", "head_dim"))
    train = c["kind"] in ("train", "packed")

    def rnd(*shape, grad=False):
        return torch.randn(shape, generator=g, device=dev, dtype=dtype).requires_grad_(grad)

    lead = () if c["kind"] == "packed" else (B,)
    s = {"case": c, "q": rnd(*lead, Sq, H, d, grad=train), "k": rnd(*lead, Sk, Hk, d, grad=train),
         "v": rnd(*lead, Sk, Hk, d, grad=train), "bias": None, "padding": None}
    if c["mask"] != "none":
        s["bias"] = rnd(B, Hk, Sq if c["mask"] == "query" else 1, Sk, grad=train)
    if c["padded"]:
        first = torch.tensor([Sk - n for n in _valid_keys(c)], device=dev)
        s["padding"] = torch.arange(Sk, device=dev)[None, :] >= first[:, None]
    if train:
        s["dout"] = rnd(*lead, Sq, H, d)
    if c["kind"] == "packed":
        lens = torch.tensor([0] + [int(n) for n in c["lengths"].split(",")], device=dev)
        s["cu"] = lens.cumsum(0).to(torch.int32)
        s["longest"] = int(lens.max())
    return s


def run(s):
    c, q, k, v, bias = s["case"], s["q"], s["k"], s["v"], s["bias"]
    if c["kind"] == "packed":
        out = flash_sparse_attn_varlen_func(q, k, v, s["cu"], s["cu"], s["longest"], s["longest"], is_causal=True,
                                            deterministic=c["deterministic"])
        return (out, *torch.autograd.grad(out, (q, k, v), s["dout"]))
    mask = None
    if bias is not None:
        mask = create_mask(bias, s["padding"], c["batch"], c["seqlen_q"], c["seqlen_k"], c["window"],
                           torch.finfo(bias.dtype).min)
    if c["kind"] == "train":
        out = flash_sparse_attn_func(q, k, v, attn_mask=mask, attn_bias=bias, is_causal=c["causal"],
                                     deterministic=c["deterministic"])
        learned = (q, k, v) if bias is None else (q, k, v, bias)
        return (out, *torch.autograd.grad(out, learned, s["dout"]))
    with torch.no_grad():
        return flash_sparse_attn_func(q, k, v, attn_mask=mask, attn_bias=bias, is_causal=c["causal"])


def work(case):
    """Bytes: what is read of q, k, v, bias and output gradient (of k and v only the kept rows, where the queries share
    them) and what is written of the output and the gradients, once each. Operations: 4 d for each kept and visible
    (query, key) pair forward, 10 d backward; a kept key is anywhere in its row with equal likelihood."""
    c = case
    B, Sq, Sk, H, Hk, d = (c[n] for n in ("batch", "seqlen_q", "seqlen_k", "heads", "kv_heads", "head_dim"))
    train = c["kind"] in ("train", "packed")
    pairs = kept_rows = 0.0
    for n in ([int(x) for x in c["lengths"].split(",")] if c["kind"] == "packed" else _valid_keys(c)):
        rows = n if c["kind"] == "packed" else min(Sq, n)
        kept = n if c["mask"] == "none" else min(c["window"], n)
        seen = rows * (n - rows) + rows * (rows + 1) / 2 if c["causal"] else rows * n
        pairs += seen * kept / n
        kept_rows += n if c["mask"] == "query" else kept
    q_bytes = 2.0 * B * Sq * H * d
    bias = 0 if c["mask"] == "none" else 2.0 * B * Hk * Sk * (Sq if c["mask"] == "query" else 1)
    total = 2 * q_bytes + 2 * kept_rows * Hk * d * 2 + bias
    if train:
        total += 2 * q_bytes + 2 * 2.0 * B * Sk * Hk * d + bias  # dOut read; dQ, dK, dV, dBias written
    return {"bytes": total, "flops": pairs * H * d * (14.0 if train else 4.0)}


def tolerance(case):
    """One rounding of inputs, probabilities and results to the data type, fp32 sums in between."""
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
