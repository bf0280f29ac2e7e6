"""Backward kernel of row-broadcast masks and biases (head dims up to 128), at the sizes where its two passes can go wrong: more keys
than dQ is summed over in tensor memory, whole 64-key tiles masked out, query heads without any kept key, more rows than keys,
single rows, ragged ends. Against the same sums in 64 bits.

Bound: P, dS, O (through D = rowsum(dO o O)) and the result are each rounded to 16 bits once, a relative error of at most half an ulp,
u = 2^-9 (bf16) or 2^-12 (fp16), in each; four of them bound the 2-norm of the difference relative to that of the result."""
import pytest
import torch

from flash_sparse_attn import flash_sparse_attn_func
from flash_sparse_attn import flash_sparse_attn_interface as iface

pytestmark = pytest.mark.gpu

# (batch, queries, keys, heads, kv heads, head dim, mask heads, bias heads, bias batch, causal)
CASES = [
    (1, 300, 4200, 4, 2, 64, 0, 0, 1, False),     # 66 steps a row: sums leave tensor memory on the way
    (1, 130, 8256, 3, 1, 128, 1, 1, 1, False),    # 129 steps less the masked tiles
    (2, 4300, 4300, 2, 2, 72, 0, 2, 2, True),
    (1, 129, 127, 4, 1, 128, 0, 1, 1, True),      # two rows see no key
    (1, 400, 64, 2, 1, 64, 0, 0, 1, True),        # whole tiles of rows see no key
    (3, 1, 200, 4, 2, 128, 2, 2, 3, False),       # a single query
    (2, 257, 383, 6, 2, 96, 6, 6, 2, True),       # mask and bias per query head, one head without a kept key
    (2, 193, 320, 4, 2, 128, 1, 1, 1, True),      # dBias summed over batch and heads
]


def exact(q, k, v, mask, bias, dout, causal):
    """out, dq, dk, dv (and dbias) in 64 bits."""
    H, Sq, Sk = q.shape[2], q.shape[1], k.shape[1]
    leaves = [t.detach().double().requires_grad_() for t in (q, k, v)] + ([bias.detach().double().requires_grad_()] if bias is not None else [])
    rep = lambda t: t.repeat_interleave(H // t.shape[1], 1)  # noqa: E731
    Q, K, V = (t.transpose(1, 2) for t in leaves[:3])
    s = Q @ rep(K).transpose(-1, -2) * q.shape[-1] ** -0.5
    if bias is not None:
        s = s + rep(leaves[3])
    seen = torch.ones(Sq, Sk, dtype=torch.bool, device=q.device)
    if causal:
        seen = torch.arange(Sk, device=q.device)[None] <= torch.arange(Sq, device=q.device)[:, None] + Sk - Sq
    seen = seen[None, None].expand(q.shape[0], H, Sq, Sk)
    if mask is not None:
        seen = seen & rep(mask)
    alive = seen.any(-1, keepdim=True)
    p = torch.softmax(s.masked_fill(~seen & alive, float("-inf")), -1) * alive
    out = (p @ rep(V)).transpose(1, 2)
    return [out] + list(torch.autograd.grad(out, leaves, dout.double()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_gradients(case, dtype):
    B, Sq, Sk, H, Hk, d, hm, hb, bb, causal = case
    g = torch.Generator(device="cuda").manual_seed(7)
    r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=dtype)  # noqa: E731
    q, k, v, dout = r(B, Sq, H, d), r(B, Sk, Hk, d), r(B, Sk, Hk, d), r(B, Sq, H, d)
    mask = bias = None
    if hm:
        mask = torch.rand((B, hm, 1, Sk), generator=g, device="cuda") < 0.4
        mask[..., Sk // 3: Sk // 3 + 150] = False  # whole 64-key tiles where there are that many keys
        mask[..., 0] = True
        if hm == H:
            mask[0, 1] = False
    if hb:
        bias = r(bb, hb, 1, Sk).requires_grad_()
    for t in (q, k, v):
        t.requires_grad_()
    learned = [q, k, v] + ([bias] if hb else [])
    runs = []
    iface.set_compaction("off")
    try:
        for _ in range(2):
            out = flash_sparse_attn_func(q, k, v, attn_mask=mask, attn_bias=bias, is_causal=causal)
            runs.append([out.detach(), *torch.autograd.grad(out, learned, dout)])
    finally:
        iface.set_compaction("auto")
    want = exact(q, k, v, mask, bias, dout, causal)
    bound = 4 * (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), runs[0], want):
        err = ((got.double() - ref).norm() / ref.norm().clamp_min(1e-30)).item()
        assert err <= bound, (name, err, bound)
    assert torch.equal(runs[0][1], runs[1][1])  # dQ has one order of summation
