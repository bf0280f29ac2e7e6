"""How exactly the backward kernel of row-broadcast masks (head dims up to 128) adds up dQ, dK and dV. The tensor core truncates the
sums it holds, so a long one comes out too small; next to the 16-bit rounding of P, dS and the result that is hard to see, so the inputs
here make all of these exact. Q and K are non-zero in different columns: every score is 0 and P is a power of two. V is non-zero in
one column, with few bits there and pairs of keys of opposite sign, so that D = 0; dO has few bits in that column, so that dS = P dO V is
exact. K takes the sign of V's column: the terms of each dQ element are positive. Q and dO are positive, so are those of dV, and those of
a row of dK have one sign.

Bound: what n additions in tensor memory lose if each loses half a unit in the last of 24 bits, n 2^-24 (an addition takes in 16 products,
aligned to the largest of them, and measured it loses up to 1.5 times that; the kernel makes fewer of them than the bounds of dK and dV
allow for); the 32-bit sums of what leaves tensor memory round to nearest. A result is the
rounded exact one unless such a loss moves it over a boundary of rounding, one fp16 step (at most 2^-10 of it) further on, which
happens with a probability of loss / step: that mean has a standard deviation of at most sqrt(loss 2^-10 / N) over N elements, and four
of them are allowed."""
import pytest
import torch

from flash_sparse_attn import flash_sparse_attn_func
from flash_sparse_attn import flash_sparse_attn_interface as iface

pytestmark = pytest.mark.gpu


def _exact_inputs(B, Sq, Sk, H, Hk, seed):
    """q, k, v, dout in fp16, as described above."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    ints = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, device="cuda")  # noqa: E731
    q, k, v = (torch.zeros(B, n, h, 128, device="cuda", dtype=torch.float16) for n, h in ((Sq, H), (Sk, Hk), (Sk, Hk)))
    q[..., :64] = (ints(1024, 2048, B, Sq, H, 64) / 1024).half()
    sign = (1 - 2 * (torch.arange(Sk, device="cuda") % 2)).view(1, Sk, 1, 1)
    k[..., 64:] = (ints(1024, 2048, B, Sk, Hk, 64) * sign / 1024).half()
    v[..., :1] = (ints(8, 16, B, Sk // 2, Hk, 1).repeat_interleave(2, 1) * sign / 8).half()
    dout = (ints(1024, 2048, B, Sq, H, 128) / 1024).half()
    dout[..., :1] = (ints(64, 128, B, Sq, H, 1) / 64).half()
    return q, k, v, dout


def _shortfall(got, exact):
    """Mean relative difference to the rounded exact values, over the elements that are not zero; negative: too small."""
    used = exact != 0
    return ((got.double() - exact.half().double()) / exact)[used].mean().item()


def _bound(additions, elements):
    loss = additions * 2.0 ** -24
    return loss + 4 * (loss * 2.0 ** -10 / elements) ** 0.5


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("Sk", [2048, 8192])
def test_dq_sums(Sk, deterministic):
    """dQ leaves tensor memory every 128 keys: eight additions of 16 keys each."""
    B, Sq, H, Hk = 2, 256, 32, 16
    q, k, v, dout = _exact_inputs(B, Sq, Sk, H, Hk, Sk)
    q.requires_grad_()
    iface.set_compaction("off")
    try:
        out = flash_sparse_attn_func(q, k, v, softmax_scale=0.125, deterministic=deterministic)
        dq, = torch.autograd.grad(out, q, dout)
    finally:
        iface.set_compaction("auto")
    ds = dout[..., 0].double()[..., None] / Sk  # times V's column: dS, (B, Sq, H, 1)
    kv = torch.einsum("bkh,bkhd->bhd", v[..., 0].double(), k.double()).repeat_interleave(H // Hk, 1)
    exact = ds * kv[:, None] * 0.125
    loss, bound = _shortfall(dq, exact), _bound(8, B * Hk * 64 * 64)  # (64 values of dO's column, 64 columns of K: the others repeat them)
    assert abs(loss) <= bound, (loss, bound)


@pytest.mark.parametrize("B,Sq,Sk,H,Hk", [(2, 4096, 4096, 32, 8), (4, 4160, 4096, 16, 2)])
def test_dk_dv_sums(B, Sq, Sk, H, Hk):
    """dK and dV leave tensor memory within 64 steps of 64 queries, 256 additions of 16 queries each, whether one CTA works on all queries
    of all heads of the group (4 heads x 64 tiles of 64 queries), or on half of them (8 heads x 33 and 32 tiles)."""
    q, k, v, dout = _exact_inputs(B, Sq, Sk, H, Hk, Sq)
    k.requires_grad_(), v.requires_grad_()
    iface.set_compaction("off")
    try:
        out = flash_sparse_attn_func(q, k, v, softmax_scale=0.125)
        dk, dv = torch.autograd.grad(out, (k, v), dout)
    finally:
        iface.set_compaction("auto")
    G = H // Hk
    heads = lambda t: t.double().view(B, Sq, Hk, G, *t.shape[3:])  # noqa: E731
    dv_exact = (heads(dout).sum((1, 3)) / Sk)[:, None].expand(B, Sk, Hk, 128)
    c = torch.einsum("bqhg,bqhgd->bhd", heads(dout[..., 0]), heads(q)) / Sk * 0.125
    dk_exact = v[..., :1].double() * c[:, None]
    # (dV is the same for every key, dK for every key with the same of 8 values of V)
    for name, got, exact, n in (("dk", dk, dk_exact, B * Hk * 64 * 8), ("dv", dv, dv_exact, B * Hk * 127)):
        loss, bound = _shortfall(got, exact), _bound(256, n)
        assert abs(loss) <= bound, (name, loss, bound)
