"""How exactly the backward kernel of row-broadcast masks (head dims up to 128) adds up dQ, dK and dV. The tensor core truncates the
sums it holds, so a long one comes out too small; next to the 16-bit rounding of P, dS and the result that is hard to see, so the inputs
here make all of these exact. Q and K are non-zero in different columns: every score is 0 and P is a power of two. V is non-zero in
one column, with few bits there and pairs of keys of opposite sign, so that D = 0; dO has few bits in that column, so that dS = P dO V is
exact. K takes the sign of V's column: the terms of each dQ element are positive. Q and dO are positive, so are those of dV, and those of
a row of dK have one sign.

Bound: a sum of n additions in tensor memory, each of which loses less than one unit in the last of 24 bits (2^-23 of it) and on average
half of that, is too small by at most n 2^-24 on average; the 32-bit sums of what leaves tensor memory round to nearest. A result is the
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
    return ((got.double() - exact.half().double()) / exact)[used].mean().item(), int(used.sum())


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
    loss, n = _shortfall(dq, exact)
    assert abs(loss) <= _bound(8, n), (loss, _bound(8, n))
