"""Backward at head dims above 128: the three passes (dK, dV, dQ) at tile remainders, with 64-key tiles that hold no kept key, rows
before the first visible key, more keys than queries, head groups, on the full key range and on gathered keys, against the oracle;
and the same bits on a second run (no atomics)."""
import pytest
import torch

from oracle import oracle

from test_gpu_attention import _kernel_status_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route", ["off", "auto"])
@pytest.mark.parametrize("B,Sq,Sk,H,Hk,d,causal,dtype", [
    (1, 1, 300, 2, 1, 256, False, torch.bfloat16), (2, 65, 65, 2, 2, 136, True, torch.float16), (1, 128, 513, 4, 1, 256, True, torch.bfloat16),
    (1, 700, 260, 2, 1, 192, True, torch.bfloat16), (1, 1023, 1023, 4, 2, 256, True, torch.float16), (2, 257, 640, 3, 3, 256, False, torch.bfloat16),
])
def test_gradients(B, Sq, Sk, H, Hk, d, causal, dtype, route):
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn import flash_sparse_attn_interface as iface

    dev = torch.device("cuda:0")
    q, k, v, bias, dout = oracle.make_inputs(B, Sq, Sk, H, Hk, d, (B, Hk, 1, Sk), seed=Sq + Sk, dtype=dtype, device="cpu")
    mask = torch.rand(B, Hk, 1, Sk, generator=torch.Generator().manual_seed(1)) < 0.4
    mask[..., 64:192] = False  # two 64-key tiles without a kept key
    mask[..., -1] = True
    want = oracle.attention_forward_backward(q, k, v, mask, bias, dout, None, causal)
    iface.set_compaction(route)
    try:
        runs = []
        for _ in range(2):
            leaves = [t.to(dev).requires_grad_() for t in (q, k, v, bias)]
            out = flash_sparse_attn_func(*leaves[:3], attn_mask=mask.to(dev), attn_bias=leaves[3], is_causal=causal)
            runs.append((out, *torch.autograd.grad(out, leaves, dout.to(dev))))
    finally:
        iface.set_compaction("auto")
    for name, got, ref in zip(("out", "dq", "dk", "dv", "dbias"), runs[0], (want[0], *want[2:])):
        ok, msg = oracle.within_tolerance(oracle.error_report(name, got.detach().cpu(), ref), name in ("dk", "dv", "dbias"))
        assert ok, msg
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("Sq,Sk,d,kept,deterministic", [(200, 65536, 256, None, True), (64, 4160, 256, None, False), (130, 20000, 192, None, True),
                                                        (100, 40000, 136, 0.9, False)])
def test_dq_over_many_keys(Sq, Sk, d, kept, deterministic):
    """dQ over more keys than the tensor core sums up in one go (4096), in fp16: within 1 % of the error that rounding dS and
    dQ to 16 bits makes of the exact ones (truncated sums over all 65536 keys made it 3 %)."""
    from flash_sparse_attn import flash_sparse_attn_func

    dev, dtype, H = torch.device("cuda:0"), torch.float16, 2
    gen = torch.Generator(device=dev).manual_seed(Sk)
    q, k, v, dout = (torch.randn(1, n, h, d, generator=gen, device=dev, dtype=dtype) for n, h in ((Sq, H), (Sk, 1), (Sk, 1), (Sq, H)))
    mask = None if kept is None else torch.rand((1, 1, 1, Sk), generator=gen, device=dev) < kept
    q.requires_grad_()
    out = flash_sparse_attn_func(q, k, v, mask, None, deterministic=deterministic)
    dq, = torch.autograd.grad(out, q, dout)
    torch.cuda.synchronize()
    _kernel_status_ok()
    Q, G = (t.detach()[0].double().transpose(0, 1) for t in (q, dout))
    K, V = k[0, :, 0].double(), v[0, :, 0].double()
    s = Q @ K.T * d ** -0.5
    if mask is not None:
        s = s.masked_fill(~mask[0], float("-inf"))
    P = torch.softmax(s, -1)
    dP = G @ V.T
    dS = P * (dP - (P * dP).sum(-1, keepdim=True))
    exact = dS @ K * d ** -0.5
    rounded = (dS.to(dtype).double() @ K * d ** -0.5).to(dtype).double()
    err = (dq[0].double().transpose(0, 1) - exact).norm().item()
    assert err <= 1.01 * (rounded - exact).norm().item(), err / (rounded - exact).norm().item()
