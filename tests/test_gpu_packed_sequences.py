"""Packed sequences in one launch: outputs, LSE and gradients against the fp32 oracle run on every sequence by itself, at
boundaries inside, at and around the 64- and 128-row tiles, with sequences that have fewer keys than queries, no queries or no keys."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _packed(lq, lk, H, Hk, d, dtype, causal, deterministic):
    from flash_sparse_attn import flash_sparse_attn_varlen_func

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(sum(lq) + d)
    q, k, v = (torch.randn(n, h, d, generator=g).to(dtype) for n, h in ((sum(lq), H), (sum(lk), Hk), (sum(lk), Hk)))
    dout = torch.randn(sum(lq), H, d, generator=g).to(dtype)
    cu_q, cu_k = (torch.tensor([0] + n, dtype=torch.int32).cumsum(0).to(torch.int32) for n in (lq, lk))
    qd, kd, vd = (t.to(dev).requires_grad_() for t in (q, k, v))
    out, lse, _ = flash_sparse_attn_varlen_func(qd, kd, vd, cu_q.to(dev), cu_k.to(dev), max(lq), max(lk), is_causal=causal,
                                                deterministic=deterministic, return_attn_probs=True)
    got = (out, *torch.autograd.grad(out, (qd, kd, vd), dout.to(dev)))
    want = [torch.zeros(t.shape) for t in (q, q, k, v)]
    for i in range(len(lq)):
        a, b = slice(int(cu_q[i]), int(cu_q[i + 1])), slice(int(cu_k[i]), int(cu_k[i + 1]))
        if lq[i] and lk[i]:
            r = oracle.attention_forward_backward(q[None, a], k[None, b], v[None, b], None, None, dout[None, a], None, causal)
            for t, x, rows in zip(want, (r[0], r[2], r[3], r[4]), (a, a, b, b)):
                t[rows] = x[0].float()
            assert torch.allclose(lse[:, a].cpu(), r[1][0].float(), atol=2e-2, rtol=0)
        else:
            assert torch.isposinf(lse[:, a]).all()
    for name, x, w in zip(("out", "dq", "dk", "dv"), got, want):
        ok, msg = oracle.within_tolerance(oracle.error_report(name, x.detach().cpu()[None], w[None]), name in ("dk", "dv"))
        assert ok, msg
    return got


@pytest.mark.parametrize("lq,lk", [
    ([63, 1, 64, 128, 127, 2], None), ([129, 300, 255], None), ([5, 700, 3], [200, 650, 1]), ([100, 0, 40, 90], [30, 77, 0, 200]),
    ([1, 1, 1, 1], None), ([1024, 1, 513], None),
])
@pytest.mark.parametrize("d,dtype,causal,deterministic", [(64, torch.bfloat16, True, False), (128, torch.float16, True, True),
                                                          (128, torch.bfloat16, False, False), (96, torch.bfloat16, True, False)])
def test_packed_sequences(lq, lk, d, dtype, causal, deterministic):
    _packed(lq, lk or lq, 4, 2, d, dtype, causal, deterministic)


def test_one_launch_equals_sequence_by_sequence(monkeypatch):
    """The same call with the single launch switched off: equal up to the order of the sums (a tile's split, the dQ adds)."""
    from flash_sparse_attn import flash_sparse_attn_interface as iface

    args = ([300, 17, 700, 128, 255], [300, 17, 700, 128, 255], 8, 2, 128, torch.bfloat16, True, False)
    one = _packed(*args)
    monkeypatch.setattr(iface, "_one_launch", lambda *a: None)
    many = _packed(*args)
    for a, b in zip(one, many):
        assert (a - b).float().norm() <= 4e-3 * b.float().norm()  # one bf16 rounding of each result
