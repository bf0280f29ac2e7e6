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


@pytest.mark.parametrize("lengths", [[100, 29, 300, 1, 82], [64, 64, 128], [257, 3, 3, 700]])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("which", ["q", "k", "v", "dout"])
@pytest.mark.parametrize("d,dtype,causal", [(64, torch.bfloat16, True), (128, torch.float16, False), (128, torch.bfloat16, True)])
def test_non_finite_values_stay_in_their_sequence(lengths, value, which, d, dtype, causal):
    """One sequence's q, k, v or output gradient holds non-finite values: every other sequence has the bits it has without."""
    from flash_sparse_attn import flash_sparse_attn_varlen_func

    dev = torch.device("cuda:0")
    n, H, Hk = sum(lengths), 4, 2
    cu = torch.tensor([0] + lengths, device=dev).cumsum(0).to(torch.int32)
    gen = torch.Generator(device=dev).manual_seed(n + d)
    t = {x: torch.randn(n, h, d, generator=gen, device=dev, dtype=dtype) for x, h in (("q", H), ("k", Hk), ("v", Hk), ("dout", H))}

    def run():
        leaves = [t[x].detach().clone().requires_grad_() for x in "qkv"]
        out, lse, _ = flash_sparse_attn_varlen_func(*leaves, cu, cu, max(lengths), max(lengths), is_causal=causal,
                                                    deterministic=True, return_attn_probs=True)
        return (out.detach(), lse.t(), *torch.autograd.grad(out, leaves, t["dout"]))

    clean = run()
    for i in range(len(lengths)):
        a, b = int(cu[i]), int(cu[i + 1])
        keep = t[which].clone()
        t[which][a:b] = value
        got = run()
        t[which].copy_(keep)
        others = torch.ones(n, dtype=torch.bool, device=dev)
        others[a:b] = False
        for name, x, y in zip(("out", "lse", "dq", "dk", "dv"), got, clean):
            assert torch.equal(x[others], y[others]), (name, i)


@pytest.mark.parametrize("lengths", [[1] * 40 + [200] + [3] * 30, [2, 0, 1] * 400 + [129]])
def test_many_short_sequences(lengths):
    """More sequences than one and than two rounds of the search for a tile's sequence tell apart."""
    _packed(lengths, lengths, 2, 1, 64, torch.bfloat16, True, True)


def test_boundaries_may_change_before_the_backward():
    from flash_sparse_attn import flash_sparse_attn_varlen_func

    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(1)
    leaves = [torch.randn(500, h, 64, generator=gen, device=dev, dtype=torch.bfloat16).requires_grad_() for h in (4, 2, 2)]
    dout = torch.randn(500, 4, 64, generator=gen, device=dev, dtype=torch.bfloat16)
    got = []
    for change in (False, True):
        cu = torch.tensor([0, 200, 500], device=dev, dtype=torch.int32)
        out = flash_sparse_attn_varlen_func(*leaves, cu, cu, 300, 300, is_causal=True, deterministic=True)
        if change:
            cu.copy_(torch.tensor([0, 100, 500], device=dev))
        got.append(torch.autograd.grad(out, leaves, dout))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("causal", [False, True])
def test_rows_outside_every_sequence(causal):
    """Through the C ABI: boundaries that leave out tokens at both ends. Those give 0, LSE = +inf and gradients 0, also where their
    q, k, v hold NaN; the sequences have the results they have without."""
    import ctypes

    from flash_sparse_attn import _lib
    from flash_sparse_attn import flash_sparse_attn_interface as iface

    lib, dev, dtype = _lib.load(), torch.device("cuda:0"), torch.bfloat16
    for name in ("fdma_fwd_varlen", "fdma_bwd_varlen"):
        getattr(lib, name).argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p]
    stream = torch.cuda.current_stream(dev).cuda_stream
    H, Hk, d, before, after = 4, 2, 64, 70, 35
    lengths = [130, 1, 300]
    total = before + sum(lengths) + after
    gen = torch.Generator(device=dev).manual_seed(5)
    q, k, v, dout = (torch.randn(1, total, h, d, generator=gen, device=dev).to(dtype) for h in (H, Hk, Hk, H))
    inside = torch.zeros(total, dtype=torch.bool, device=dev)
    inside[before:total - after] = True

    def run(q, k, v, dout, cu):
        n = q.shape[1]
        cu = torch.tensor(cu, device=dev, dtype=torch.int32)
        out, lse = torch.full_like(q, 7.0), torch.full((1, H, n), 7.0, device=dev)
        p = _lib.FwdParams()
        iface._fill_fwd(p, q, k, v, None, None, out, lse, d ** -0.5, causal)
        assert lib.fdma_fwd_varlen(ctypes.addressof(p), cu.data_ptr(), cu.data_ptr(), cu.numel() - 1, stream) == 0
        grads = [torch.full_like(t, 7.0) for t in (q, k, v)]
        bp = _lib.BwdParams()
        iface._fill_fwd(bp.f, q, k, v, None, None, out, lse, d ** -0.5, causal)
        bp.dout, (bp.dq, bp.dk, bp.dv) = dout.data_ptr(), (g.data_ptr() for g in grads)
        for name, t in zip(("do", "dq", "dk", "dv"), (dout, *grads)):
            for dim, s in zip(("batch", "row", "head"), iface._bsh(t)):
                setattr(bp, f"{name}_{dim}_stride", s)
        bp.deterministic = 1
        need = lib.fdma_bwd_workspace_bytes(ctypes.byref(bp))
        ws = torch.empty(need, dtype=torch.uint8, device=dev)
        bp.f.workspace, bp.f.workspace_bytes = ws.data_ptr(), need
        assert lib.fdma_bwd_varlen(ctypes.addressof(bp), cu.data_ptr(), cu.data_ptr(), cu.numel() - 1, stream) == 0
        torch.cuda.synchronize()
        return out[0], lse[0].t(), *(g[0] for g in grads)

    cu = torch.tensor([0] + lengths).cumsum(0)
    want = run(*(t[:, inside].contiguous() for t in (q, k, v, dout)), cu.tolist())
    for t in (q, k, v):
        t[:, ~inside] = float("nan")
    got = run(q, k, v, dout, (cu + before).tolist())
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        rest = a[~inside]
        assert torch.isposinf(rest).all() if name == "lse" else (rest == 0).all(), name
        err = (a[inside].float() - b.float()).norm() / b.float().norm()  # (query tiles are cut at other rows)
        assert err <= 4e-3, (name, err)
