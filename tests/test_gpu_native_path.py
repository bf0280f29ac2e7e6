"""The default route of an eager call (native host path, gathered keys written back by the finish kernel, head dims below
the tile's) at the sizes where it can go wrong: head dims around the tile widths 64 / 128 / 256, key counts one beside a
tile, lists shared by batch or heads, more kv heads than one CTA of the finish kernel takes. Against the fp32 oracle with
the bounds of `oracle.within_tolerance`."""
import pytest
import torch

from oracle import oracle

from test_gpu_attention import check, _kernel_status_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


# (B, Sq, Sk, H, Hk, d), window, mask heads (0: one per kv head), bias heads (0: none), dtype, deterministic
CASES = [
    ((1, 129, 257, 2, 1, 8), 100, 0, 1, torch.bfloat16, False),      # a single 16-byte piece per row
    ((2, 200, 385, 4, 2, 40), 129, 0, 2, torch.bfloat16, False),     # below the 64-wide tile, 16-byte rows that are not 32
    ((2, 256, 512, 4, 2, 64), 128, 0, 2, torch.float16, False),
    ((1, 320, 640, 8, 2, 64), 300, 0, 8, torch.bfloat16, True),      # per-query-head bias, deterministic
    ((1, 192, 513, 4, 4, 72), 200, 0, 4, torch.bfloat16, False),     # just above 64
    ((1, 300, 1000, 6, 2, 96), 333, 0, 2, torch.bfloat16, True),
    ((2, 256, 384, 4, 2, 128), 60, 1, 2, torch.bfloat16, False),     # one list for all heads
    ((1, 128, 129, 40, 20, 120), 64, 0, 20, torch.bfloat16, False),  # 20 kv heads: two head groups of the finish kernel
    ((1, 130, 384, 4, 2, 136), 100, 0, 2, torch.bfloat16, False),    # just above 128
    ((1, 256, 640, 4, 1, 200), 257, 0, 1, torch.bfloat16, True),
    ((1, 256, 640, 2, 2, 256), 257, 0, 0, torch.bfloat16, False),    # no bias
]


@pytest.mark.parametrize("geom,window,mask_heads,bias_heads,dtype,det", CASES)
def test_gathered_route(dev, geom, window, mask_heads, bias_heads, dtype, det):
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.utils.mask import create_mask

    B, Sq, Sk, H, Hk, d = geom
    q, k, v, bias, dout = oracle.make_inputs(B, Sq, Sk, H, Hk, d, (B, bias_heads or Hk, 1, Sk), seed=3, dtype=dtype)
    sel = bias[:, :: bias.shape[1] // (mask_heads or Hk)].contiguous()
    mask = create_mask(sel.to(dev), None, B, Sq, Sk, window, torch.finfo(dtype).min)
    assert torch.equal(mask.cpu(), oracle.create_mask(sel, None, B, Sq, Sk, window, torch.finfo(dtype).min))
    ref = oracle.attention_forward_backward(q, k, v, mask.cpu(), bias if bias_heads else None, dout, None, True)
    ql, kl, vl, bl = (t.to(dev).requires_grad_(True) for t in (q, k, v, bias))
    out = flash_sparse_attn_func(ql, kl, vl, mask, bl if bias_heads else None, is_causal=True, deterministic=det)
    assert out.grad_fn.name() == "FlashSparseAttnBackward"
    out.backward(dout.to(dev))
    torch.cuda.synchronize()
    _kernel_status_ok()
    check("out", out.detach().cpu(), ref[0], dtype)
    check("dq", ql.grad.cpu(), ref[2], dtype)
    check("dk", kl.grad.cpu(), ref[3], dtype, reduced=True)
    check("dv", vl.grad.cpu(), ref[4], dtype, reduced=True)
    if bias_heads:
        check("dbias", bl.grad.cpu(), ref[5], dtype, reduced=True)
    dropped = ~mask[:, :, 0].cpu().expand(B, Hk, Sk)
    assert bool((kl.grad.cpu().permute(0, 2, 1, 3)[dropped] == 0).all())


@pytest.mark.parametrize("d", [24, 64, 80, 128])
@pytest.mark.parametrize("rows", [1, 200])
def test_full_range_route(dev, d, rows):
    """No gathering (the mask keeps most keys, or differs by query): ragged lengths, head dims beside the tiles."""
    from flash_sparse_attn import flash_sparse_attn_func

    B, Sq, Sk, H, Hk = 2, 200, 330, 4, 2
    dtype = torch.bfloat16
    q, k, v, bias, dout = oracle.make_inputs(B, Sq, Sk, H, Hk, d, (B, Hk, rows, Sk), seed=5, dtype=dtype)
    g = torch.Generator().manual_seed(1)
    mask = torch.rand((B, Hk, rows, Sk), generator=g) < 0.9
    ref = oracle.attention_forward_backward(q, k, v, mask, bias, dout, None, True)
    ql, kl, vl, bl = (t.to(dev).requires_grad_(True) for t in (q, k, v, bias))
    out = flash_sparse_attn_func(ql, kl, vl, mask.to(dev), bl, is_causal=True)
    out.backward(dout.to(dev))
    torch.cuda.synchronize()
    _kernel_status_ok()
    check("out", out.detach().cpu(), ref[0], dtype)
    check("dq", ql.grad.cpu(), ref[2], dtype)
    check("dk", kl.grad.cpu(), ref[3], dtype, reduced=True)
    check("dv", vl.grad.cpu(), ref[4], dtype, reduced=True)
    check("dbias", bl.grad.cpu(), ref[5], dtype, reduced=True)


def test_threads_and_streams(dev):
    """Calls from several host threads on streams of their own give what one thread gives."""
    import threading

    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.utils.mask import create_mask

    B, S, H, Hk, d = 1, 512, 4, 2, 64
    dtype = torch.bfloat16
    q, k, v, bias, dout = (t.to(dev) for t in oracle.make_inputs(B, S, S, H, Hk, d, (B, Hk, 1, S), seed=9, dtype=dtype))

    def step():
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v, bias)]
        mask = create_mask(leaves[3].detach(), None, B, S, S, 128, torch.finfo(dtype).min)
        out = flash_sparse_attn_func(leaves[0], leaves[1], leaves[2], mask, leaves[3], is_causal=True, deterministic=True)
        return (out.detach(), *torch.autograd.grad(out, leaves, dout))

    want = step()
    torch.cuda.synchronize()
    results = {}

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                results[i] = step()
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    _kernel_status_ok()
    for r in results.values():
        assert all(torch.equal(a, b) for a, b in zip(r, want))


def test_forward_mode_tangent_is_not_dropped(dev):
    """The node has no jvp: a dual tensor must reach the Python path, which refuses it, and not lose its tangent."""
    from flash_sparse_attn import flash_sparse_attn_func

    q, k, v = (torch.randn(1, 128, 2, 64, device=dev, dtype=torch.bfloat16) for _ in range(3))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(q, torch.ones_like(q))
        with pytest.raises((RuntimeError, NotImplementedError)):
            flash_sparse_attn_func(dual, k, v, is_causal=True)
