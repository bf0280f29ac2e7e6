"""The whole call -- create_mask, gathered-keys forward and backward -- recorded once into a CUDA graph and replayed
on new data: nothing in the library allocates, synchronises or reads device results on the host once the one-time
set-up of a first (eager) call is done. Replayed results are compared with an eager call on the same data
(bit-exact for out, dK, dV and dBias; dQ is accumulated with reduce-adds whose order is not fixed, so it is compared
within 1e-2 of its largest value) and with the fp32 oracle at the usual tolerances."""
import pytest
import torch

from oracle import oracle

from test_gpu_attention import check, _kernel_status_ok

pytestmark = pytest.mark.gpu


def test_forward_backward_in_a_cuda_graph():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.utils.mask import create_mask

    dev = torch.device("cuda:0")
    B, S, H, Hk, d, W = 1, 1024, 4, 2, 128, 256
    dtype = torch.bfloat16
    min_dtype = torch.finfo(dtype).min

    def data(seed):
        q, k, v, bias, dout = oracle.make_inputs(B, S, S, H, Hk, d, (B, Hk, 1, S), seed=seed, dtype=dtype)
        return [t.to(dev) for t in (q, k, v, bias, dout)]

    static = data(1)
    q, k, v, bias, dout = static
    for t in (q, k, v, bias):
        t.requires_grad_(True)

    def call():
        mask = create_mask(bias.detach(), None, B, S, S, W, min_dtype)
        out = flash_sparse_attn_func(q, k, v, attn_mask=mask, attn_bias=bias, is_causal=True)
        out.backward(dout)
        return out

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # eager warm-up: one-time set-up of the library, gradient buffers
        for _ in range(2):
            call()
    torch.cuda.current_stream().wait_stream(side)
    for t in (q, k, v, bias):
        t.grad.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out_static = call()

    for seed in (2, 3):
        fresh = data(seed)
        with torch.no_grad():
            for dst, src in zip(static, fresh):
                dst.copy_(src)
            for t in (q, k, v, bias):
                t.grad.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _kernel_status_ok()
        got = [out_static.detach().clone()] + [t.grad.detach().clone() for t in (q, k, v, bias)]
        # eager call on the same data
        e = [t.detach().clone().requires_grad_(i < 4) for i, t in enumerate(fresh)]
        mask = create_mask(e[3].detach(), None, B, S, S, W, min_dtype)
        o = flash_sparse_attn_func(e[0], e[1], e[2], attn_mask=mask, attn_bias=e[3], is_causal=True)
        o.backward(e[4])
        want = [o.detach(), e[0].grad, e[1].grad, e[2].grad, e[3].grad]
        for name, a, b_ in zip(("out", "dq", "dk", "dv", "dbias"), got, want):
            if name == "dq":
                assert (a.float() - b_.float()).abs().max() <= 1e-2 * b_.float().abs().max(), name
            else:
                assert torch.equal(a, b_), name
        ref = oracle.attention_forward_backward(*(t.detach().cpu() for t in fresh[:3]), mask.cpu(),
                                                fresh[3].detach().cpu(), fresh[4].cpu(), None, True)
        check("out", got[0].cpu(), ref[0], dtype)
        check("dq", got[1].cpu(), ref[2], dtype)
        check("dk", got[2].cpu(), ref[3], dtype, reduced=True)
        check("dv", got[3].cpu(), ref[4], dtype, reduced=True)
        check("dbias", got[4].cpu(), ref[5], dtype, reduced=True)


def test_replay_beside_eager_launches():
    """A captured forward replayed on one stream while eager calls of another size run on a second one, several hundred of
    each: every launch hands out its own work items, whatever runs beside it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from flash_sparse_attn import flash_sparse_attn_func

    dev, dtype = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator(device=dev).manual_seed(2)
    small = [torch.randn(1, 1024, h, 64, generator=g, device=dev, dtype=dtype) for h in (4, 2, 2)]
    large = [torch.randn(2, 2048, h, 64, generator=g, device=dev, dtype=dtype) for h in (16, 2, 2)]
    with torch.no_grad():
        want_small, want_large = (flash_sparse_attn_func(*t, is_causal=True) for t in (small, large))
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = flash_sparse_attn_func(*small, is_causal=True)
        streams = torch.cuda.Stream(), torch.cuda.Stream()
        replays, eager = [], []
        for i in range(600):
            with torch.cuda.stream(streams[0]):
                out.fill_(float("nan"))
                graph.replay()
                replays.append((out == want_small).all())
            with torch.cuda.stream(streams[1]):
                eager.append((flash_sparse_attn_func(*large, is_causal=True) == want_large).all())
        torch.cuda.synchronize()
    assert torch.stack(replays).all() and torch.stack(eager).all()
