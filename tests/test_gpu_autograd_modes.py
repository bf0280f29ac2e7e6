"""The autograd node of the native host path under the autograd features a training program combines it with: saved-tensor
hooks and checkpointing, compiled autograd, second derivatives, threads that share a graph, tracing. The results are compared
with those of a plain call, bit for bit (deterministic gradients)."""
import threading

import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

DTYPE = torch.bfloat16
ROUTES = ["gathered", "bits", "dense", "packed"]


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def make(dev, route, d=64, seed=3):
    """(leaves, dout, call): one attention call on the given route of the native path as a function of its leaves."""
    from flash_sparse_attn import flash_sparse_attn_func, flash_sparse_attn_varlen_func
    from flash_sparse_attn.utils.mask import create_mask

    B, S, H, Hk = 2, 256, 4, 2
    rows = S if route == "bits" else 1
    q, k, v, bias, dout = (t.to(dev) for t in oracle.make_inputs(B, S, S, H, Hk, d, (B, Hk, rows, S), seed=seed, dtype=DTYPE))
    if route == "packed":
        leaves = [t.reshape(B * S, -1, d).requires_grad_(True) for t in (q, k, v)]
        cu = torch.tensor([0, 200, B * S], device=dev, dtype=torch.int32)

        def call(q, k, v):
            return flash_sparse_attn_varlen_func(q, k, v, cu, cu, 312, 312, is_causal=True, deterministic=True)

        return leaves, dout.reshape(B * S, H, d), call
    leaves = [t.requires_grad_(True) for t in (q, k, v, bias)]
    mask = create_mask(bias.detach(), None, B, S, S, 100, torch.finfo(DTYPE).min) if route != "dense" else None

    def call(q, k, v, bias):
        return flash_sparse_attn_func(q, k, v, mask, bias, is_causal=True, deterministic=True)

    return leaves, dout, call


def plain(leaves, dout, call):
    out = call(*leaves)
    assert out.grad_fn.name() == "FlashSparseAttnBackward"
    return (out.detach(), *torch.autograd.grad(out, leaves, dout))


def same(got, want):
    torch.cuda.synchronize()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("tail", [False, True])
def test_non_reentrant_checkpoint(dev, route, tail):
    """A checkpointed region that ends with the attention (the first node to unpack), or goes on after it."""
    from torch.utils.checkpoint import checkpoint

    leaves, dout, call = make(dev, route)

    def region(*t):
        out = call(*(x * 1.0 for x in t))
        return out * 1.0 if tail else out

    want = torch.autograd.grad(region(*leaves), leaves, dout)
    got = torch.autograd.grad(checkpoint(region, *leaves, use_reentrant=False), leaves, dout)
    same(got, want)


@pytest.mark.parametrize("route", ROUTES)
def test_compiled_autograd(dev, route):
    from torch._dynamo import compiled_autograd

    leaves, dout, call = make(dev, route)
    want = plain(leaves, dout, call)
    for _ in range(2):  # the second time from the cache of compiled graphs
        for t in leaves:
            t.grad = None
        out = call(*leaves)
        with compiled_autograd._enable(torch.compile(backend="eager", dynamic=False)):
            out.backward(dout)
        same([t.grad for t in leaves], want[1:])


@pytest.mark.parametrize("route", ROUTES)
def test_backward_twice(dev, route):
    leaves, dout, call = make(dev, route)
    want = plain(leaves, dout, call)
    out = call(*leaves)
    same(torch.autograd.grad(out, leaves, dout, retain_graph=True), want[1:])
    same(torch.autograd.grad(out, leaves, dout), want[1:])
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, leaves, dout)


def test_threads_share_a_graph(dev):
    """Two threads run the same graph backward, which is kept: neither sees the other's release of it."""
    leaves, dout, call = make(dev, "gathered")
    want = plain(leaves, dout, call)
    out = call(*leaves)
    torch.cuda.synchronize()
    results = []

    def work():
        for _ in range(10):
            results.append(torch.autograd.grad(out, leaves, dout, retain_graph=True))

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(results) == 20
    for r in results:
        same(r, want[1:])


@pytest.mark.parametrize("route", ROUTES)
def test_undefined_gradient(dev, route):
    """A consumer that returns no gradient for its input: the node is run without one."""
    leaves, dout, call = make(dev, route)

    class Drop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, g):
            return None

    grads = torch.autograd.grad(Drop.apply(call(*leaves)), leaves, dout, allow_unused=True)
    assert all(g is None or not g.any() for g in grads)


@pytest.mark.parametrize("route", ROUTES)
def test_second_derivative_is_refused(dev, route):
    """The gradients have no derivative of their own: a gradient penalty must fail, not train without the attention."""
    leaves, dout, call = make(dev, route)
    want = plain(leaves, dout, call)
    out = call(*leaves)
    grads = torch.autograd.grad(out, leaves, dout, create_graph=True)
    same([g.detach() for g in grads], want[1:])
    assert all(g.requires_grad for g in grads)
    with pytest.raises(RuntimeError, match="twice|second|not implemented|once_differentiable"):
        sum(g.float().pow(2).sum() for g in grads).backward()


def test_jit_trace_records_the_call(dev):
    """A traced function computes on its inputs; the call must not be baked in as a constant."""
    from flash_sparse_attn import flash_sparse_attn_func

    q, k, v, bias, _ = (t.to(dev) for t in oracle.make_inputs(1, 128, 128, 2, 1, 64, (1, 1, 128, 128), seed=1, dtype=DTYPE))

    def f(q, k, v, bias):
        return flash_sparse_attn_func(q, k, v, None, bias, is_causal=True)

    with torch.no_grad():
        traced = torch.jit.trace(f, (q, k, v, bias), check_trace=False)
        q2 = q.flip(1)
        assert torch.equal(traced(q2, k, v, bias), f(q2, k, v, bias))


def test_create_graph_without_a_bias_gradient(dev):
    """Inputs that are absent or not learned have no gradient; the others still carry the refusal of a second derivative."""
    from flash_sparse_attn import flash_sparse_attn_func

    leaves, dout, call = make(dev, "dense")
    q, k, v, bias = leaves
    for b in (None, bias.detach()):
        out = flash_sparse_attn_func(q, k, v.detach(), None, b, is_causal=True)
        dq, dk = torch.autograd.grad(out, (q, k), dout, create_graph=True)
        assert dq.requires_grad and dk.requires_grad
        with pytest.raises(RuntimeError, match="twice"):
            (dq.float().sum() + dk.float().sum()).backward()
