"""Layouts that the tensor-core kernels do not load themselves (bases off 16 bytes, strides that are no multiple of 8
elements, expanded dimensions) in q, k, v, bias and the output's gradient, on the routes whose kernels need more than the
general path: gathered keys, bit-packed masks, packed sequences. Against the same call on dense tensors, whose values
they hold."""
import pytest
import torch

from oracle import oracle

from test_gpu_attention import _kernel_status_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def odd_stride(t):
    """The same values with rows d + 1 elements apart and a base off 16 bytes."""
    wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 1, dtype=t.dtype, device=t.device)
    wide[..., 1:] = t
    return wide[..., 1:]


def off_base(t):
    """The same values, dense, from a base that is 2 bytes off."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


def expand_batch(t):
    return t[:1].expand_as(t)


LAYOUTS = {"odd_stride": odd_stride, "off_base": off_base, "expanded": expand_batch}
# ways a program uses the output, and with it the layout of its gradient: all rows stepped over with stride 0, rows of an
# odd width
USES = {
    "sum": lambda out, extra: out.sum(1),
    "sum_heads": lambda out, extra: out.sum(2),
    "sum_batch": lambda out, extra: out.sum(0),
    "cat": lambda out, extra: torch.cat([extra[..., : 3], out.flatten(-2)], -1),
    "cat_full": lambda out, extra: torch.cat([out.flatten(-2), extra[..., : 5]], -1)[..., 1:],
    "off_base": None,
}


def inputs(dev, route, d, dtype):
    B, S, H, Hk = 2, 256, 4, 2
    rows = S if route == "bits" else 1
    q, k, v, bias, dout = (t.to(dev) for t in oracle.make_inputs(B, S, S, H, Hk, d, (B, Hk, rows, S), seed=7, dtype=dtype))
    return q, k, v, bias, dout


def attend(route, q, k, v, bias, mask):
    from flash_sparse_attn import flash_sparse_attn_func, flash_sparse_attn_varlen_func

    if route == "packed":
        B, S = q.shape[:2]
        cu = torch.tensor([0, 100, B * S], device=q.device, dtype=torch.int32)
        flat = [t if t.dim() == 3 else t.flatten(0, 1) for t in (q, k, v)]
        return flash_sparse_attn_varlen_func(*flat, cu, cu, B * S, B * S, is_causal=True, deterministic=True).view(q.shape)
    return flash_sparse_attn_func(q, k, v, mask, bias, is_causal=True, deterministic=True)


def close(name, got, want, dtype):
    # the same sums in another order, or on the CUDA cores: twice the rounding of the results to 16 bits
    err = ((got.double() - want.double()).norm() / want.double().norm()).item()
    assert err < (1e-2 if dtype == torch.bfloat16 else 2e-3), (name, err)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("use", list(USES))
@pytest.mark.parametrize("route", ["gathered", "bits", "packed", "dense"])
def test_output_gradient(dev, route, use, d, dtype):
    if d == 256 and (route not in ("gathered", "dense") or dtype != torch.bfloat16):
        pytest.skip("no other kernel at this head dim")
    from flash_sparse_attn.utils.mask import create_mask

    q, k, v, bias, dout = inputs(dev, route, d, dtype)
    B, S = q.shape[:2]
    mask = create_mask(bias, None, B, S, S, 100, torch.finfo(dtype).min) if route in ("gathered", "bits") else None
    leaves = [t.requires_grad_(True) for t in ((q, k, v) if route == "packed" else (q, k, v, bias))]
    out = attend(route, q, k, v, bias, mask)
    extra = torch.zeros(B, S, 8, device=dev, dtype=dtype)
    seen = {}
    out.register_hook(lambda g: seen.__setitem__("g", g))
    if use == "off_base":
        got = torch.autograd.grad(out, leaves, off_base(dout), retain_graph=True)
    else:
        y = USES[use](out, extra)
        gen = torch.Generator(device=dev).manual_seed(1)
        got = torch.autograd.grad(y, leaves, torch.randn(y.shape, generator=gen, device=dev, dtype=dtype), retain_graph=True)
    g = seen["g"]
    assert g.data_ptr() % 16 or any(s % 8 or s == 0 for s in g.stride()[:-1])  # the layout is what it is meant to be
    want = torch.autograd.grad(out, leaves, g.contiguous().clone())
    torch.cuda.synchronize()
    _kernel_status_ok()
    for n, a, b in zip(("dq", "dk", "dv", "dbias"), got, want):
        close(n, a, b, dtype)


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("which", ["q", "kv", "bias", "all"])
@pytest.mark.parametrize("route", ["gathered", "bits", "packed", "dense"])
def test_inputs(dev, route, which, layout, d):
    from flash_sparse_attn.utils.mask import create_mask

    if d == 256 and route not in ("gathered", "dense"):
        pytest.skip("no other kernel at this head dim")
    if route == "packed" and (which == "bias" or layout == "expanded"):
        pytest.skip("packed calls have no bias and no batch")
    dtype = torch.bfloat16
    q, k, v, bias, dout = inputs(dev, route, d, dtype)
    B, S = q.shape[:2]
    f = LAYOUTS[layout]
    if route == "packed":
        q, k, v = (t.flatten(0, 1) for t in (q, k, v))
        dout = dout.flatten(0, 1)
    if which in ("q", "all"):
        q = f(q)
    if which in ("kv", "all"):
        k, v = f(k), f(v)
    if which in ("bias", "all"):
        bias = f(bias)

    def step(q, k, v, bias):
        t = [x.detach().requires_grad_(True) for x in (q, k, v, bias)]
        mask = create_mask(bias.contiguous(), None, B, S, S, 100, torch.finfo(dtype).min) if route in ("gathered", "bits") else None
        if route == "packed":
            from flash_sparse_attn import flash_sparse_attn_varlen_func

            cu = torch.tensor([0, 100, B * S], device=dev, dtype=torch.int32)
            out = flash_sparse_attn_varlen_func(t[0], t[1], t[2], cu, cu, B * S, B * S, is_causal=True, deterministic=True)
            t = t[:3]
        else:
            out = attend(route, *t, mask)
        return (out.detach(), *torch.autograd.grad(out, t, dout))

    got = step(q, k, v, bias)
    want = step(*(x.contiguous().clone(memory_format=torch.contiguous_format) for x in (q, k, v, bias)))
    torch.cuda.synchronize()
    _kernel_status_ok()
    for n, a, b in zip(("out", "dq", "dk", "dv", "dbias"), got, want):
        close(n, a, b, dtype)
