"""Single-query forward over a list of kept keys (create_mask -> flash_sparse_attn_func) and over a plain bool mask or no
mask, at the sizes where the decode kernel can go wrong: lists around its 16-row stages, head groups that do not fill or
exceed the 16 rows of a product, head dims beside the 32-wide blocks, lists so long that several clusters share them.
Against the fp32 oracle with the bounds of `oracle.within_tolerance`."""
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


# (B, Sk, H, Hk, d), window, bias heads, dtype, padded
CASES = [
    ((1, 40, 2, 2, 8), 15, 2, torch.bfloat16, False),         # one stage, not full; a single 16-byte piece per row
    ((2, 100, 6, 2, 40), 17, 2, torch.bfloat16, False),       # one key into the second stage; groups of 3
    ((3, 333, 4, 2, 64), 64, 4, torch.float16, True),         # bias row per query head; lists of unequal length
    ((1, 1000, 24, 2, 96), 500, 2, torch.bfloat16, False),    # groups of 12
    ((2, 4097, 16, 1, 128), 1024, 1, torch.bfloat16, True),   # groups of 16, odd key count
    ((1, 700, 40, 2, 128), 123, 1, torch.bfloat16, False),    # groups of 20: two head blocks; one bias row for all
    ((2, 600, 16, 2, 200), 300, 2, torch.float16, False),
    ((1, 900, 16, 1, 256), 77, 1, torch.bfloat16, False),     # 16 heads at d > 128: two head blocks
    ((1, 70000, 2, 1, 128), 20000, 1, torch.bfloat16, False),  # several clusters per list, merge kernel
]


@pytest.mark.parametrize("geom,window,bias_heads,dtype,padded", CASES)
def test_kept_list(dev, geom, window, bias_heads, dtype, padded):
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.utils.mask import create_mask

    B, Sk, H, Hk, d = geom
    q, k, v, bias, _ = (None if t is None else t.to(dev)
                        for t in oracle.make_inputs(B, 1, Sk, H, Hk, d, (B, bias_heads, 1, Sk), seed=4, dtype=dtype))
    sel = bias if bias_heads in (1, Hk) else bias[:, ::H // Hk].contiguous()
    padding = None
    if padded:  # the last sequence has fewer valid keys than the window
        padding = torch.arange(Sk, device=dev)[None] >= torch.tensor([0] * (B - 1) + [Sk - window // 2], device=dev)[:, None]
        k[-1, : Sk - window // 2] = float("nan")  # rows that are not kept are never read
        v[-1, : Sk - window // 2] = float("nan")
    mask = create_mask(sel, padding, B, 1, Sk, window, torch.finfo(dtype).min)
    with torch.no_grad():
        out = flash_sparse_attn_func(q, k, v, mask, bias)
    torch.cuda.synchronize()
    _kernel_status_ok()
    ref = oracle.attention_forward(q, k.nan_to_num(), v.nan_to_num(), mask, bias, None, False)[0]
    check("out", out, ref, dtype)


@pytest.mark.parametrize("Sk,with_mask", [(1, False), (31, True), (5000, False), (40000, True)])
def test_bool_mask_and_no_mask(dev, Sk, with_mask):
    from flash_sparse_attn import flash_sparse_attn_func

    B, H, Hk, d, dtype = 2, 8, 2, 64, torch.bfloat16
    q, k, v, bias, _ = (t.to(dev) for t in oracle.make_inputs(B, 1, Sk, H, Hk, d, (B, Hk, 1, Sk), seed=8, dtype=dtype))
    mask = None
    if with_mask:
        mask = torch.rand((B, H, 1, Sk), generator=torch.Generator().manual_seed(2)).to(dev) < 0.2
        mask[0, 1] = False  # a head that sees nothing: output 0
    with torch.no_grad():
        out = flash_sparse_attn_func(q, k, v, mask, bias)
    torch.cuda.synchronize()
    _kernel_status_ok()
    ref = oracle.attention_forward(q, k, v, mask, bias, None, False)[0]
    check("out", out, ref, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Sk,d,H,window", [(1000, 256, 8, 500), (30000, 256, 8, 4096), (3000, 192, 6, 128), (2000, 136, 2, 2000),
                                           (70000, 256, 2, 20000)])
def test_probabilities_stay_in_32_bits_above_head_dim_128(dev, Sk, d, H, window, dtype):
    """Above head dim 128 the result is as far from the exact one as rounding it to 16 bits makes it: fp32 sums of some
    hundred to ten thousand terms add a relative 1e-5, probabilities of 16 bits would add 15 % of the rounding."""
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.utils.mask import create_mask

    B, Hk = 4, 2
    q, k, v, bias, _ = (t.to(dev) for t in oracle.make_inputs(B, 1, Sk, H, Hk, d, (B, Hk, 1, Sk), seed=6, dtype=dtype))
    with torch.no_grad():
        mask = create_mask(bias, None, B, 1, Sk, window, torch.finfo(dtype).min)
        out = flash_sparse_attn_func(q, k, v, mask, bias)
    torch.cuda.synchronize()
    _kernel_status_ok()
    group = H // Hk
    k64, v64 = (t.double().repeat_interleave(group, 2).transpose(1, 2) for t in (k, v))
    s = q.double().transpose(1, 2) @ k64.transpose(-1, -2) * d ** -0.5 + bias.double().repeat_interleave(group, 1)
    s = s.masked_fill(~mask.repeat_interleave(group, 1), float("-inf"))
    exact = (torch.softmax(s, -1) @ v64).transpose(1, 2)
    err, rounding = ((x.double() - exact).norm().item() for x in (out, exact.to(dtype)))
    assert err <= 1.02 * rounding, (err / rounding)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,pad,shift", [(64, 2, 0), (64, 4, 4), (64, 0, 2), (128, 4, 0), (128, 12, 8), (128, 0, 4)])
@pytest.mark.parametrize("geom", [(1, 1, 4, 2), (3, 333, 8, 2), (2, 5000, 24, 2), (1, 70000, 2, 1)])
@pytest.mark.parametrize("with_mask", [False, True])
def test_rows_aligned_to_4_or_8_bytes(dev, geom, with_mask, d, pad, shift, dtype):
    """K / V rows `pad` elements apart and `shift` elements off their base stay on the decode kernels, with the
    probabilities in 32 bits, as the kernels for such rows have them: within 2 % of the rounding of the exact result."""
    from flash_sparse_attn import flash_sparse_attn_func
    from flash_sparse_attn.flash_sparse_attn_interface import set_kernel_path

    B, Sk, H, Hk = geom
    q, k, v, bias, _ = (t.to(dev) for t in oracle.make_inputs(B, 1, Sk, H, Hk, d, (B, Hk, 1, Sk), seed=6, dtype=dtype))
    mask = torch.rand((B, Hk, 1, Sk), generator=torch.Generator().manual_seed(2)).to(dev) < 0.5 if with_mask else None
    if with_mask:
        mask[..., 0] = True

    def odd(t):
        flat = torch.full((B * Sk * Hk * (d + pad) + shift,), float("nan"), device=dev, dtype=dtype)
        view = flat[shift:].view(B, Sk, Hk, d + pad)[..., :d]
        return view.copy_(t)

    set_kernel_path("decode")
    try:
        with torch.no_grad():
            out = flash_sparse_attn_func(q, odd(k), odd(v), mask, bias)
    finally:
        set_kernel_path("auto")
    torch.cuda.synchronize()
    _kernel_status_ok()
    k64, v64 = (t.double().repeat_interleave(H // Hk, 2).transpose(1, 2) for t in (k, v))
    s = q.double().transpose(1, 2) @ k64.transpose(-1, -2) * d ** -0.5 + bias.double().repeat_interleave(H // Hk, 1)
    if with_mask:
        s = s.masked_fill(~mask.repeat_interleave(H // Hk, 1), float("-inf"))
    exact = (torch.softmax(s, -1) @ v64).transpose(1, 2)
    err, rounding = ((x.double() - exact).norm().item() for x in (out, exact.to(dtype)))
    assert err <= 1.02 * rounding + 1e-6 * exact.norm().item(), (err / rounding)
