"""Gradients of row-broadcast masks and biases (head dims up to 128) against 64 bits, over the routes the backward takes: the two-pass
kernel, the single pass for few queries over many keys, gathered keys with positions, packed sequences.

Bound: 1.01 times the error of the same formulas in 64 bits with the roundings the data type asks for and no others: O (as the forward
pass returned it, through D = rowsum(dO o O)), P and dS before they enter a product, and the result. Rounding is the same in both but
where 32-bit sums fall on the other side of a boundary, which moves the error by far less than the hundredth."""
import pytest
import torch

from flash_sparse_attn import flash_sparse_attn_func, flash_sparse_attn_varlen_func
from flash_sparse_attn import flash_sparse_attn_interface as iface
from oracle import oracle

pytestmark = pytest.mark.gpu


def _gradients(q, k, v, dout, out, mask, bias, causal, dtype):
    """dq, dk, dv, dbias of (Sq, H, d) queries over (Sk, Hk, d) keys in 64 bits; `dtype`: with the roundings to it, D from `out`.
    mask, bias: (heads, Sk) or None; dbias: per query head."""
    rnd = (lambda t: t.to(dtype).double()) if dtype else (lambda t: t)
    H, Hk, d, Sq, Sk = q.shape[1], k.shape[1], q.shape[2], q.shape[0], k.shape[0]
    dq, dk, dv = (torch.zeros(t.shape, dtype=torch.float64, device=q.device) for t in (q, k, v))
    dbias = torch.zeros(H, Sk, dtype=torch.float64, device=q.device)
    seen = torch.ones(Sq, Sk, dtype=torch.bool, device=q.device).tril(Sk - Sq) if causal else None
    for h in range(H):
        Q, K, V, G = q[:, h].double(), k[:, h * Hk // H].double(), v[:, h * Hk // H].double(), dout[:, h].double()
        s = Q @ K.T * d ** -0.5
        if bias is not None:
            s += bias[h * bias.shape[0] // H].double()
        if causal:
            s = s.masked_fill(~seen, float("-inf"))
        if mask is not None:
            s = s.masked_fill(~mask[h * mask.shape[0] // H], float("-inf"))
        p = torch.softmax(s, -1).nan_to_num(0.0)  # (rows that see no key)
        dp = G @ V.T
        D = (G * (out[:, h].double() if dtype else p @ V)).sum(-1, keepdim=True)
        ds = p * (dp - D)
        dq[:, h] = rnd(ds) @ K * d ** -0.5
        dk[:, h * Hk // H] += rnd(ds).T @ Q * d ** -0.5
        dv[:, h * Hk // H] += rnd(p).T @ G
        dbias[h] = ds.sum(0)
    return dq, dk, dv, dbias


def _check(got, exact, rounded, dtype, what):
    err, model = (got.double() - exact).norm().item(), (rounded.to(dtype).double() - exact).norm().item()
    assert err <= 1.01 * model, (what, err / model, model / exact.norm().item())


def _run(B, Sq, Sk, H, Hk, d, hm, hb, bb, causal, route, deterministic, dtype, keep=0.4, edit_mask=None):
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk)
    r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=dtype)  # noqa: E731
    q, k, v, dout = r(B, Sq, H, d), r(B, Sk, Hk, d), r(B, Sk, Hk, d), r(B, Sq, H, d)
    mask = bias = None
    if hm:
        mask = torch.rand((B, hm, 1, Sk), generator=g, device="cuda") < keep
        mask[..., Sk // 3: Sk // 3 + 150] = False  # whole 64-key tiles
        if edit_mask:
            edit_mask(mask)
    if hb:
        bias = r(bb, hb, 1, Sk).requires_grad_()
    for t in (q, k, v):
        t.requires_grad_()
    learned = [q, k, v] + ([bias] if hb else [])
    iface.set_compaction(route)
    try:
        out = flash_sparse_attn_func(q, k, v, attn_mask=mask, attn_bias=bias, is_causal=causal, deterministic=deterministic)
        runs = [torch.autograd.grad(out, learned, dout, retain_graph=True) for _ in range(2)]
    finally:
        iface.set_compaction("auto")
    with torch.no_grad():
        sides = []
        for rounding in (None, dtype):
            per = [_gradients(q[b], k[b], v[b], dout[b], out[b], None if mask is None else mask[b, :, 0],
                              None if bias is None else bias[b % bb, :, 0], causal, rounding) for b in range(B)]
            sides.append([torch.stack(x) for x in zip(*per)])
        if hb:
            for side in sides:
                side[3] = side[3].view(B, hb, H // hb, 1, Sk).sum(2)
                if bb == 1:
                    side[3] = side[3].sum(0, keepdim=True)
        for name, got, exact, rounded in zip(("dq", "dk", "dv", "dbias"), runs[0], *sides):
            _check(got, exact, rounded, dtype, name)
    fixed = 3 + (hb == Hk and bb == B)  # (dBias summed over heads or the batch by atomics: in no fixed order)
    if deterministic:
        assert all(torch.equal(a, b) for a, b in zip(runs[0][:fixed], runs[1][:fixed]))


def _packed(lq, lk, H, Hk, d, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(sum(lk))
    r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=dtype)  # noqa: E731
    q, k, v, dout = r(sum(lq), H, d), r(sum(lk), Hk, d), r(sum(lk), Hk, d), r(sum(lq), H, d)
    cq, ck = (torch.tensor([0] + x, device="cuda").cumsum(0).to(torch.int32) for x in (lq, lk))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = flash_sparse_attn_varlen_func(*leaves, cq, ck, max(lq), max(lk), is_causal=causal)
    grads = torch.autograd.grad(out, leaves, dout)
    with torch.no_grad():
        sides = []
        for rounding in (None, dtype):
            per = []
            for i in range(len(lq)):
                rows, keys = slice(cq[i], cq[i + 1]), slice(ck[i], ck[i + 1])
                per.append(_gradients(q[rows], k[keys], v[keys], dout[rows], out[rows], None, None, causal, rounding)[:3])
            sides.append([torch.cat(x) for x in zip(*per)])
        for name, got, exact, rounded in zip(("dq", "dk", "dv"), grads, *sides):
            _check(got, exact, rounded, dtype, name)


# (batch, queries, keys, heads, kv heads, head dim, mask heads, bias heads, bias batch, causal, route, deterministic)
FEW_QUERIES = [
    (1, 128, 8192, 8, 2, 128, 0, 0, 1, False, "off", False),
    (2, 65, 3000, 6, 2, 96, 2, 2, 2, True, "off", False),
    (1, 200, 5000, 4, 4, 128, 4, 4, 1, False, "off", False),
    (2, 100, 4200, 4, 1, 72, 0, 1, 1, False, "off", False),     # dBias summed over the batch
    (1, 300, 6000, 12, 4, 128, 4, 4, 1, True, "off", False),
    (1, 129, 2050, 8, 2, 128, 8, 8, 1, True, "off", False),     # mask and bias per query head
    (1, 128, 16384, 8, 2, 128, 2, 2, 1, True, "auto", False),   # gathered keys and their positions
    (1, 70, 9000, 4, 2, 64, 2, 2, 1, True, "auto", True),
    (1, 128, 4096, 4, 2, 64, 0, 0, 1, True, "off", True),
    (1, 128, 8192, 8, 2, 64, 2, 2, 1, False, "off", True),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", FEW_QUERIES, ids=lambda c: "x".join(map(str, c)))
def test_few_queries(case, dtype):
    _run(*case, dtype)


@pytest.mark.parametrize("B,Sk,H,Hk,d", [(1, 4101, 4, 1, 64), (2, 9001, 8, 2, 128)])
def test_single_query(B, Sk, H, Hk, d):
    """Against the oracle, with its tolerances (the few numbers of one row say little about the error of rounding)."""
    q, k, v, bias, dout = oracle.make_inputs(B, 1, Sk, H, Hk, d, (B, Hk, 1, Sk), seed=Sk, dtype=torch.bfloat16, device="cpu")
    mask = torch.rand(B, Hk, 1, Sk, generator=torch.Generator().manual_seed(1)) < 0.4
    want = oracle.attention_forward_backward(q, k, v, mask, bias, dout, None, False)
    iface.set_compaction("off")
    try:
        leaves = [t.cuda().requires_grad_() for t in (q, k, v, bias)]
        out = flash_sparse_attn_func(*leaves[:3], attn_mask=mask.cuda(), attn_bias=leaves[3])
        grads = torch.autograd.grad(out, leaves, dout.cuda())
    finally:
        iface.set_compaction("auto")
    for name, got, ref in zip(("dq", "dk", "dv", "dbias"), grads, want[2:]):
        ok, msg = oracle.within_tolerance(oracle.error_report(name, got.cpu(), ref), name != "dq")
        assert ok, msg


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lq,lk,H,Hk,d", [([64, 70], [4100, 3000], 4, 2, 128), ([60, 3, 100], [70, 5000, 3000], 4, 4, 64),
                                          ([129, 1, 200, 31], [129, 900, 4000, 128], 8, 2, 96)])
def test_packed_few_queries(lq, lk, H, Hk, d, causal, dtype):
    """Packed sequences of few queries over many keys: key tiles and query tiles that hold rows of several sequences."""
    _packed(lq, lk, H, Hk, d, causal, dtype)


def test_packed_few_queries_isolated():
    """Fixed-point sums twice the same; a NaN in one sequence stays there; rows outside every sequence are zero."""
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    q, k, v, dout = r(200, 4, 128), r(6000, 2, 128), r(6000, 2, 128), r(200, 4, 128)
    cq, ck = (torch.tensor(x, device="cuda", dtype=torch.int32) for x in ([0, 70, 190], [0, 2500, 5900]))
    grads = []
    for nan in (False, False, True):
        if nan:
            q[10, 1], k[20, 0], v[2499, 1] = float("nan"), float("nan"), float("inf")
        leaves = [t.clone().requires_grad_() for t in (q, k, v)]
        out = flash_sparse_attn_varlen_func(*leaves, cq, ck, 120, 3400, is_causal=True, deterministic=True)
        grads.append(torch.autograd.grad(out, leaves, dout))
    for a, b, c, rows, end in zip(*grads, (70, 2500, 2500), (190, 5900, 5900)):
        assert torch.equal(a, b)
        assert torch.equal(a[rows:end], c[rows:end]) and not c[:rows].isfinite().all()
        assert not a[end:].any() and not c[end:].any()


def test_packed_few_queries_time():
    """2 x 64 queries over 2 x 16384 keys take no more than three times as long as the same number of scores in 2 x 1024 rows."""
    def run(lq, lk):
        q, k, v, dout = (torch.randn(2 * n, h, 128, device="cuda", dtype=torch.bfloat16) for n, h in ((lq, 8), (lk, 2), (lk, 2), (lq, 8)))
        leaves = [t.requires_grad_() for t in (q, k, v)]
        cq, ck = (torch.tensor([0, n, 2 * n], device="cuda", dtype=torch.int32) for n in (lq, lk))
        return _backward_time(flash_sparse_attn_varlen_func(*leaves, cq, ck, lq, lk), leaves, dout)

    few, many = run(64, 16384), run(1024, 1024)
    assert few <= 3 * many, (few, many)


def _time(leaves, dout, **kwargs):
    return _backward_time(flash_sparse_attn_func(*leaves, **kwargs), leaves, dout)


def _backward_time(out, leaves, dout):
    """Device time of five backward passes, the best of three."""
    torch.autograd.grad(out, leaves, dout, retain_graph=True)
    best = float("inf")
    for _ in range(3):
        start, stop = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(10_000_000)  # the launches queue up behind it
        start.record()
        for _ in range(5):
            torch.autograd.grad(out, leaves, dout, retain_graph=True)
        stop.record()
        stop.synchronize()
        best = min(best, start.elapsed_time(stop))
    return best


def _normal(Sq, Sk, H, Hk, d):
    q, k, v, dout = (torch.randn(1, n, h, d, device="cuda", dtype=torch.bfloat16) for n, h in ((Sq, H), (Sk, Hk), (Sk, Hk), (Sq, H)))
    return [t.requires_grad_() for t in (q, k, v)], dout


def _some_heads_empty(mask):
    mask[:, 1] = False  # between heads that have kept keys
    mask[0, 4:7] = False


# Two-pass kernel, several query heads per CTA of the row pass (from 12 row tiles x heads per SM on): Q and dO of the next head come in
# while the last one's dQ is stored, activity bits alternate between two tables, sums start again; odd and even numbers of key tiles
MANY_HEADS = [
    (8, 1024, 320, 32, 8, 128, 0, 0, 1, False, "off", False),
    (8, 1000, 1100, 32, 4, 64, 32, 32, 8, True, "off", True),   # mask and bias per head, some heads without a kept key
    (4, 2048, 128, 32, 32, 128, 1, 0, 1, False, "off", False),
]
# ... and more keys than the 2048 that dQ was once summed over: positions, ragged ends, fixed order
MANY_KEYS = [
    (1, 2100, 8256, 2, 1, 64, 1, 1, 1, True, "off", True),
    (1, 5000, 6000, 4, 2, 128, 2, 2, 1, True, "auto", False),
    (1, 1400, 5000, 8, 4, 128, 4, 4, 1, False, "auto", True),
]


# dBias per query head of a group (in shared memory up to 16 heads, beyond in memory), summed over the batch, over the heads
DBIAS = [
    (2, 300, 400, 16, 1, 128, 0, 16, 1, True, "off", False),
    (1, 300, 400, 17, 1, 64, 17, 17, 1, False, "off", False),
    (2, 500, 900, 4, 2, 64, 2, 4, 2, True, "auto", False),
    (3, 300, 400, 6, 2, 128, 0, 2, 1, False, "off", False),
    (3, 300, 400, 6, 2, 96, 2, 1, 3, True, "off", False),
    (2, 300, 400, 4, 4, 128, 1, 1, 1, False, "off", False),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("case", MANY_HEADS + MANY_KEYS + DBIAS, ids=lambda c: "x".join(map(str, c)))
def test_two_passes(case, dtype):
    _run(*case, dtype, keep=0.6, edit_mask=_some_heads_empty if case[6] > 8 else None)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_long(causal, dtype):
    _packed([2500, 300, 2177], [2500, 333, 4200], 4, 2, 128, causal, dtype)


def test_few_queries_time():
    """128 queries over 65536 keys take no more than three times as long as the same number of scores in 2048 rows: their dQ is not
    left to the eight chains of 1024 key tiles that eight heads have."""
    few, many = (_time(*_normal(Sq, Sk, 8, 2, 128)) for Sq, Sk in ((128, 65536), (2048, 4096)))
    assert few <= 3 * many, (few, many)


def test_long_masks():
    """Masks of more than 4096 tiles of 64 keys: gradients, and tiles without a kept key are skipped (11 kept keys of 300000 take no more
    than 0.4 of the time of half the keys)."""
    _run(1, 130, 262209, 2, 1, 64, 1, 1, 1, False, "off", False, torch.float16, keep=0.01)
    leaves, dout = _normal(1024, 300000, 8, 2, 64)
    dense = torch.rand((1, 2, 1, 300000), device="cuda") < 0.5
    sparse = torch.zeros_like(dense)
    sparse[..., ::30000] = True
    iface.set_compaction("off")
    try:
        times = [_time(leaves, dout, attn_mask=m) for m in (sparse, dense)]
    finally:
        iface.set_compaction("auto")
    assert times[0] <= 0.4 * times[1], times


def test_dbias_per_head_time():
    """A bias per query head adds its sums to memory once per CTA, not in every step: no more than 1.12 of the time with one per kv head."""
    times = []
    for heads in (16, 4):
        g = torch.Generator(device="cuda").manual_seed(heads)
        r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.bfloat16)  # noqa: E731
        leaves = [t.requires_grad_() for t in (r(4, 2048, 16, 128), r(4, 2048, 4, 128), r(4, 2048, 4, 128), r(4, heads, 1, 2048))]
        dout = r(4, 2048, 16, 128)
        out = flash_sparse_attn_func(*leaves[:3], attn_bias=leaves[3])
        times.append(_backward_time(out, leaves, dout))
    assert times[0] <= 1.12 * times[1], times
