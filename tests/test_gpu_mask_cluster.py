"""Selection with positions where a row is split over the CTAs of a cluster: lengths around the segments' and chunks'
edges, odd and unaligned rows, ties across segments, pre-masks. Selection is exact: bits and positions are compared with
the CPU oracle's mask."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sk,window,levels,padded", [
    (1, 1, 5, 2, 0, False), (1, 1, 2048, 2048, 0, False), (1, 3, 2049, 700, 0, False), (2, 2, 4097, 1024, 3, True),
    (1, 1, 16384, 1, 0, False), (1, 8, 16391, 5000, 2, False), (1, 1, 65536, 2048, 0, True), (1, 2, 65537, 4096, 5, False),
    (40, 8, 8193, 512, 0, True), (700, 1, 2500, 300, 4, False), (1, 1, 262144, 3000, 0, False), (1, 1, 262145, 3000, 1, False),
])
def test_rows_split_over_ctas(B, H, Sk, window, levels, padded, dtype):
    from flash_sparse_attn.utils.mask import create_mask

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(Sk + window)
    bias = torch.randn((B, H, 1, Sk), generator=g)
    if levels:  # few distinct values: ties at the threshold in every segment
        # (+ 0.0: no negative zeros -- the radix select orders them below the positive ones, the oracle's sort does not)
        bias = (bias * levels / 2).round().clamp(-levels, levels) + 0.0
    bias = bias.to(dtype)
    min_dtype = torch.finfo(dtype).min
    bias[..., ::97] = min_dtype  # never selected
    bias[..., 3] = float("inf")
    bias[..., 4 % Sk] = float("-inf")
    padding = None
    if padded:
        first = (torch.arange(B) * (Sk - 1) // max(B, 1)).clamp(max=Sk - 1)
        padding = torch.arange(Sk)[None, :] >= first[:, None]
    want = oracle.create_mask(bias, padding, B, 1, Sk, window, min_dtype)
    got = create_mask(bias.to(dev), None if padding is None else padding.to(dev), B, 1, Sk, window, min_dtype)
    assert torch.equal(got.cpu(), want)
    kept = got._fdma_kept[0]
    pos, rows = kept.key_pos.cpu(), want.reshape(B, H, Sk)
    for b in range(0, B, max(1, B // 8)):
        for h in range(H):
            sel = rows[b, h].nonzero().flatten()
            assert int(kept.count[b, h]) == sel.numel()
            assert torch.equal(pos[b, h, : sel.numel()].long(), sel)
            assert (pos[b, h, sel.numel():] == 2147483647).all()
