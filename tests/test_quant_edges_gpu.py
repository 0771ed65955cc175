"""FP8 block quantiser: blocks that hold NaN, infinities, both, or nothing else, byte for byte."""
import pytest
import torch

from oracle import gdpa_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim", [64, 128])
def test_blocks_with_nan_and_infinity(head_dim):
    """One sequence of six blocks, the last of one row; a NaN (either sign, the smallest payload and the largest) does not count
    for its block's scale and becomes -448, as does everything of a block whose scale is infinite and that is not finite."""
    import ads_model_kernel_library_b200.gdpa as G

    off = torch.tensor([0, 641])
    g = torch.Generator().manual_seed(head_dim)
    x = torch.randn(641, 3, head_dim, generator=g).to(torch.bfloat16)
    bits = x.view(torch.int16)
    bits[3, 0, 0], bits[127, 0, head_dim - 1] = 0x7F81, -1  # block 0, head 0: two NaN among finite values
    bits[130, 1, 5], x[200, 1, 9] = 0x7FFF, float("inf")  # block 1, head 1: NaN and infinity
    bits[256:384, 2] = 0x7FC0  # block 2, head 2: NaN only
    x[400, 0, 1] = -float("inf")  # block 3, head 0
    bits[640, 1, 0] = 0x7FC0  # block 5, a single row
    x[640, 2] = 0
    x8, scales, blocks = G.quantize_fp8_blockwise(x.cuda(), off.cuda())
    # a NaN as 0 gives the scale without it
    r8, rscales, rblocks = orc.quantize_fp8_blockwise(x.nan_to_num(0, float("inf"), -float("inf")), off)
    want = torch.where(x.isfinite(), r8.view(torch.uint8), torch.tensor(0xFE, dtype=torch.uint8))  # 0xFE: -448
    assert torch.equal(blocks.cpu(), rblocks) and torch.equal(scales.cpu()[:6], rscales)
    assert torch.equal(x8.cpu().view(torch.uint8), want)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("lengths", [[300, 129], [1, 40]])
@pytest.mark.parametrize("head_dim", [32, 64, 128])
def test_a_negative_zero_keeps_its_sign(head_dim, lengths, fp32):
    """Of both kernels, in blocks of finite values, blocks with an infinity and blocks of zeros only: -0, and what is so small
    that it is rounded to it."""
    import ads_model_kernel_library_b200.gdpa as G

    off = torch.tensor([0, *torch.tensor(lengths).cumsum(0)])
    x = torch.randn(int(off[-1]), 3, head_dim, generator=torch.Generator().manual_seed(7))
    x = x.to(torch.float32 if fp32 else torch.bfloat16)
    x[:, 0, ::3] = -0.0
    x[:, 0, 1::5] = 0.0
    x[:, 1] = -0.0
    x[:, 1, ::2] = 0.0
    x[:, 0, 2::7] = -1e-30
    x[-1, 2, :5] = torch.tensor([-float("inf"), -0.0, 0.0, -1.0, 1.0])
    x8, scales, _ = G.quantize_fp8_blockwise(x.cuda(), off.cuda())
    r8, rscales, _ = orc.quantize_fp8_blockwise(x.nan_to_num(0, float("inf"), -float("inf")), off)
    want = torch.where(x.isfinite(), r8.view(torch.uint8), torch.tensor(0xFE, dtype=torch.uint8))
    assert torch.equal(scales.cpu()[: rscales.shape[0]], rscales)
    assert torch.equal(x8.cpu().view(torch.uint8), want)


@pytest.mark.parametrize("offset_dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("rows", [-1, 0, 1])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_both_sides_of_the_rule_by_average_length(head_dim, rows, offset_dtype):
    """One row less than the one-pass kernel takes (8192 values a sequence and head on average), as many, and one more."""
    import ads_model_kernel_library_b200.gdpa as G

    lens = [1, 0, 127, 128, 129, 40, 3, 128, 20]
    lens += [8192 // head_dim * (len(lens) + 1) + rows - sum(lens)]
    assert lens[-1] > 0
    off = torch.tensor([0, *torch.tensor(lens).cumsum(0)], dtype=offset_dtype)
    x = torch.randn(sum(lens), 3, head_dim, generator=torch.Generator().manual_seed(head_dim)).to(torch.bfloat16)
    x8, scales, blocks = G.quantize_fp8_blockwise(x.cuda(), off.cuda())
    r8, rscales, rblocks = orc.quantize_fp8_blockwise(x, off)
    assert torch.equal(blocks.cpu(), rblocks) and torch.equal(scales.cpu()[: rscales.shape[0]], rscales)
    assert torch.equal(x8.cpu().view(torch.uint8), r8.view(torch.uint8))
