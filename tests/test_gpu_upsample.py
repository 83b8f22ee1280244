"""GPU tests of the convex field upsampling kernel (MatchStereo.upsample_field, models/match_stereo.py:73-84)
through the C ABI: against the reference's own outputs (golden files) and against the oracle."""
import pytest
import torch

from _cases import assert_close_sum_of_products, golden_upsample_names, load_golden_upsample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", golden_upsample_names())
def test_kernel_matches_reference_vectors(name):
    import matchattention_b200 as ma
    c = load_golden_upsample(name)
    out = ma.upsample_field(c["field"].cuda(), c["mask"].cuda(), c["factor"]).cpu()
    scale = float(c["field"].float().abs().max()) * c["factor"]
    assert_close_sum_of_products(out, c["out"], c["dtype"], scale, name)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(2, 48, 48, 2, 2), (1, 37, 131, 2, 4), (2, 96, 96, 2, 2), (1, 9, 300, 3, 8), (1, 5, 4, 8, 1)])
def test_kernel_matches_oracle(shape, dtype):
    import matchattention_b200 as ma
    import oracle
    B, H, W, D, f = shape
    g = torch.Generator().manual_seed(H * W + f)
    field = (torch.randn(B, H, W, D, generator=g) * 4).to(dtype)
    mask = (torch.randn(B, 9 * f * f, H, W, generator=g) * 2).to(dtype)
    ref = oracle.upsample_field(field, mask, f)
    out = ma.upsample_field(field.cuda(), mask.cuda(), f).cpu()
    assert_close_sum_of_products(out, ref, dtype, float(field.float().abs().max()) * f)
    if dtype != torch.float32:
        same = (out.view(torch.int16) == ref.view(torch.int16)).float().mean().item()
        assert same > 0.99, f"only {same:.3%} bit-identical to the oracle"


def test_constant_field_is_reproduced():
    """The weights are a convex combination: away from the zero-padded border a constant field comes
    back as factor * constant whatever the mask says."""
    import matchattention_b200 as ma
    B, H, W, D, f = 1, 12, 14, 2, 4
    field = torch.full((B, H, W, D), 1.5, device="cuda")
    mask = torch.randn(B, 9 * f * f, H, W, device="cuda")
    out = ma.upsample_field(field, mask, f)
    inner = out[:, f:-f, f:-f]
    assert torch.allclose(inner, torch.full_like(inner, 1.5 * f), atol=1e-5)


def test_bad_arguments_raise():
    import matchattention_b200 as ma
    field = torch.zeros(1, 4, 4, 2, device="cuda")
    with pytest.raises(ValueError):
        ma.upsample_field(field, torch.zeros(1, 36, 4, 5, device="cuda"), 2)
    with pytest.raises(RuntimeError):
        ma.upsample_field(field, torch.zeros(1, 81, 4, 4, device="cuda"), 3)        # factor 3 is not built
    with pytest.raises(RuntimeError):
        ma.upsample_field(field.cpu(), torch.zeros(1, 36, 4, 4), 2)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("factor", [2, 4])
@pytest.mark.parametrize("H,W", [(1, 1), (2, 2), (3, 31), (2, 33), (1, 63), (3, 64), (2, 65), (5, 98), (2, 129),
                                 (900, 1), (901, 2), (900, 33), (903, 64), (460, 65), (301, 130)])
def test_pairs_of_cells_at_the_edges_of_a_warp(H, W, factor, dtype):
    """Widths around the 32 and 64 cells of a warp, odd and even, down to a map of one cell; the high maps fill the chip and
    take two fine rows per thread."""
    import matchattention_b200 as ma
    import oracle
    g = torch.Generator().manual_seed(H * W + factor)
    field = (torch.randn(2, H, W, 2, generator=g) * 4).to(dtype)
    mask = (torch.randn(2, 9 * factor * factor, H, W, generator=g) * 2).to(dtype)
    out = ma.upsample_field(field.cuda(), mask.cuda(), factor).cpu()
    assert_close_sum_of_products(out, oracle.upsample_field(field, mask, factor), dtype, float(field.float().abs().max()) * factor)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("factor,W", [(2, 8), (4, 8), (4, 6), (2, 7)])
def test_logits_at_the_ends_of_the_type(factor, W, dtype):
    """Logits at the type's lowest and largest value (a caller's mask) are ordinary numbers to a softmax: nine equal
    ones weigh 1/9 each, one that stands out takes all."""
    import matchattention_b200 as ma
    H, low, top = 3, torch.finfo(dtype).min, torch.finfo(dtype).max
    field = torch.ones(1, H, W, 2, dtype=dtype)
    for fill, pick in ((low, None), (top, None), (low, top), (low, 0.0)):
        mask = torch.full((1, 9, factor * factor, H, W), fill, dtype=dtype)
        if pick is not None:
            mask[:, 4] = pick                        # the cell itself
        out = ma.upsample_field(field.cuda(), mask.view(1, -1, H, W).cuda(), factor).float().cpu()
        if pick is None:                             # cells inside the map's border see nine ones
            out = out[:, factor:-factor, factor:-factor]
        # nine weights and nine products, each rounded to the type, then the sum
        assert (out - factor).abs().max() <= 4 * torch.finfo(dtype).eps * factor


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,factor,W", [(2, 2, 64), (2, 4, 36), (2, 4, 62), (2, 2, 33), (3, 4, 32)])
def test_the_address_does_not_change_the_bits(D, factor, W, dtype):
    """The same mask one, two, four or eight elements into a buffer reaches other kernels and loads; the result is the same."""
    import matchattention_b200 as ma
    g = torch.Generator().manual_seed(W)
    field = (torch.randn(2, 5, W, D, generator=g) * 4).to(dtype).cuda()
    mask = (torch.randn(2, 9 * factor * factor, 5, W, generator=g) * 3).to(dtype).cuda()
    want = ma.upsample_field(field, mask, factor)
    for shift in (1, 2, 4, 8):
        moved = torch.empty(mask.numel() + shift, dtype=dtype, device="cuda")[shift:].view(mask.shape).copy_(mask)
        assert torch.equal(ma.upsample_field(field, moved, factor), want), shift


@pytest.mark.parametrize("factor", [2, 4])
@pytest.mark.parametrize("H,W", [(1, 2), (2, 4), (1, 62), (3, 64), (2, 66), (5, 98), (2, 130)])
def test_float32_pairs_at_the_edges_of_a_warp(H, W, factor):
    """Even widths around the 64 cells of a warp, down to a map of two cells."""
    import matchattention_b200 as ma
    import oracle
    g = torch.Generator().manual_seed(H * W + factor)
    field = torch.randn(2, H, W, 2, generator=g) * 4
    mask = torch.randn(2, 9 * factor * factor, H, W, generator=g) * 2
    out = ma.upsample_field(field.cuda(), mask.cuda(), factor).cpu()
    assert_close_sum_of_products(out, oracle.upsample_field(field, mask, factor), torch.float32, float(field.abs().max()) * factor)
