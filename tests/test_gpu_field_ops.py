"""GPU tests of the consistency-mask and local-disparity kernels through the library: against the C
oracle on the golden inputs and on larger seeded inputs, and -- where the reference's Python code is
present -- against the reference's own functions run on the same GPU (the strictest check: same
PyTorch build, same arithmetic)."""
import pytest
import torch

from _cases import golden_names_with_prefix, load_golden_arrays, ulp16

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.float16, torch.bfloat16]


def _ma():
    import matchattention_b200
    return matchattention_b200


def _close16(got, ref, dt, ulps=1.0):
    g, r = got.float().cpu(), ref.float().cpu()
    if dt == torch.float32:
        return bool(((g - r).abs() <= 1e-4 * r.abs().clamp_min(1.0)).all())
    return bool(((g - r).abs() <= ulps * ulp16(r, dt)).all())


@pytest.mark.parametrize("name", golden_names_with_prefix("consistency_"))
def test_consistency_mask_kernel_matches_oracle(name):
    import oracle
    c = load_golden_arrays(name)
    want_mask, want_diff = oracle.consistency_mask(c["field"], c["threshold"])
    mask, diff = _ma().consistency_mask(c["field"].cuda(), c["threshold"], return_diff=True)
    torch.cuda.synchronize()
    assert _close16(diff, want_diff, c["dtype"]), name
    decided = (want_diff.float() - c["threshold"]).abs() > 2 * ulp16(want_diff.float(), torch.float16)
    assert torch.equal(mask.cpu()[decided], want_mask[decided])


@pytest.mark.parametrize("dtype", DTYPES)
def test_consistency_mask_kernel_on_a_large_field(dtype):
    import oracle
    g = torch.Generator().manual_seed(5)
    field = (torch.randn(2, 96, 128, 2, generator=g) * 3).to(dtype)
    want_mask, want_diff = oracle.consistency_mask(field)
    mask, diff = _ma().consistency_mask(field.cuda(), return_diff=True)
    assert _close16(diff, want_diff, dtype)
    decided = (want_diff.float() - 2).abs() > 2 * ulp16(want_diff.float(), torch.float16)
    assert torch.equal(mask.cpu()[decided], want_mask[decided])
    assert torch.equal(_ma().consistency_mask(field.cuda()), mask)


@pytest.mark.parametrize("name", golden_names_with_prefix("disparity_"))
def test_local_disparity_kernel_matches_oracle(name):
    import oracle
    c = load_golden_arrays(name)
    dt = c["dtype"]
    want_flow, want_blur, want_centre = oracle.local_disparity(c["volume"])
    flow, blur, centre = _ma().local_disparity_estimator(c["volume"].cuda(), return_debug=True)
    torch.cuda.synchronize()
    assert _close16(blur, want_blur, dt)
    clear = c["gap"] > (1e-6 if dt == torch.float32 else 0.0)
    assert torch.equal(centre.cpu()[clear], want_centre[clear])
    assert _close16(flow.cpu()[clear], want_flow[clear], dt)
    assert (flow[..., 1] == 0).all()


def _reference():
    from oracle import ref_loader
    if not ref_loader.available():
        pytest.skip("the reference's Python code is not present (oracle/make_ref.py places it under oracle/_ref/)")
    return ref_loader.import_reference()


@pytest.mark.parametrize("dtype", DTYPES)
def test_consistency_mask_kernel_matches_reference_on_the_gpu(dtype):
    _, blocks = _reference()
    g = torch.Generator().manual_seed(6)
    field = (torch.randn(2, 96, 128, 2, generator=g) * 3).to(dtype).cuda()
    want = blocks.MatchAttentionLayer.consistency_mask(None, field)
    mask, diff = _ma().consistency_mask(field, return_diff=True)
    decided = (diff.float() - 2).abs() > 2 * ulp16(diff.float().cpu(), torch.float16).cuda()
    assert decided.float().mean() > 0.95
    assert torch.equal(mask[decided], want[decided])
    mismatch = (mask != want).float().mean().item()
    assert mismatch < 2e-3, f"{mismatch:.2e} of the mask differs from the reference"


@pytest.mark.parametrize("dtype", DTYPES)
def test_local_disparity_kernel_matches_reference_on_the_gpu(dtype):
    _reference()
    from models.cost_volume import local_disparity_estimator
    import torch.nn.functional as F
    g = torch.Generator().manual_seed(7)
    B, D, H, W = 2, 48, 48, 48
    vol = torch.softmax(torch.randn(B, D, H, W, generator=g) * 2.0, dim=1).to(dtype).cuda()
    want = local_disparity_estimator(vol.clone())
    flow = _ma().local_disparity_estimator(vol)
    blur = F.avg_pool1d(vol.permute(0, 2, 3, 1).reshape(B, -1, D), kernel_size=5, stride=1, padding=2).float()
    top2 = blur.topk(2, dim=-1).values
    clear = ((top2[..., 0] - top2[..., 1]) > (1e-6 if dtype == torch.float32 else 0.0)).view(B, H, W)
    assert clear.float().mean() > 0.5
    assert _close16(flow[..., 0][clear], want[..., 0][clear], dtype)
    assert (flow[..., 1] == 0).all()


@pytest.mark.parametrize("name", golden_names_with_prefix("flowinit_"))
def test_flow_init_kernels_match_oracle(name):
    import oracle
    c = load_golden_arrays(name)
    dt, H, W = c["dtype"], c["H"], c["W"]
    want_flow, want_prob, want_blur, want_centre = oracle.flow_init(c["correlation"], H, W)
    flow, prob, blur, centre = _ma().flow_init(c["correlation"].cuda(), H, W, return_debug=True)
    torch.cuda.synchronize()
    assert _close16(prob, want_prob, dt) and _close16(blur, want_blur, dt)
    clear = c["gap"] > (1e-6 if dt == torch.float32 else 0.0)
    assert torch.equal(centre.cpu()[clear], want_centre[clear])
    assert _close16(flow.cpu().view(-1, H * W, 2)[clear], want_flow.view(-1, H * W, 2)[clear], dt, ulps=2.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,W", [(12, 16), (9, 37)])
def test_flow_init_kernels_match_reference_on_the_gpu(dtype, H, W):
    """The reference's GlobalCorrelation.forward(stereo=False) on the same GPU against the kernels, fed with
    the correlation the module itself computes."""
    _reference()
    from models.cost_volume import GlobalCorrelation
    import torch.nn.functional as F
    torch.manual_seed(11)
    B, C = 1, 32
    mod = GlobalCorrelation(C).eval().cuda().to(dtype)
    x = (torch.randn(2 * B, H, W, C) * 8).cuda().to(dtype)
    with torch.inference_mode():
        xn = mod.norm(x)
        ref, tgt = xn.chunk(2, dim=0)
        corr = torch.matmul(mod.q(ref).view(B, -1, C), mod.k(tgt).view(B, -1, C).transpose(-2, -1)) * mod.scale
        want_flow, want_prob = mod(x, stereo=False)
        blur = F.avg_pool2d(want_prob.view(2 * B, H * W, H * W), kernel_size=5, stride=1, padding=2).float()
    flow, prob = _ma().flow_init(corr, H, W)
    assert _close16(prob, want_prob, dtype)
    top2 = blur.topk(2, dim=-1).values
    clear = ((top2[..., 0] - top2[..., 1]) > (1e-6 if dtype == torch.float32 else 0.0)).view(2 * B, H, W)
    assert clear.float().mean() > 0.5
    assert _close16(flow[clear], want_flow[clear], dtype, ulps=2.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,W,sharpness", [(5, 5, 2.0), (8, 15, 2.0), (11, 11, 2.0), (8, 16, 2.0), (5, 51, 2.0), (16, 16, 300.0),
                                           (72, 72, 2.0)])
def test_flow_init_kernels_at_the_edges_of_their_tiles(H, W, sharpness, dtype):
    """Token counts around one chunk of 120 / 128 targets and one band of rows, rows of prob that are and are not
    16-byte aligned, the long bands of large maps, and scores spread so widely that no shared reference serves a tile."""
    import oracle
    g = torch.Generator().manual_seed(H * W)
    second = torch.randn(1, H * W, 16, generator=g)
    first = second.roll(3, 1) + 0.3 * torch.randn(1, H * W, 16, generator=g)
    corr = (torch.matmul(first, second.transpose(1, 2)) * sharpness / 4.0).to(dtype)
    want_flow, want_prob, want_blur, want_centre = oracle.flow_init(corr, H, W)
    flow, prob, blur, centre = _ma().flow_init(corr.cuda(), H, W, return_debug=True)
    steps = ((prob.float().cpu() - want_prob.float()).abs() - 2.0 ** -24).clamp_min(0)     # float16: below 2^-14 the spacing is 2^-24
    assert _close16(want_prob.float() + steps, want_prob, dtype) and _close16(blur, want_blur, dtype)
    same = centre.cpu() == want_centre
    assert same.float().mean() > 0.98           # the rest: equal box averages
    off = (flow.cpu().float().view(-1, H * W, 2)[same] - want_flow.float().view(-1, H * W, 2)[same]).abs().max().item()
    limit = 1e-3 if dtype == torch.float32 else 2.0 * float(ulp16(torch.tensor(float(max(H, W))), dtype))
    assert off <= limit         # the flow is a position on the map, rounded, minus the token's own


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D,H,W", [(5, 1, 31), (7, 3, 11), (40, 2, 33), (63, 5, 13), (159, 2, 17)])
def test_local_disparity_kernel_at_the_edges_of_its_shares(D, H, W, dtype):
    """Disparity counts that leave shares short or empty, and pixel counts around one warp."""
    import oracle
    g = torch.Generator().manual_seed(D)
    vol = torch.softmax(torch.randn(2, D, H, W, generator=g) * 2.0, dim=1).to(dtype)
    want_flow, want_blur, want_centre = oracle.local_disparity(vol)
    flow, blur, centre = _ma().local_disparity_estimator(vol.cuda(), return_debug=True)
    assert _close16(blur, want_blur, dtype)
    same = centre.cpu() == want_centre
    assert same.float().mean() > 0.98           # the rest: equal box averages
    assert _close16(flow.cpu()[same], want_flow[same], dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,W", [(5, 6), (10, 13), (6, 22), (12, 21), (71, 74), (68, 77)])
def test_flow_init_rows_aligned_to_two_and_four_elements(H, W, dtype):
    """Token counts that are multiples of 2 or 4 but not of 8, around a chunk, below and above 5000: the same bits as the
    any-alignment kernels, which an operand that starts one element off takes."""
    g = torch.Generator().manual_seed(H * W)
    corr = (torch.randn(2, H * W, H * W, generator=g) * 2.0).to(dtype).cuda()
    odd = torch.empty(corr.numel() + 1, dtype=dtype, device="cuda")[1:].view_as(corr).copy_(corr)
    for got, want in zip(_ma().flow_init(corr, H, W, return_debug=True), _ma().flow_init(odd, H, W, return_debug=True)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", DTYPES)
def test_local_disparity_of_an_infinite_value(dtype):
    """A window that holds an infinity has an infinite average: the first such window is the arg max, and its flow is
    infinity over infinity."""
    vol = torch.rand(2, 40, 3, 5).to(dtype)
    vol[:, 17, 1, 2] = float("inf")
    flow, blur, centre = _ma().local_disparity_estimator(vol.cuda(), return_debug=True)
    assert (blur[:, 1, 2] == float("inf")).all() and (centre[:, 1, 2] == 15).all() and flow[:, 1, 2, 0].isnan().all()
    assert torch.isfinite(flow).sum() == flow.numel() - 2


# Token counts on either side of the thresholds: column sums 32 columns wide from 5800 tokens on in 16 bits (rows aligned to 2,
# 4 and 8 elements), from 6600 on in float32 (5000 in rows aligned to single elements), 16-bit rows of an odd count from 9400 on;
# short bands at odd counts below 10000, long ones from 5000 (odd: 10000) on.
BEYOND_THRESHOLDS = [(71, 73, torch.float16), (84, 72, torch.float32), (98, 96, torch.float16), (97, 97, torch.bfloat16),
                     (76, 76, torch.bfloat16), (80, 73, torch.bfloat16), (78, 75, torch.float16), (78, 75, torch.bfloat16),
                     (77, 76, torch.float16), (77, 76, torch.bfloat16), (75, 77, torch.float16), (88, 76, torch.float32),
                     (83, 83, torch.float32), (70, 73, torch.float32), (69, 71, torch.float32), (101, 101, torch.float16)]


@pytest.mark.parametrize("H,W,dtype", BEYOND_THRESHOLDS)
def test_flow_init_kernels_beyond_their_thresholds(H, W, dtype):
    """Short and long bands, narrow and wide column sums of every alignment, remainders of their batches of rows."""
    import oracle
    g = torch.Generator().manual_seed(H * W)
    second = torch.randn(1, H * W, 16, generator=g)
    first = second.roll(3, 1) + 0.3 * torch.randn(1, H * W, 16, generator=g)
    corr = (torch.matmul(first, second.transpose(1, 2)) / 2.0).to(dtype)
    want_flow, want_prob, want_blur, want_centre = oracle.flow_init(corr, H, W)
    flow, prob, blur, centre = _ma().flow_init(corr.cuda(), H, W, return_debug=True)
    steps = ((prob.float().cpu() - want_prob.float()).abs() - 2.0 ** -24).clamp_min(0)     # float16: below 2^-14 the spacing is 2^-24
    assert _close16(want_prob.float() + steps, want_prob, dtype)
    # 16 bits: an average of probabilities that are one step off, a relative 2^-10 (2^-7) at most, is less than two of its own
    # steps off, and rounding adds less than one
    assert _close16(blur, want_blur, dtype, ulps=3.0)
    same = centre.cpu() == want_centre
    assert same.float().mean() > 0.98           # the rest: equal box averages


@pytest.mark.parametrize("dtype", DTYPES)
def test_flow_init_of_a_row_without_numbers(dtype):
    """A token whose scores are not numbers has no arg max: its pooled maximum stays at minus infinity, its window at the
    far end of the map; the tokens two and more away do not see it."""
    H, W = 12, 14
    corr = torch.randn(1, H * W, H * W).to(dtype)
    corr[0, 70] = float("nan")
    flow, prob, blur, centre = _ma().flow_init(corr.cuda(), H, W, return_debug=True)
    assert (blur[0, 68:73] == -float("inf")).all() and prob[0].view(H * W, -1)[70].isnan().all()
    away = torch.ones(H * W, dtype=torch.bool)
    away[68:73] = False
    assert (blur[0].cpu()[away] > 0).all() and torch.isfinite(flow[0].cpu().view(-1, 2)[away]).all()
    assert ((centre >= 0) & (centre < H * W)).all()
