"""flow_init where every chunk of targets holds the largest box average: more chunks than a warp looks at together, and more
than a block keeps."""
import pytest
import torch

import matchattention_b200 as ma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,W", [(5, 7), (34, 32), (72, 71), (129, 128)])
def test_equal_averages_keep_the_first_target(H, W, dtype):
    N = H * W
    if N > 16384 and dtype == torch.float32:
        pytest.skip("2.2 GB of probabilities, 1.1 GB of scores")
    corr = torch.zeros(1, N, N, dtype=dtype, device="cuda")
    flow, prob, blur, centre = ma.flow_init(corr, H, W, return_debug=True)
    # a box of 25 equal terms first lies inside the row at target 2, which the window's clamp moves to row 2
    assert torch.equal(centre.view(-1).cpu(), torch.full((2 * N,), 2 * W + 2, dtype=centre.dtype))
    p = torch.tensor(1.0 / N, dtype=torch.float32).to(dtype)
    assert torch.equal(prob.view(-1)[:: N // 3].cpu(), p.expand(prob.numel()).contiguous()[:: N // 3])
    assert torch.isfinite(flow).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,W,late,half", [(72, 71, 33 * 120, 0), (72, 71, 33 * 64, 1), (129, 128, 33 * 120, 0), (129, 128, 256 * 64, 1)],
                         ids=["rows, chunk 33 on", "columns, band 33 on", "rows, large map", "columns, band 256 on"])
def test_the_largest_average_lies_in_a_late_chunk(H, W, late, half, dtype):
    """One largest box per token, in a late chunk (row half: 120 targets each) or band (column half: 64), beyond those that a
    warp looks at together and that a block keeps; the tokens of a block of eight have up to three different targets."""
    N = H * W
    gen = torch.Generator().manual_seed(N + half)
    target = torch.full((N,), -1)
    height = torch.zeros(N)
    # every fourth token has a peak: a high one, late for every other block of eight, and a lower one, always late
    high, low = torch.arange(3, N - 8, 8), torch.arange(7, N - 8, 8)
    middle = (late + N) // 2        # (never within a box of each other)
    target[high] = torch.randint(4, late - 8, (len(high),), generator=gen)
    target[high[::2]] = torch.randint(late + 4, middle - 8, (len(high[::2]),), generator=gen)
    target[low] = torch.randint(middle + 8, N - 4, (len(low),), generator=gen)
    height[high], height[low] = 10.0, 9.0
    scores = torch.zeros(N, N, device="cuda")
    peak = torch.nonzero(target >= 0).view(-1)
    for off in range(-2, 3):        # peaks five targets wide: the box around the middle holds all of it
        scores[peak.cuda(), (target[peak] + off).cuda()] = (height[peak] - abs(off)).cuda()
    corr = (scores if half == 0 else scores.t()).to(dtype).contiguous().view(1, N, N)
    flow, prob, blur, centre = ma.flow_init(corr, H, W, return_debug=True)
    # the box of token i sees the rows i - 2 .. i + 2: the higher peak among them
    token = torch.arange(16, N - 16)
    source = torch.where(token % 8 == 0, token - 1, torch.where(token % 8 >= 6, token // 8 * 8 + 7, token // 8 * 8 + 3))
    want = target[source]
    clamped = (want // W).clamp(2, H - 3) * W + (want % W).clamp(2, W - 3)
    assert torch.equal(centre.view(2, N)[half].cpu()[token], clamped.to(centre.dtype))
    p = prob.view(2, N, N)[half]
    box = torch.zeros(len(token), dtype=torch.float64, device="cuda")
    for di in range(-2, 3):
        for dj in range(-2, 3):
            box += p[(token + di).cuda(), (want + dj).cuda()].double()
    # 24 float32 additions and a division, then one rounding to the type
    step = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype] + 25 * 2.0 ** -24
    assert ((blur.view(2, N)[half].double()[token.cuda()] * 25 - box).abs() <= step * box).all()
