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
        pytest.skip("3.3 GB of probabilities")
    corr = torch.zeros(1, N, N, dtype=dtype, device="cuda")
    flow, prob, blur, centre = ma.flow_init(corr, H, W, return_debug=True)
    # a box of 25 equal terms first lies inside the row at target 2, which the window's clamp moves to row 2
    assert torch.equal(centre.view(-1).cpu(), torch.full((2 * N,), 2 * W + 2, dtype=centre.dtype))
    p = torch.tensor(1.0 / N, dtype=torch.float32).to(dtype)
    assert torch.equal(prob.view(-1)[:: N // 3].cpu(), p.expand(prob.numel()).contiguous()[:: N // 3])
    assert torch.isfinite(flow).all()
