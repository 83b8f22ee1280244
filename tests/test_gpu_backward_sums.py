"""Token sums of the backward against the accumulating kernel: maps of more tiles than the coefficients are fetched ahead,
every split of a token's channels over lanes, row bands, two batch items."""
import pytest
import torch

from _cases import make_inputs

pytestmark = pytest.mark.gpu


def _both(mo, q, k, v, g_out, g_attn, H, W, h, r, scale, rows):
    """(d_max_offset, d_q, d_k, d_v) by the gathered and by the accumulating call, through the C ABI."""
    from matchattention_b200 import _lib
    B, C = q.size(0), q.size(2)
    code = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}[q.dtype]
    head = [t.data_ptr() for t in (mo, q, k, v, g_out)] + [g_attn.data_ptr() if g_attn is not None else None]
    shape = (B, H, W, h, C // h, r, r, code, _lib.L1_NORM, scale, *rows)
    stream = torch.cuda.current_stream().cuda_stream
    size = _lib.lib.matchattn_backward_workspace_bytes(B, H, W, h, C // h, r, code, *rows)
    assert size > 0
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    got = [torch.empty_like(t) for t in (mo, q, k, v)]
    _lib.check(_lib.lib.matchattn_fused_backward_ws(*head, got[1].data_ptr(), got[2].data_ptr(), got[3].data_ptr(), got[0].data_ptr(), *shape,
                                                    ws.data_ptr(), size, stream))
    want = [torch.empty_like(mo), torch.empty_like(q), torch.zeros(k.shape, device="cuda"), torch.zeros(v.shape, device="cuda")]
    _lib.check(_lib.lib.matchattn_fused_backward(*head, want[1].data_ptr(), want[2].data_ptr(), want[3].data_ptr(), want[0].data_ptr(), *shape,
                                                 stream))
    return got, want


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.float16, 2e-3), (torch.bfloat16, 1.6e-2)], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("per_head", [False, True], ids=["shared", "per-head"])
@pytest.mark.parametrize("B,H,W,h,hd,r,band", [(1, 97, 103, 8, 16, 1, None), (2, 61, 85, 4, 64, 1, None), (1, 90, 101, 4, 8, 1, None),
                                               (2, 23, 31, 4, 40, 2, None), (1, 29, 37, 4, 80, 2, None), (1, 24, 26, 4, 128, 2, None),
                                               (2, 30, 27, 4, 32, 2, (7, 19)), (2, 40, 33, 2, 16, 1, (0, 13)), (1, 19, 21, 1, 256, 1, None)])
def test_token_sums_match_the_accumulating_kernel(B, H, W, h, hd, r, band, per_head, dtype, tol):
    mo, q, k, v = make_inputs(91 + hd, B, H, W, h, hd, r, dtype, kind="flow", spread=5.0, border_frac=0.1, per_head=per_head)
    if not per_head:
        mo = mo[:, :, :1].expand_as(mo).contiguous()
    gen = torch.Generator().manual_seed(92)
    g_out = torch.randn(q.shape, generator=gen).to(dtype)
    g_attn = torch.randn(B, H * W, h, (2 * r + 2) ** 2, generator=gen).to(dtype)
    rows = band or (0, H)
    cut = slice(rows[0] * W, rows[1] * W)
    mo, q, g_out, g_attn = (t[:, cut].contiguous().cuda() for t in (mo, q, g_out, g_attn))
    got, want = _both(mo, q, k.cuda(), v.cuda(), g_out, g_attn, H, W, h, r, hd ** -0.5, rows)
    # the same float32 terms summed in another order and rounded once: the tolerance of the type, over the largest value
    for g, ref, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        ref = ref.double()
        assert (g.double() - ref).abs().max() <= tol * ref.abs().max(), key
