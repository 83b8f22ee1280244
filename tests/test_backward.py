"""Backward of the operator.

CPU: the plain-loop restatement of the gradient formulas (oracle/matchattn_backward.py) against the gradients
autograd gives over the reference's own functions (tests/golden/backward_*.npz).
GPU: the CUDA backward, through the autograd function and the reference-compatible module, against the same
vectors, and against autograd over the reference's functions run on the same GPU (float32 and float16)."""
import numpy as np
import pytest
import torch

from _cases import golden_names_with_prefix, load_golden_arrays, make_inputs


def _rel(got, ref):
    got, ref = torch.as_tensor(got).double().cpu(), torch.as_tensor(ref).double().cpu()
    return float((got - ref).abs().max() / ref.abs().max().clamp_min(1e-6))


@pytest.mark.parametrize("name", golden_names_with_prefix("backward_"))
def test_backward_restatement_matches_reference_autograd(name):
    from oracle import matchattn_backward
    c = load_golden_arrays(name)
    got = matchattn_backward.backward(c["max_offset"], c["q"], c["k"], c["v"], c["g_out"], c["g_attn"], c["H"], c["W"],
                                      c["r"], c["scale"])
    for g, key in zip(got, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(g, c[key]) < 1e-5, key


@pytest.mark.gpu
@pytest.mark.parametrize("name", golden_names_with_prefix("backward_"))
def test_backward_kernel_matches_reference_autograd_vectors(name):
    import matchattention_b200 as ma
    c = load_golden_arrays(name)
    leaves = [c[n].cuda().requires_grad_(True) for n in ("max_offset", "q", "k", "v")]
    out, attn = ma.match_attention_autograd(*leaves, c["H"], c["W"], c["r"], c["scale"])
    ((out * c["g_out"].cuda()).sum() + (attn * c["g_attn"].cuda()).sum()).backward()
    for leaf, key in zip(leaves, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(leaf.grad, c[key]) < 1e-4, key


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.float16, 2e-2)], ids=["f32", "f16"])
@pytest.mark.parametrize("need_attn_grad", [True, False])
def test_backward_kernel_matches_reference_autograd_on_the_gpu(dtype, tol, need_attn_grad):
    """Through MF_FusedForwardOps (the reference's module interface) on a model-like shape; in float16 the
    reference's autograd rounds every intermediate to 16 bits while the kernel works in float32, hence the
    looser bound there."""
    from oracle import ref_loader
    if not ref_loader.available():
        pytest.skip("the reference's Python code is not present (oracle/make_ref.py places it under oracle/_ref/)")
    impl, _ = ref_loader.import_reference()
    import matchattention_b200 as ma
    B, H, W, h, hd, r = 2, 24, 31, 4, 16, 1
    inputs = make_inputs(55, B, H, W, h, hd, r, dtype, kind="flow", spread=5.0, border_frac=0.1, per_head=True)
    g = torch.Generator().manual_seed(56)
    g_out = torch.randn(inputs[1].shape, generator=g).to(dtype).cuda()
    g_attn = torch.randn(B, H * W, h, 16, generator=g).to(dtype).cuda()

    def run(fn):
        leaves = [t.cuda().requires_grad_(True) for t in inputs]
        out, attn = fn(*leaves)
        loss = (out.float() * g_out.float()).sum()
        if need_attn_grad:
            loss = loss + (attn.float() * g_attn.float()).sum()
        loss.backward()
        return [t.grad for t in leaves]

    want = run(lambda mo, q, k, v: ref_loader.reference_op(impl, mo, q, k, v, H, W, h, r, hd ** -0.5))
    module = ma.MF_FusedForwardOps()
    got = run(lambda mo, q, k, v: module(mo, q, k, v, H, W, [r, r], 16, attn_type="l1_norm", scale=hd ** -0.5))
    for gg, ww, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(gg, ww) < tol, key


@pytest.mark.gpu
def test_inference_path_is_untouched_by_autograd_support():
    import matchattention_b200 as ma
    mo, q, k, v = (t.cuda() for t in make_inputs(57, 1, 12, 13, 2, 16, 1, torch.float16, kind="self"))
    with torch.no_grad():
        out, attn = ma.MF_FusedForwardOps()(mo, q.requires_grad_(True), k, v, 12, 13, [1, 1], 16, scale=0.25)
    assert not out.requires_grad and out.grad_fn is None


@pytest.mark.gpu
@pytest.mark.parametrize("h,hd,r", [(3, 12, 1), (2, 8, 3), (2, 24, 2), (8, 16, 1)],
                         ids=["scalar-hd12", "scalar-r3", "vector-hd24-r2", "vector-hd16-r1"])
def test_backward_kernels_match_the_restatement(h, hd, r):
    """Autograd against the float64 plain-loop restatement, on either way it takes: gathered sums for head widths that are
    multiples of 8 and r <= 2 (the ids say "vector"), the accumulating kernel one element at a time otherwise."""
    import matchattention_b200 as ma
    from oracle import matchattn_backward
    B, H, W = 1, 9, 10
    mo, q, k, v = make_inputs(57, B, H, W, h, hd, r, torch.float32, kind="flow", spread=3.0, border_frac=0.2,
                              per_head=True)
    gen = torch.Generator().manual_seed(58)
    g_out = torch.randn(q.shape, generator=gen)
    g_attn = torch.randn(B, H * W, h, (2 * r + 2) ** 2, generator=gen)
    want = matchattn_backward.backward(mo, q, k, v, g_out, g_attn, H, W, r, hd ** -0.5)
    leaves = [t.cuda().requires_grad_(True) for t in (mo, q, k, v)]
    out, attn = ma.match_attention_autograd(*leaves, H, W, r, hd ** -0.5)
    ((out * g_out.cuda()).sum() + (attn * g_attn.cuda()).sum()).backward()
    for leaf, ref, key in zip(leaves, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(leaf.grad, ref) < 1e-4, key


@pytest.mark.gpu
@pytest.mark.parametrize("per_head", [False, True], ids=["shared", "per-head"])
@pytest.mark.parametrize("B,H,W,h,hd,r,kind", [(1, 4, 4, 2, 8, 1, "raw"), (1, 6, 7, 1, 40, 2, "raw"), (2, 9, 17, 2, 16, 1, "flow"),
                                               (1, 17, 9, 2, 80, 2, "raw"), (1, 8, 16, 4, 24, 1, "self"), (1, 8, 8, 4, 128, 1, "flow"),
                                               (1, 10, 33, 2, 16, 1, "corner")])
def test_gathered_backward_at_the_edges_of_its_tiles(B, H, W, h, hd, r, kind, per_head):
    """Maps of one bucket, of one tile and one token more, windows that stick out of the map on every side, and all
    queries on the corner token; with one centre per query (one list for all heads) and with one per head."""
    import matchattention_b200 as ma
    from oracle import matchattn_backward
    mo, q, k, v = make_inputs(61 + hd, B, H, W, h, hd, r, torch.float32, kind="raw" if kind == "corner" else kind, spread=3.0,
                              border_frac=0.3, per_head=per_head)
    if kind == "corner":
        mo = mo * 0 - 40.0 + torch.arange(h, dtype=torch.float32).view(1, 1, h, 1) * (40.0 if per_head else 0.0)
    if not per_head:
        mo = mo[:, :, :1].expand_as(mo).contiguous()
    gen = torch.Generator().manual_seed(62)
    g_out = torch.randn(q.shape, generator=gen)
    g_attn = torch.randn(B, H * W, h, (2 * r + 2) ** 2, generator=gen)
    want = matchattn_backward.backward(mo, q, k, v, g_out, g_attn, H, W, r, hd ** -0.5)
    leaves = [t.cuda().requires_grad_(True) for t in (mo, q, k, v)]
    out, attn = ma.match_attention_autograd(*leaves, H, W, r, hd ** -0.5)
    got = torch.autograd.grad([out, attn], leaves, [g_out.cuda(), g_attn.cuda()])
    for g, ref, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        ref = torch.as_tensor(ref).double()         # on one token the score gradients cancel: d_q and d_k are zero up to rounding
        assert (g.double().cpu() - ref).abs().max() < 1e-4 * max(ref.abs().max().item(), 0.05), key


def _accumulate(mo, q, k, v, g_out, g_attn, H, W, r, scale, dk, dv):
    """matchattn_fused_backward through the C ABI: d_max_offset and d_q; dk and dv (float32) are added to."""
    from matchattention_b200 import _lib
    B, N, C = q.shape
    h = mo.size(2)
    d_q, d_mo = torch.empty_like(q), torch.empty_like(mo)
    code = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}[q.dtype]
    _lib.check(_lib.lib.matchattn_fused_backward(
        mo.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), g_out.data_ptr(), g_attn.data_ptr() if g_attn is not None else None,
        d_q.data_ptr(), dk.data_ptr(), dv.data_ptr(), d_mo.data_ptr(), B, H, W, h, C // h, r, r, code, _lib.L1_NORM, scale, 0, H,
        torch.cuda.current_stream().cuda_stream))
    return d_mo, d_q


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.float16, 2e-3), (torch.bfloat16, 1.6e-2)], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("need_attn_grad", [True, False])
@pytest.mark.parametrize("h,hd,r", [(3, 12, 1), (2, 8, 3), (2, 24, 2), (8, 16, 1)],
                         ids=["scalar-hd12", "scalar-r3", "vector-hd24-r2", "vector-hd16-r1"])
def test_accumulating_backward_kernels_match_the_restatement(h, hd, r, need_attn_grad, dtype, tol):
    """Both kernels of the accumulating entry point (one element at a time; eight channels at a time), on top of what dk
    and dv hold.  16-bit types: float32 arithmetic on the rounded inputs, one rounding of d_q and d_max_offset (2^-11,
    2^-8), four times that."""
    from oracle import matchattn_backward
    B, H, W = 2, 9, 10
    mo, q, k, v = make_inputs(57, B, H, W, h, hd, r, dtype, kind="flow", spread=3.0, border_frac=0.2, per_head=True)
    gen = torch.Generator().manual_seed(58)
    g_out = torch.randn(q.shape, generator=gen).to(dtype)
    g_attn = torch.randn(B, H * W, h, (2 * r + 2) ** 2, generator=gen).to(dtype)
    want = matchattn_backward.backward(*(t.float() for t in (mo, q, k, v, g_out)), (g_attn if need_attn_grad else g_attn * 0).float(),
                                       H, W, r, hd ** -0.5)
    dk, dv = torch.full(k.shape, 0.5, device="cuda"), torch.full(v.shape, -2.0, device="cuda")
    d_mo, d_q = _accumulate(*(t.cuda() for t in (mo, q, k, v, g_out)), g_attn.cuda() if need_attn_grad else None, H, W, r, hd ** -0.5, dk, dv)
    for got, ref, key in zip((d_mo, d_q, dk - 0.5, dv + 2.0), want, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(got, ref) < tol, key


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("h,hd,r,gathered", [(2, 16, 1, True), (2, 24, 1, True), (2, 16, 1, False), (2, 24, 2, True), (2, 24, 2, False),
                                             (2, 12, 1, False)])
def test_an_infinite_gradient_of_a_weight(h, hd, r, gathered, dtype):
    """Every route gives the values of the definition, sign(q - k) times the gradient of the score: not finite where that is
    not, a channel with q = k (0 times infinity) included."""
    from oracle import matchattn_backward
    from test_gpu_backward_sums import _both
    B, H, W = 1, 9, 10
    mo, q, k, v = make_inputs(67, B, H, W, h, hd, r, dtype, kind="flow", spread=3.0, per_head=True)
    q[..., 3] = k[..., 3] = 0.5
    mo[0, 37, 0] = torch.tensor([4.53125, 4.28125])         # all four windows count
    gen = torch.Generator().manual_seed(68)
    g_out = torch.randn(q.shape, generator=gen).to(dtype)
    g_attn = torch.randn(B, H * W, h, (2 * r + 2) ** 2, generator=gen).to(dtype)
    g_attn[0, 37, 0, (2 * r + 2) + 1] = float("inf")
    with np.errstate(invalid="ignore"):
        want = matchattn_backward.backward(*(t.float() for t in (mo, q, k, v, g_out, g_attn)), H, W, r, hd ** -0.5)
    assert np.isfinite(want[2]).sum() < want[2].size
    args = [t.cuda() for t in (mo, q, k, v, g_out, g_attn)]
    if gathered:
        got, _ = _both(*args, H, W, h, r, hd ** -0.5, (0, H))
    else:
        dk, dv = torch.zeros(k.shape, device="cuda"), torch.zeros(v.shape, device="cuda")
        got = (*_accumulate(*args, H, W, r, hd ** -0.5, dk, dv), dk, dv)
    tol = {torch.float32: 1e-4, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]        # those of the tests above
    for g, ref, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        g, ref = g.double().cpu(), torch.as_tensor(ref).double()
        finite = ref.isfinite()
        assert torch.equal(g.isfinite(), finite), key
        assert (g[finite] - ref[finite]).abs().max() <= tol * ref[finite].abs().max(), key


def _step(inputs, g_out, g_attn, H, W, r, scale):
    import matchattention_b200 as ma
    out, attn = ma.match_attention_autograd(*inputs, H, W, r, scale)
    return lambda: torch.autograd.grad([out, attn], inputs, [g_out, g_attn])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float16, 2e-3)], ids=["f32", "f16"])
@pytest.mark.parametrize("offset", [16, 4])
def test_training_on_arrays_that_are_not_32_byte_aligned(offset, dtype, tol):
    """Views some bytes into a buffer: the backward with a workspace declines and the accumulating one serves, with the
    gradients of the aligned arrays (float32 sums in another order; 16 bits: one rounding apart)."""
    B, H, W, h, hd, r = 1, 20, 33, 4, 16, 1
    inputs = [t.cuda() for t in make_inputs(63, B, H, W, h, hd, r, dtype, kind="flow", spread=3.0, per_head=True)]
    gen = torch.Generator(device="cuda").manual_seed(64)
    g_out = torch.randn(inputs[1].shape, generator=gen, device="cuda").to(dtype)
    g_attn = torch.randn(B, H * W, h, 16, generator=gen, device="cuda").to(dtype)

    def moved(t):
        skip = offset // t.element_size()
        return torch.empty(t.numel() + skip, dtype=dtype, device="cuda")[skip:].view(t.shape).copy_(t)

    want = _step([t.requires_grad_(True) for t in inputs], g_out, g_attn, H, W, r, hd ** -0.5)()
    views = [inputs[0].detach().requires_grad_(True)] + [moved(t.detach()).requires_grad_(True) for t in inputs[1:]]
    assert views[1].data_ptr() % 32 == offset % 32
    got = _step(views, g_out, g_attn, H, W, r, hd ** -0.5)()
    for g, w, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(g, w) < tol, key


@pytest.mark.gpu
def test_training_without_room_for_the_workspace():
    """When the workspace (44 MB here) finds no room the accumulating call serves: the same gradients, no workspace.  The limit
    is the caching allocator's own, far below what the device holds."""
    from matchattention_b200 import _lib
    B, H, W, h, hd, r = 1, 192, 192, 4, 8, 2
    inputs = [t.cuda().requires_grad_(True) for t in make_inputs(65, B, H, W, h, hd, r, torch.float32, kind="self")]
    gen = torch.Generator(device="cuda").manual_seed(66)
    g_out = torch.randn(inputs[1].shape, generator=gen, device="cuda")
    g_attn = torch.randn(B, H * W, h, 36, generator=gen, device="cuda")
    want = _step(inputs, g_out, g_attn, H, W, r, 0.25)()
    nbytes = _lib.lib.matchattn_backward_workspace_bytes(B, H, W, h, hd, r, _lib.F32, 0, H)
    assert nbytes > 40 << 20
    backward = _step(inputs, g_out, g_attn, H, W, r, 0.25)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    try:        # room for the gradients (16 MB, in one 20 MB segment), not for the workspace
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (24 << 20)) /
                                                   torch.cuda.get_device_properties(0).total_memory)
        got = backward()
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.cuda.max_memory_allocated() - held < nbytes
    for g, w, key in zip(got, want, ("d_max_offset", "d_q", "d_k", "d_v")):
        assert _rel(g, w) < 1e-5, key
