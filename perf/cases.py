"""The work that users of this package have it do, as cases that can be timed and compared.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare(case, seed)`` makes the
inputs that a caller holds before the call (device tensors, seeded), ``run(state)`` is one pass through the public
entry points.  Six kinds of use:

  operator     ``MF_FusedForwardOps``, the drop-in behind the model's ``mat_impl`` switch: one call, both outputs
  layer        what one attention layer of the patched model calls: ``consistency_mask`` of the field, the self branch
               (``self_attention_core``) and the cross branch (``cross_attention_core`` with gate and view swap)
  train        the operator forward and backward through autograd
  upsample     ``upsample_field``, the convex upsampling between stages (x2) and at the end (x4)
  stereo_init  ``stereo_volume`` and ``local_disparity_estimator``: correlation to first disparity field
  flow_init    ``flow_init``: all-pairs correlation to first flow field
"""
import math

import torch

import matchattention_b200 as ma

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
ESIZE = {"f16": 2, "bf16": 2, "f32": 4}

# Head widths of the models' stages (four heads each): 1/4 and 1/8 of the image with 3x3 sub-windows (r = 1),
# 1/16 and 1/32 with 5x5 ones (r = 2).
WIDTHS = {1: (8, 16, 32, 64), 2: (32, 40, 80, 128)}


def listed():
    return [
        # the coarsest stage of the smallest model at 1536x1536: few queries, wide windows, launch-bound
        dict(name="operator_48x48_r2_f16", kind="operator", B=2, H=48, W=48, h=4, hd=40, r=2, dtype="f16", offsets="disparity"),
        # one pair of 416x832 at 1/4 resolution in full precision, disparity-like random centres
        dict(name="operator_104x208_f32", kind="operator", B=1, H=104, W=208, h=8, hd=16, r=1, dtype="f32", offsets="cross"),
        # the benchmark's default: batch of four 1536x1536 maps at 1/4, flow-like random centres, some beyond the border
        dict(name="operator_384x384_b4_f16", kind="operator", B=4, H=384, W=384, h=8, hd=16, r=1, dtype="f16", offsets="flow"),
        # a ragged crop through a wide-headed stage in bfloat16, every head with a centre of its own
        dict(name="operator_187x313_bf16", kind="operator", B=2, H=187, W=313, h=4, hd=64, r=1, dtype="bf16", offsets="self"),
        # 1/16 stage of the smallest model at 1536x1536, as the patched model runs a layer of it
        dict(name="layer_96x96_r2_f16", kind="layer", B=2, H=96, W=96, h=4, hd=32, r=2, dtype="f16"),
        # 1/8 stage of the largest model at 2176x3840
        dict(name="layer_272x480_f16", kind="layer", B=2, H=272, W=480, h=4, hd=64, r=1, dtype="f16"),
        # training on one 1536x1536 map at 1/4, gradients of both outputs (a cross branch)
        dict(name="train_384x384_f16", kind="train", B=1, H=384, W=384, h=8, hd=16, r=1, dtype="f16", offsets="flow", attn_grad=True),
        # training on crops at a coarse stage in full precision, the attention weights discarded (a self branch)
        dict(name="train_45x79_r2_f32", kind="train", B=2, H=45, W=79, h=4, hd=32, r=2, dtype="f32", offsets="self", attn_grad=False),
        # the last step of the model at 1536x1536
        dict(name="upsample_384x384_x4_f16", kind="upsample", B=2, H=384, W=384, factor=4, dtype="f16"),
        # the first step of the stereo model at 2176x3840 (1/32 resolution)
        dict(name="stereo_init_68x120_f16", kind="stereo_init", B=1, H=68, W=120, dtype="f16"),
        # the first step of the flow model at 1536x1536 and at 4096x4096 (1/32 resolution)
        dict(name="flow_init_48x48_f16", kind="flow_init", B=1, H=48, W=48, dtype="f16"),
        dict(name="flow_init_128x128_f16", kind="flow_init", B=1, H=128, W=128, dtype="f16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dtype(rng):
    return rng.choice(("f16", "f16", "f16", "bf16", "f32"))


def _stage(rng, most):
    """Token map, heads and window of a stage, at most `most` elements in one [B, H*W, C] tensor of two views."""
    while True:
        r = rng.choice((1, 1, 2))
        h, hd = 4, rng.choice(WIDTHS[r])
        if r == 1 and rng.random() < 0.25:
            h, hd = 8, 16
        hi = 480 if r == 1 else 160
        H, W = _log_int(rng, 24, hi), _log_int(rng, 24, hi)
        if 2 * H * W * h * hd * (1 if r == 1 else 2) <= most:
            return dict(H=H, W=W, h=h, hd=hd, r=r)


def draw(rng):
    kind = rng.choice(("operator",) * 6 + ("layer",) * 4 + ("train",) * 4 + ("upsample",) * 2 + ("stereo_init",) * 2 +
                      ("flow_init",) * 2)
    dtype = _dtype(rng)
    if kind == "operator":
        return dict(kind=kind, B=rng.choice((1, 2, 2)), dtype=dtype, offsets=rng.choice(("flow", "cross", "disparity", "self")),
                    **_stage(rng, 70_000_000))
    if kind == "layer":
        return dict(kind=kind, B=2, dtype=dtype, **_stage(rng, 70_000_000))
    if kind == "train":
        return dict(kind=kind, B=rng.choice((1, 2)), dtype=dtype, offsets=rng.choice(("flow", "cross", "disparity", "self")),
                    attn_grad=rng.random() < 0.5, **_stage(rng, 24_000_000))
    if kind == "upsample":
        return dict(kind=kind, B=2, H=_log_int(rng, 32, 544), W=_log_int(rng, 32, 544), factor=rng.choice((2, 4)), dtype=dtype)
    if kind == "stereo_init":
        return dict(kind=kind, B=rng.choice((1, 1, 2, 4)), H=_log_int(rng, 16, 128), W=_log_int(rng, 24, 159), dtype=dtype)
    hi = 128 if dtype != "f32" else 88
    return dict(kind=kind, B=1, H=_log_int(rng, 16, hi), W=_log_int(rng, 16, hi), dtype=dtype)


# ---- inputs ---------------------------------------------------------------------------------------------

def _smooth(g, B, C, H, W, lo, hi):
    """Fields that vary slowly over the map, in [lo, hi]: [B, C, H, W]."""
    coarse = torch.rand(B, C, 7, 7, generator=g, device="cuda") * (hi - lo) + lo
    return torch.nn.functional.interpolate(coarse, size=(H, W), mode="bilinear", align_corners=True)


def _grid(H, W):
    ys, xs = torch.meshgrid(torch.arange(H, device="cuda", dtype=torch.float32),
                            torch.arange(W, device="cuda", dtype=torch.float32), indexing="ij")
    return torch.stack((xs, ys), -1).view(1, H * W, 1, 2)


def _clamped(centre, H, W, r, dtype):
    """Centres as the model hands them to the operator: limited to the map in the tensor type."""
    centre = centre.to(dtype)
    x = centre[..., :1].clamp(torch.tensor(float(r), dtype=dtype).item(), torch.tensor(W - 1 - r - 1e-3, dtype=dtype).item())
    y = centre[..., 1:].clamp(torch.tensor(float(r), dtype=dtype).item(), torch.tensor(H - 1 - r - 1e-3, dtype=dtype).item())
    return torch.cat((x, y), -1).contiguous()


def _centres(g, B, H, W, h, r, offsets, dtype):
    N, grid = H * W, _grid(H, W)

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo

    if offsets == "self":          # small, every head its own
        return _clamped(grid + uniform(-3.0, 3.0, B, N, h, 2), H, W, r, dtype)
    if offsets == "disparity":     # a smooth disparity field, shared by the heads
        d = _smooth(g, B, 1, H, W, -W / 8.0, 0.0).view(B, N, 1, 1)
        return _clamped((grid + torch.cat((d, torch.zeros_like(d)), -1)).expand(B, N, h, 2), H, W, r, dtype)
    if offsets == "cross":         # random disparities of up to 16 tokens, shared by the heads
        d = uniform(-16.0, 0.0, B, N, 1, 1)
        return _clamped((grid + torch.cat((d, torch.zeros_like(d)), -1)).expand(B, N, h, 2), H, W, r, dtype)
    # "flow": uniform in +-24 tokens, shared by the heads; a tenth of the centres lies at or beyond the border, unclamped
    mo = _clamped((grid + uniform(-24.0, 24.0, B, N, 1, 2)).expand(B, N, h, 2), H, W, r, dtype)
    edge = torch.randint(0, 4, (B, N, 1, 1), generator=g, device="cuda")
    depth, along = uniform(-(r + 1.0), r + 1.0, B, N, 1, 1), uniform(0.0, 1.0, B, N, 1, 1)
    bx = torch.where(edge == 0, depth, torch.where(edge == 1, (W - 1) - depth, along * (W - 1)))
    by = torch.where(edge == 2, depth, torch.where(edge == 3, (H - 1) - depth, along * (H - 1)))
    border = torch.cat((bx, by), -1).expand(B, N, h, 2).to(dtype)
    pick = uniform(0.0, 1.0, B, N, 1, 1) < 0.1
    return torch.where(pick, border, mo).contiguous()


def _features(g, n, channels):
    return torch.randn(n, channels, generator=g, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype, kind = DTYPES[case["dtype"]], case["kind"]
    B, H, W = case["B"], case["H"], case["W"]
    s = dict(case=case)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda").to(dtype)

    if kind in ("operator", "layer", "train"):
        N, h, hd, r = H * W, case["h"], case["hd"], case["r"]
        C, M = h * hd, (2 * r + 2) ** 2
        s.update(scale=hd ** -0.5, M=M)
        if kind == "layer":
            # a field whose two views agree but for noise (about the share of occlusions that real pairs have)
            d = _smooth(g, B // 2, 1, H, W, 0.0, W / 8.0)
            sign = torch.cat((-d, d)).view(B, H, W, 1)
            field = torch.cat((sign, torch.zeros_like(sign)), -1)
            field = field + torch.randn(B, H, W, 2, generator=g, device="cuda") * torch.tensor([0.5, 0.0], device="cuda")
            s["field"] = field.to(dtype).contiguous()
            s["cross_centre"] = (_grid(H, W) + field.view(B, N, 1, 2)).expand(B, N, h, 2).to(dtype).contiguous()
            s["self_centre"] = (_grid(H, W) + torch.rand(B, N, h, 2, generator=g, device="cuda") * 2 - 1).to(dtype).contiguous()
            s["self_qkv"] = tuple(normal(B, N, C) for _ in range(3))
            s["cross_qkv"] = tuple(normal(B, N, C) for _ in range(3))
            s["gate"] = normal(B, N, C)
            return s
        s["inputs"] = (_centres(g, B, H, W, h, r, case["offsets"], dtype), normal(B, N, C), normal(B, N, C), normal(B, N, C))
        s["module"] = ma.MF_FusedForwardOps()
        if kind == "train":
            s["inputs"] = tuple(t.requires_grad_(True) for t in s["inputs"])
            s["g_out"] = normal(B, N, C)
            s["g_attn"] = normal(B, N, h, M) if case["attn_grad"] else None
        return s
    if kind == "upsample":
        s["field"] = (_smooth(g, B, 2, H, W, -H / 8.0, H / 8.0).permute(0, 2, 3, 1) +
                      torch.randn(B, H, W, 2, generator=g, device="cuda") * 0.25).to(dtype).contiguous()
        s["mask"] = normal(B, 9 * case["factor"] ** 2, H, W)
        return s
    # correlation of 32-channel features that have a true match in the other view, plus noise
    channels = 32
    if kind == "stereo_init":
        right = torch.randn(B, H, W, channels, generator=g, device="cuda")
        d = _smooth(g, B, 1, H, W, 0.0, W / 4.0).round().long().view(B, H, W)
        at = (torch.arange(W, device="cuda").view(1, 1, W) - d).clamp(min=0)
        left = right.gather(2, at.unsqueeze(-1).expand(B, H, W, channels))
        left = left + 0.3 * torch.randn(B, H, W, channels, generator=g, device="cuda")
        s["correlation"] = (torch.matmul(left, right.transpose(-2, -1)) * (2 * channels ** -0.5)).to(dtype).contiguous()
        return s
    N = H * W
    second = torch.randn(B, N, channels, generator=g, device="cuda")
    flow = _smooth(g, B, 2, H, W, -H / 16.0, H / 16.0).round().long()
    ys, xs = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    at = ((ys + flow[:, 1]).clamp(0, H - 1) * W + (xs + flow[:, 0]).clamp(0, W - 1)).view(B, N, 1)
    first = second.gather(1, at.expand(B, N, channels)) + 0.3 * torch.randn(B, N, channels, generator=g, device="cuda")
    s["correlation"] = (torch.matmul(first.to(dtype), second.to(dtype).transpose(-2, -1)) * (2 * channels ** -0.5)).contiguous()
    return s


# ---- one pass -------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind, H, W = case["kind"], case["H"], case["W"]
    if kind == "operator":
        r = case["r"]
        return s["module"](*s["inputs"], H, W, [r, r], s["M"], attn_type="l1_norm", scale=s["scale"])
    if kind == "layer":
        r = case["r"]
        mask = ma.consistency_mask(s["field"])
        own = ma.self_attention_core(s["self_centre"], *s["self_qkv"], H, W, r, s["scale"])
        other = ma.cross_attention_core(s["cross_centre"], *s["cross_qkv"], s["gate"], H, W, r, s["scale"],
                                        kv_shift=case["B"] // 2)
        return mask, own, other
    if kind == "train":
        r = case["r"]
        out, attn = s["module"](*s["inputs"], H, W, [r, r], s["M"], attn_type="l1_norm", scale=s["scale"])
        if s["g_attn"] is None:
            grads = torch.autograd.grad([out], s["inputs"], [s["g_out"]])
        else:
            grads = torch.autograd.grad([out, attn], s["inputs"], [s["g_out"], s["g_attn"]])
        return (out, attn) + tuple(grads)
    if kind == "upsample":
        return ma.upsample_field(s["field"], s["mask"], case["factor"])
    if kind == "stereo_init":
        volume = ma.stereo_volume(s["correlation"])
        return ma.local_disparity_estimator(volume), volume
    return ma.flow_init(s["correlation"], H, W)


# ---- what a pass cannot do without ----------------------------------------------------------------------

def work(case):
    """Each input read once and each output written once; the arithmetic of the definition."""
    e, kind, B, N = ESIZE[case["dtype"]], case["kind"], case["B"], case["H"] * case["W"]
    if kind in ("operator", "layer", "train"):
        h, C, M = case["h"], case["h"] * case["hd"], (2 * case["r"] + 2) ** 2
        forward = B * N * (4 * C * M + 30 * h * M)             # |q-k| sums, weighted sums; four softmaxes and their blend
        if kind == "operator":
            return dict(bytes=e * B * N * (4 * C + 2 * h + h * M), flops=forward)
        if kind == "layer":
            return dict(bytes=e * B * N * ((4 * C + 2 * h) + (5 * C + 2 * h + h * M) + 3), flops=2 * forward)
        # forward: q, k, v, centres in, out, attn out; backward: those inputs, d_out (d_attn) in, four gradients out
        grad_in = C + (h * M if case["attn_grad"] else 0)
        return dict(bytes=e * B * N * ((4 * C + 2 * h + h * M) + (3 * C + 2 * h + grad_in) + (3 * C + 2 * h)),
                    flops=3 * forward)
    if kind == "upsample":
        f2 = case["factor"] ** 2
        return dict(bytes=e * B * N * (2 + 9 * f2 + 2 * f2), flops=B * N * f2 * 9 * 8)
    if kind == "stereo_init":
        # correlation in; volume of both views out; field of both views out
        return dict(bytes=e * B * N * (case["W"] + 2 * case["W"] + 4), flops=2 * B * N * case["W"] * 12)
    return dict(bytes=e * B * N * (N + 2 * N + 4), flops=2 * B * N * N * 12)


def tolerance(case):
    """16-bit types: the spacing of the type, and for single values a score that rounds to its neighbour (scores of
    up to 20 are held in the type).  float32: sums and exponentials in another order."""
    return {"f16": {"rel": 1e-3, "max": 0.05}, "bf16": {"rel": 6e-3, "max": 0.3}, "f32": {"rel": 2e-5, "max": 2e-3}}[case["dtype"]]
