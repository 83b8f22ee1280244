"""GPU tests of the reference-facing interface: the 12-argument in-place call,
the opaque custom op, the MF_FusedForwardOps module, the drop-in module name,
streams, CUDA graphs and error reporting."""
import importlib
import sys

import pytest
import torch

from _cases import assert_close, make_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    import oracle
    B, H, W, h, hd, r = 2, 30, 36, 4, 16, 1
    inputs = make_inputs(21, B, H, W, h, hd, r, torch.float16, kind="flow", spread=5.0)
    ref = oracle.forward(*inputs, H, W, r, 0.25)
    return dict(H=H, W=W, h=h, r=r, M=16, scale=0.25, cpu=inputs, gpu=tuple(t.cuda() for t in inputs), ref=ref)


def test_module_has_reference_signature(case):
    from matchattention_b200 import MF_FusedForwardOps
    mo, q, k, v = case["gpu"]
    out, attn = MF_FusedForwardOps()(mo, q, k, v, case["H"], case["W"], [case["r"]] * 2, case["M"],
                                     attn_type="l1_norm", scale=case["scale"])
    assert out.shape == q.shape and attn.shape == (*q.shape[:2], case["h"], case["M"])
    assert_close(out, case["ref"][0], torch.float16)
    assert_close(attn, case["ref"][1], torch.float16)


def test_dropin_module_name(case):
    import matchattention_b200
    matchattention_b200.install_dropin()
    mod = importlib.import_module("match_attention")
    mo, q, k, v = case["gpu"]
    out = torch.full_like(q, float("nan"))
    attn = torch.full((*q.shape[:2], case["h"], case["M"]), float("nan"), dtype=q.dtype, device=q.device)
    ret = mod.fused_forward(mo, q, k, v, out, attn, case["H"], case["W"], [1, 1], 16, "l1_norm", case["scale"])
    assert ret is None
    assert_close(out, case["ref"][0], torch.float16)
    assert_close(attn, case["ref"][1], torch.float16)
    sys.modules.pop("match_attention", None)


def test_custom_op_is_registered_and_opaque(case):
    import matchattention_b200  # noqa: F401
    mo, q, k, v = case["gpu"]
    out, attn = torch.empty_like(q), q.new_empty(*q.shape[:2], case["h"], 16)
    torch.ops.matchattn_b200.fused_forward_ops(mo, q, k, v, out, attn, case["H"], case["W"], [1, 1], 16, "l1_norm",
                                               case["scale"])
    assert_close(out, case["ref"][0], torch.float16)
    torch.library.opcheck(torch.ops.matchattn_b200.fused_forward_ops.default,
                          (mo, q, k, v, out, attn, case["H"], case["W"], [1, 1], 16, "l1_norm", case["scale"]),
                          test_utils=("test_schema", "test_faketensor"))


def test_side_stream_and_cuda_graph(case):
    from matchattention_b200 import match_attention
    mo, q, k, v = case["gpu"]
    out, attn = torch.empty_like(q), q.new_empty(*q.shape[:2], case["h"], 16)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            match_attention(mo, q, k, v, case["H"], case["W"], 1, case["scale"], out=out, attn_out=attn)
        graph = torch.cuda.CUDAGraph()
        out.zero_()
        with torch.cuda.graph(graph, stream=side):
            match_attention(mo, q, k, v, case["H"], case["W"], 1, case["scale"], out=out, attn_out=attn)
        out.zero_()
        graph.replay()
    side.synchronize()
    assert_close(out, case["ref"][0], torch.float16)


def test_bad_arguments_raise_and_leave_the_device_usable(case):
    from matchattention_b200 import match_attention, launch, fused_forward
    mo, q, k, v = case["gpu"]
    H, W = case["H"], case["W"]
    with pytest.raises(RuntimeError):      # CPU tensors: there is no CPU path
        match_attention(*case["cpu"], H, W, 1, 0.25)
    with pytest.raises(ValueError):        # wrong map size
        match_attention(mo, q, k, v, H + 1, W, 1, 0.25)
    with pytest.raises(ValueError):        # non-contiguous input
        match_attention(mo, q.transpose(0, 1).contiguous().transpose(0, 1), k, v, H, W, 1, 0.25)
    with pytest.raises(TypeError):         # mixed dtypes
        match_attention(mo.float(), q, k, v, H, W, 1, 0.25)
    with pytest.raises(NotImplementedError):   # a scoring function that does not exist
        launch(mo, q, k, v, torch.empty_like(q), None, H, W, (1, 1), "l2_norm", 1.0)
    with pytest.raises(RuntimeError):      # rx != ry is rejected by the library
        launch(mo, q, k, v, torch.empty_like(q), None, H, W, (1, 2), "l1_norm", 1.0)
    with pytest.raises(ValueError):        # attn_num inconsistent with win_r
        fused_forward(mo, q, k, v, torch.empty_like(q), q.new_empty(*q.shape[:2], 4, 36), H, W, [1, 1], 36,
                      "l1_norm", 1.0)
    small = make_inputs(3, 1, 3, 8, 2, 8, 1, torch.float16, kind="raw")
    with pytest.raises(RuntimeError):      # window does not fit a 3-row map
        match_attention(*(t.cuda() for t in small), 3, 8, 1, 0.25)
    out, _ = match_attention(mo, q, k, v, H, W, 1, 0.25)
    torch.cuda.synchronize()
    assert_close(out, case["ref"][0], torch.float16)


def test_checked_entry_point_finds_no_stray_index():
    """matchattn_fused_forward_checked: the same results as the plain call, and not one index outside its
    array, on the inputs most likely to produce one: centres far outside the map, NaN, infinities, the
    smallest map that fits the window, odd sizes, the any-shape kernel."""
    import matchattention_b200 as ma
    from _cases import make_inputs
    for B, H, W, h, hd, r, dtype in ((2, 33, 29, 8, 16, 1, torch.float16), (1, 4, 4, 2, 16, 1, torch.float32),
                                     (1, 17, 19, 4, 40, 2, torch.bfloat16), (1, 12, 14, 5, 12, 1, torch.float16)):
        mo, q, k, v = (t.cuda() for t in make_inputs(91, B, H, W, h, hd, r, dtype, kind="raw"))
        mo[0, 0, 0, 0] = float("nan")
        mo[0, 1, 0, 1] = float("inf")
        mo[0, 2, :, :] = -60000.0
        out, attn = torch.empty_like(q), q.new_empty(B, H * W, h, (2 * r + 2) ** 2)
        violations, first = ma.ops.launch_checked(mo, q, k, v, out, attn, H, W, r, hd ** -0.5)
        assert (violations, first) == (0, 0)
        want_out, want_attn = ma.match_attention(mo, q, k, v, H, W, r, hd ** -0.5)
        torch.cuda.synchronize()
        same = lambda a, b: torch.equal(torch.nan_to_num(a.float(), nan=7.0), torch.nan_to_num(b.float(), nan=7.0))
        assert same(out, want_out) and same(attn, want_attn)


@pytest.mark.parametrize("around", ["plain", "parameter", "subclass", "device_mode", "dispatch_mode", "inference_mode", "training"])
def test_host_extension_and_python_path_agree(case, around):
    """Ordinary calls are served by the host extension; subclasses and dispatch modes take the Python path."""
    import contextlib
    from torch.utils._python_dispatch import TorchDispatchMode
    from matchattention_b200 import MF_FusedForwardOps, self_attention_core

    class Sub(torch.Tensor):
        pass

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    mo, q, k, v = case["gpu"]
    if around == "parameter":
        q = torch.nn.Parameter(q, requires_grad=False)
    if around == "subclass":
        q = q.as_subclass(Sub)
    if around == "training":
        q = q.clone().requires_grad_(True)
    context = {"device_mode": torch.device("cuda"), "dispatch_mode": Mode(), "inference_mode": torch.inference_mode()}
    with context.get(around, contextlib.nullcontext()):
        out, attn = MF_FusedForwardOps()(mo, q, k, v, case["H"], case["W"], [1, 1], 16, scale=case["scale"])
        own = self_attention_core(mo, q.detach(), k, v, case["H"], case["W"], 1, case["scale"], clamp=False)
    assert_close(out, case["ref"][0], torch.float16)
    assert_close(attn, case["ref"][1], torch.float16)
    assert_close(own, case["ref"][0], torch.float16)
    assert out.requires_grad == (around == "training")


def test_a_torch_function_mode_sees_the_operator(case):
    """A mode (a tracer, a logger) is shown the custom op, as it is for any other operator; the one behind
    torch.set_default_device is not in the way."""
    from torch.overrides import TorchFunctionMode

    from matchattention_b200 import MF_FusedForwardOps

    class Log(TorchFunctionMode):
        seen = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            Log.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    def call():
        return MF_FusedForwardOps()(*case["gpu"], case["H"], case["W"], [case["r"]] * 2, case["M"], attn_type="l1_norm",
                                    scale=case["scale"])

    want = call()
    with Log():
        got = call()
    assert any("fused_forward_ops" in name for name in Log.seen), Log.seen
    with torch.device("cuda"):
        placed = call()
    for a, b, c in zip(want, got, placed):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("train", [False, True])
def test_the_profiler_shows_the_operator(case, train):
    """torch.profiler lists the operator by the custom op's name, with its inputs, in inference and in training."""
    from matchattention_b200 import MF_FusedForwardOps
    inputs = [t.detach().requires_grad_(train) for t in case["gpu"]]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU], record_shapes=True,
                                acc_events=True) as prof:
        MF_FusedForwardOps()(*inputs, case["H"], case["W"], [case["r"]] * 2, case["M"], attn_type="l1_norm", scale=case["scale"])
    events = [e for e in prof.events() if e.name == "matchattn_b200::fused_forward_ops"]
    assert len(events) == 1 and list(events[0].input_shapes[1]) == list(case["gpu"][1].shape)


def test_a_tensor_with_the_negative_bit_stands_for_its_values(case):
    """A lazily negated view (torch keeps a bit instead of new values) gives what the values give, through every entry
    point that takes tensors."""
    import matchattention_b200 as ma
    mo, q, k, v = case["gpu"]
    H, W, r, scale = case["H"], case["W"], case["r"], case["scale"]
    g = torch.Generator(device="cuda").manual_seed(5)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    field, mask, corr, flow = normal(2, 4, 6, 2), normal(2, 36, 4, 6), normal(1, 3, 24, 24), normal(1, 48, 48)
    volume = normal(2, 24, 3, 5).abs()
    for call in (lambda s: ma.match_attention_autograd(mo, s(q), k, v, H, W, r, scale),
                 lambda s: ma.match_attention(mo, q, s(k), v, H, W, r, scale),
                 lambda s: ma.cross_attention_core(mo, q, k, v, s(q), H, W, r, scale),
                 lambda s: ma.self_attention_core(mo, q, k, s(v), H, W, r, scale),
                 lambda s: ma.upsample_field(s(field), s(mask), 2), lambda s: ma.stereo_volume(s(corr)),
                 lambda s: ma.consistency_mask(s(field)), lambda s: ma.local_disparity_estimator(s(volume)),
                 lambda s: ma.flow_init(s(flow), 6, 8)):
        want, got = call(lambda t: -t), call(torch._neg_view)
        for a, b in zip(*((x if isinstance(x, tuple) else (x,)) for x in (want, got))):
            assert torch.equal(a, b)
    leaf = q.detach().requires_grad_(True)
    out, _ = ma.match_attention_autograd(mo, leaf, k, v, H, W, r, scale)
    want, got = (torch.autograd.grad(out, leaf, f(q), retain_graph=True)[0] for f in (torch.neg, torch._neg_view))
    assert torch.equal(want, got)


def test_wrong_arguments_raise_alike_on_every_path(case):
    """What a refused argument raises is the same with and without the native entry (in inference the custom op words it)."""
    from torch.overrides import TorchFunctionMode

    from matchattention_b200 import MF_FusedForwardOps

    class Python(TorchFunctionMode):                # takes calls off the native entry
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    def call(train, win_r=(1, 1), M=16, scale=0.25):
        inputs = [t.detach().requires_grad_(train) for t in case["gpu"]]
        return MF_FusedForwardOps()(*inputs, case["H"], case["W"], win_r, M, attn_type="l1_norm", scale=scale)

    for train in (False, True):
        for error, kwargs in ((ValueError if train else RuntimeError, dict(scale="x")), (TypeError if train else RuntimeError, dict(scale=None)),
                              (RuntimeError, dict(win_r=[-1, -1], M=0))):
            with pytest.raises(error) as native:
                call(train, **kwargs)
            assert not isinstance(native.value, NotImplementedError)
            with Python(), pytest.raises(error):
                call(train, **kwargs)
    with pytest.raises(TypeError):                  # an int is no list of two; the training path takes it
        call(False, win_r=1)
    assert call(True, win_r=1)[0].shape == case["gpu"][1].shape
