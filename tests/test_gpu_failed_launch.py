"""A call that fails on the host (enqueued into a stream capture that has become invalid) reports its error once: the next
call, on a sound stream, succeeds."""
import ctypes

import pytest
import torch

from _cases import make_inputs

pytestmark = pytest.mark.gpu
H, W, B = 24, 26, 2
CAPTURE_THREAD_LOCAL = 1


def _entry_points():
    """name -> call(stream) through the C ABI; the tensors live as long as the returned dict."""
    from matchattention_b200 import _lib
    lib, calls = _lib.lib, {}

    def plain(entry, *args, behind=()):
        return lambda stream: entry(*[x.data_ptr() if torch.is_tensor(x) else x for x in args], stream,
                                    *[x.data_ptr() if torch.is_tensor(x) else x for x in behind])

    def operator(h, hd, r, dtype, code, entry=lib.matchattn_fused_forward, before=(), behind=()):
        """`before`, `behind`: further arguments on either side of the stream."""
        t = [x.cuda() for x in make_inputs(5, B, H, W, h, hd, r, dtype, kind="self")]
        out, attn = torch.empty_like(t[1]), torch.empty(B, H * W, h, (2 * r + 2) ** 2, dtype=dtype, device="cuda")
        shape = (B, H, W, h, hd, r, r, code, _lib.L1_NORM, hd ** -0.5, 0, H)
        return plain(entry, *t, out, attn, *shape, *before, behind=behind)

    def backward(gathered):
        h, hd, r = 4, 32, 1
        mo, q, k, v = (x.cuda() for x in make_inputs(6, B, H, W, h, hd, r, torch.float32, kind="self"))
        grads = [torch.empty_like(x) for x in (q, k, v, mo)]
        size = lib.matchattn_backward_workspace_bytes(B, H, W, h, hd, r, _lib.F32, 0, H)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        args = (mo, q, k, v, q, None, *grads, B, H, W, h, hd, r, r, _lib.F32, _lib.L1_NORM, hd ** -0.5, 0, H)
        return plain(lib.matchattn_fused_backward_ws, *args, ws, size) if gathered else plain(lib.matchattn_fused_backward, *args)

    half = torch.float16
    calls["heads on lanes"] = operator(4, 16, 1, torch.float32, _lib.F32)
    calls["heads on lanes, r = 2"] = operator(4, 40, 2, half, _lib.F16)
    calls["a head per lane"] = operator(4, 16, 1, half, _lib.F16)
    calls["any shape"] = operator(4, 12, 1, torch.float32, _lib.F32)
    calls["checked"] = operator(4, 16, 1, half, _lib.F16, lib.matchattn_fused_forward_checked,
                                before=(torch.zeros(2, dtype=torch.int64, device="cuda"),))
    binned = lib.matchattn_workspace_bytes(B, H, W, 4, 16, 1, _lib.F16, 0, H)
    for name, strategy in (("binned", 2), ("staged", 5), ("staged blocks", 6)):
        calls[name] = operator(4, 16, 1, half, _lib.F16, lib.matchattn_fused_forward_ws,
                               behind=(torch.empty(binned, dtype=torch.uint8, device="cuda"), binned, strategy))
    calls["backward, gathered"], calls["backward, accumulating"] = backward(True), backward(False)
    field, mask = torch.randn(B, H, W, 2, device="cuda", dtype=half), torch.randn(B, 36, H, W, device="cuda", dtype=half)
    calls["upsampling"] = plain(lib.matchattn_upsample_field, field, mask, field.new_empty(B, 2 * H, 2 * W, 2), B, H, W, 2, 2, _lib.F16)
    corr, vol = torch.randn(1, H, W, W, device="cuda", dtype=half), torch.empty(2, W, H, W, device="cuda", dtype=half)
    calls["stereo volume"] = plain(lib.matchattn_stereo_volume, corr, vol, 1, H, W, _lib.F16)
    wide = torch.empty(2, 150, H, 150, device="cuda")
    calls["stereo volume, large shared memory"] = plain(lib.matchattn_stereo_volume, torch.randn(1, H, 150, 150, device="cuda"), wide, 1,
                                                        H, 150, _lib.F32)
    calls["disparity"] = plain(lib.matchattn_local_disparity, vol.abs(), field, None, None, 2, W, H, W, _lib.F16)
    calls["mask"] = plain(lib.matchattn_consistency_mask, field, field.new_empty(B, H, W, 1), None, B, H, W, 2.0, _lib.F16)
    N, size = H * W, lib.matchattn_flow_init_scratch_bytes(1, H, W)
    pairs, scratch = torch.randn(1, N, N, device="cuda", dtype=half), torch.empty(size, dtype=torch.uint8, device="cuda")
    calls["flow_init"] = plain(lib.matchattn_flow_init, pairs, torch.empty(2, N, N, device="cuda", dtype=half), torch.empty_like(field), None,
                               None, scratch, size, 1, H, W, _lib.F16)
    words = (ctypes.c_void_p * 1)(field.data_ptr()), (ctypes.c_void_p * 1)(mask.data_ptr()), (ctypes.c_size_t * 1)(64)
    calls["copy"] = lambda stream: lib.matchattn_copy_blocks(*words, 1, 0, stream)
    calls["copy kernel"] = lambda stream: lib.matchattn_copy_blocks(*words, 1, 1, stream)
    return calls


def test_a_failed_call_leaves_no_error_for_the_next_one():
    calls = _entry_points()
    cuda = ctypes.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    handle, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    for name, call in calls.items():
        assert call(stream.cuda_stream) == 0, name
    stream.synchronize()
    left = {}
    for name, call in calls.items():
        assert cuda.cuStreamBeginCapture_v2(handle, CAPTURE_THREAD_LOCAL) == 0
        try:
            assert cuda.cuStreamSynchronize(handle) != 0           # not allowed in a capture, which is invalid from here on
            failed = call(stream.cuda_stream)
        finally:
            cuda.cuStreamEndCapture(handle, ctypes.byref(graph))
        assert failed > 100, name                                  # MATCHATTN_ERR_CUDA + the runtime's code
        after = calls["mask"](stream.cuda_stream)
        if after != 0:
            left[name] = after
            assert calls["mask"](stream.cuda_stream) == 0          # (reading the error has cleared it)
    stream.synchronize()
    assert not left
