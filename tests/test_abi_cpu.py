"""CPU tests of the boundary: the shared library loads, exports every symbol the
header declares, validates arguments before touching a device, and the Python
host layer refuses CPU tensors.  No kernel is launched here."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "matchattn.h")).read()
    return sorted(set(re.findall(r"MATCHATTN_API\s+[\w\s\*]+?\b(matchattn_\w+)\s*\(", text)))


def test_header_and_binding_list_the_same_symbols():
    from matchattention_b200 import _lib
    assert declared_symbols() == sorted(_lib.EXPORTS)


def test_library_exports_every_declared_symbol():
    from matchattention_b200 import _lib
    lib = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared_symbols():
        assert hasattr(lib, name), name
    assert _lib.lib.matchattn_version() >= 100
    assert _lib.strerror(0) == "ok"


def test_arguments_are_rejected_on_the_host():
    """Every one of these returns before any CUDA call, so they run without a GPU."""
    from matchattention_b200 import _lib
    f = _lib.lib.matchattn_fused_forward
    p = ctypes.c_void_p(4096)   # never dereferenced

    def call(mo=p, q=p, k=p, v=p, out=p, attn=p, B=1, H=8, W=8, h=2, hd=16, rx=1, ry=1, dtype=1, attn_type=0,
             scale=1.0, r0=0, r1=8):
        return f(mo, q, k, v, out, attn, B, H, W, h, hd, rx, ry, dtype, attn_type, scale, r0, r1, None)

    assert call(q=None) == 1
    assert call(B=0) == 2 and call(r0=5, r1=5) == 2 and call(r1=9) == 2
    assert call(H=3, r1=3) == 3
    assert call(dtype=7) == 4
    assert call(attn_type=2) == 5
    assert call(rx=1, ry=2) == 6 and call(rx=5, ry=5, H=32, W=32, r1=32) == 6
    assert call(q=ctypes.c_void_p(4097)) == 7
    assert call(B=70000) == 8
    for code in (1, 2, 3, 4, 5, 6, 7, 8):
        assert _lib.strerror(code) not in ("ok", "unknown status")


def test_block_copy_arguments_are_checked_on_the_host():
    """matchattn_copy_blocks: an empty list is fine, a negative count or a missing array or pointer is
    refused before any CUDA call."""
    from matchattention_b200 import _lib
    f = _lib.lib.matchattn_copy_blocks
    none = ctypes.POINTER(ctypes.c_void_p)()
    assert f(none, none, ctypes.POINTER(ctypes.c_size_t)(), 0, 0, None) == 0
    assert f(none, none, ctypes.POINTER(ctypes.c_size_t)(), -1, 0, None) == 1
    assert f(none, none, ctypes.POINTER(ctypes.c_size_t)(), 2, 1, None) == 1
    dst, src = (ctypes.c_void_p * 2)(4096, None), (ctypes.c_void_p * 2)(8192, 8192)
    sizes = (ctypes.c_size_t * 2)(0, 64)              # the first block is empty and skipped, the second lacks a target
    assert f(dst, src, sizes, 2, 0, None) == 1


def test_backward_alignment_is_checked_on_the_host():
    """Both backward entry points refuse arrays that their kernels cannot read, before any CUDA call: an element that
    straddles its size (7), and for the one with a workspace a centre that straddles its pair (9: the other one serves)."""
    from matchattention_b200 import _lib
    at = ctypes.c_void_p
    sizes = (1, 8, 8, 2, 16, 1, 1)

    def ws(dtype, mo=4096, **moved):
        a = [moved.get(n, 4096) for n in ("q", "k", "v", "d_out", "d_attn", "d_q", "d_k", "d_v", "d_mo")]
        return _lib.lib.matchattn_fused_backward_ws(at(mo), *map(at, a), *sizes, dtype, 0, 0.25, 0, 8, at(4096), 1 << 30, None)

    def scattered(dtype, mo=4096, **moved):
        a = [moved.get(n, 4096) for n in ("q", "k", "v", "d_out", "d_attn", "d_q", "d_k", "d_v", "d_mo")]
        return _lib.lib.matchattn_fused_backward(at(mo), *map(at, a), *sizes, dtype, 0, 0.25, 0, 8, None)

    for dtype, esize in ((_lib.F32, 4), (_lib.F16, 2), (_lib.BF16, 2)):
        assert ws(dtype, mo=4096 + esize) == 9
        assert ws(dtype, q=4096 + 16) == 9
        for call in (ws, scattered):
            assert call(dtype, mo=4097) == 7 and call(dtype, d_attn=4096 + esize // 2) == 7 and call(dtype, d_mo=4097) == 7
        assert scattered(dtype, d_k=4098) == 7
    assert "not aligned" in _lib.strerror(7) and "variant" in _lib.strerror(9)


def test_dispatch_table():
    from matchattention_b200 import describe_dispatch
    assert describe_dispatch(8, 16, 1, torch.float16) == "fast cpl=2 lph=1"
    assert describe_dispatch(8, 16, 1, torch.float16, aligned32=False) == "generic"
    assert describe_dispatch(4, 8, 1, torch.float16, aligned32=False) == "fast cpl=1 lph=1"
    assert describe_dispatch(8, 16, 1, torch.float32) == "fast cpl=1 lph=2"
    assert describe_dispatch(4, 64, 1, torch.float16) == "fast cpl=2 lph=4"
    assert describe_dispatch(4, 128, 1, torch.float32) == "fast cpl=2 lph=8"
    # 40 channels: two lanes (a 32-byte piece each and one of 16 bytes) where every row starts 32-byte aligned
    assert describe_dispatch(4, 40, 2, torch.bfloat16) == "fast cpl=3 lph=2"
    assert describe_dispatch(4, 40, 2, torch.bfloat16, aligned32=False) == "fast cpl=5 lph=1"
    assert describe_dispatch(3, 40, 2, torch.bfloat16) == "fast cpl=5 lph=1"
    assert describe_dispatch(40, 64, 2, torch.float32) == "fast cpl=2 lph=4"          # 320 lanes of the finer split do not fit a block
    assert describe_dispatch(4, 12, 1, torch.float32) == "generic"
    assert describe_dispatch(4, 16, 3, torch.float32) == "generic"


def test_cpu_tensors_are_refused():
    from matchattention_b200 import match_attention
    t = torch.zeros(1, 64, 16)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        match_attention(torch.zeros(1, 64, 2, 2), t, t, t, 8, 8, 1, 1.0)


def test_a_training_step_has_its_profiler_range(monkeypatch):
    """MATCHATTN_B200_NVTX: the autograd entry point opens and closes a range around the native call, also when it raises."""
    import types

    from matchattention_b200 import ops
    seen = []
    mo, t = torch.zeros(1, 64, 2, 2), torch.zeros(1, 64, 16)

    def native(*args):
        seen.append("call")
        if len(seen) > 3:
            raise RuntimeError("refused")
        return t, t

    monkeypatch.setattr(ops, "_NVTX", True)
    monkeypatch.setattr(ops, "_host", types.SimpleNamespace(autograd=native))
    monkeypatch.setattr(torch.cuda.nvtx, "range_push", seen.append)
    monkeypatch.setattr(torch.cuda.nvtx, "range_pop", lambda: seen.append("end"))
    ops.match_attention_autograd(mo, t, t, t, 8, 8, 1, 0.25)
    assert seen == ["matchattn_b200 B1 8x8 h2x8 r1 float32", "call", "end"]
    with pytest.raises(RuntimeError, match="refused"):
        ops.match_attention_autograd(mo, t, t, t, 8, 8, 1, 0.25)
    assert seen[-1] == "end"


def test_the_host_extension_belongs_to_one_python_and_torch(monkeypatch):
    """After an upgrade of torch (or Python) the old extension is neither taken for current by the build nor loaded."""
    from matchattention_b200 import _lib, build
    assert _lib.host.__file__ == build.host_path()
    monkeypatch.setattr(torch, "__version__", "99.0.0")
    assert build._host_stale()
    with pytest.raises(ImportError, match="99.0.0.*build it"):
        _lib._load_host()
    monkeypatch.undo()
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name: "cpython-399")
    assert build._host_stale()
