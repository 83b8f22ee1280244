"""Kernels set up while the one before them drains still see everything that came before them in the stream, and leave
nothing unfinished for what comes after: inputs rewritten in place between calls, on one stream, on two, and in a graph."""
import pytest
import torch

import matchattention_b200 as ma
from _cases import make_inputs

pytestmark = pytest.mark.gpu


def _sources(H, W, dtype):
    """Two sets of inputs: operator operands and a stereo correlation."""
    sets = []
    for seed in (1, 2):
        mo, q, k, v = (t.cuda() for t in make_inputs(seed, 2, H, W, 4, 32, 1, dtype, kind="flow", spread=6.0))
        g = torch.Generator(device="cuda").manual_seed(seed)
        corr = (torch.randn(2, H, W, W, generator=g, device="cuda") * 4).to(dtype)
        sets.append((mo, q, k, v, corr))
    return sets


def _chain(mo, q, k, v, corr, H, W):
    """Every kernel reads what the one before it wrote."""
    out, _ = ma.MF_FusedForwardOps()(mo, q, k, v, H, W, [1, 1], 16, attn_type="l1_norm", scale=32 ** -0.5)
    again, attn = ma.MF_FusedForwardOps()(mo, out, k, out, H, W, [1, 1], 16, attn_type="l1_norm", scale=32 ** -0.5)
    volume = ma.stereo_volume(corr)
    field = ma.local_disparity_estimator(volume)
    return again, attn, field, ma.consistency_mask(field)


@pytest.mark.parametrize("how", ["one stream", "two streams", "graph"])
@pytest.mark.parametrize("H,W,dtype", [(6, 7, torch.float32), (61, 83, torch.float16)])
def test_calls_in_a_row_keep_their_order(H, W, dtype, how):
    sets = _sources(H, W, dtype)
    expected = []
    for s in sets:
        expected.append([t.clone() for t in _chain(*s, H, W)])
        torch.cuda.synchronize()
    held = [t.clone() for t in sets[0]]

    def load(i):
        for dst, src in zip(held, sets[i]):
            dst.copy_(src)

    results = []
    if how == "graph":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _chain(*held, H, W)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            kept = _chain(*held, H, W)
        for i in range(8):
            load(i % 2)
            graph.replay()
            results.append([t.clone() for t in kept])
    elif how == "two streams":
        other = torch.cuda.Stream()
        for i in range(8):
            load(i % 2)                                   # on this stream, the calls on the other
            other.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(other):
                results.append(_chain(*held, H, W))
            torch.cuda.current_stream().wait_stream(other)
    else:
        for i in range(8):
            load(i % 2)
            results.append(_chain(*held, H, W))
    torch.cuda.synchronize()
    for i, got in enumerate(results):
        for a, b in zip(got, expected[i % 2]):
            assert torch.equal(a, b)
