"""Kernels set up while the one before them drains still see everything that came before them in the stream, and leave
nothing unfinished for what comes after: inputs rewritten in place between calls, on one stream, on two, and in a graph."""
import pytest
import torch

import matchattention_b200 as ma
from _cases import make_inputs

pytestmark = pytest.mark.gpu


def _sources(H, W, dtype):
    """Two sets of inputs: operator operands, gradients of the outputs, a stereo and an all-pairs correlation, mask logits."""
    sets = []
    for seed in (1, 2):
        mo, q, k, v = (t.cuda() for t in make_inputs(seed, 2, H, W, 4, 32, 1, dtype, kind="flow", spread=6.0))
        g = torch.Generator(device="cuda").manual_seed(seed)

        def normal(*shape, scale=1.0):
            return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)

        sets.append((mo, q, k, v, normal(2, H, W, W, scale=4.0), normal(1, H * W, H * W, scale=4.0), normal(4, 36, H, W),
                     normal(*q.shape), normal(2, H * W, 4, 16)))
    return sets


def _chain(mo, q, k, v, corr, pairs, logits, g_out, g_attn, H, W):
    """Outputs of calls in a row, (exact, summed in any order).  The second operator call, the disparity, the mask and the
    upsampling read what the call before them wrote; the kernels of flow_init and of the backward what the one before them
    wrote to scratch memory, which the next pass of this chain writes again."""
    op = ma.MF_FusedForwardOps()
    out, _ = op(mo, q, k, v, H, W, [1, 1], 16, attn_type="l1_norm", scale=32 ** -0.5)
    again, attn = op(mo, out, k, out, H, W, [1, 1], 16, attn_type="l1_norm", scale=32 ** -0.5)
    volume = ma.stereo_volume(corr)
    field = ma.local_disparity_estimator(volume)
    mask = ma.consistency_mask(field)
    fine = ma.upsample_field(field, logits, 2)
    flow, prob = ma.flow_init(pairs, H, W)
    inputs = [t.detach().requires_grad_(True) for t in (mo, q, k, v)]
    results = op(*inputs, H, W, [1, 1], 16, attn_type="l1_norm", scale=32 ** -0.5)
    d_mo, d_q, d_k, d_v = torch.autograd.grad(results, inputs, (g_out, g_attn))
    return (again, attn, field, mask, fine, flow, prob, d_mo, d_q), (d_k, d_v)


@pytest.mark.parametrize("how", ["one stream", "two streams", "graph"])
@pytest.mark.parametrize("H,W,dtype", [(6, 7, torch.float32), (61, 83, torch.float16)])
def test_calls_in_a_row_keep_their_order(H, W, dtype, how):
    sets = _sources(H, W, dtype)
    expected = []
    for s in sets:
        expected.append([[t.clone() for t in part] for part in _chain(*s, H, W)])
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
            results.append([[t.clone() for t in part] for part in kept])
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
    tol = {torch.float32: 2e-5, torch.float16: 2e-3}[dtype]
    for i, (exact, summed) in enumerate(results):
        for a, b in zip(exact, expected[i % 2][0]):
            assert torch.equal(a, b)
        # token sums: the same float32 terms in the order in which the queries took their places, rounded once
        for a, b in zip(summed, expected[i % 2][1]):
            assert (a.double() - b.double()).abs().max() <= tol * b.double().abs().max()
