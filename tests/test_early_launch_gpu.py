"""Kernels whose blocks are placed while the kernel in front still works (csrc/pdl.cuh) give what they give one at a time.

Chains of entry points run back to back on one stream, without a wait between them, and again with a device-wide wait after each: every output
is the same bit for bit.  Sizes lie on both sides of the rules that choose the launch (rows x columns) and of the last partial tile."""
import numpy as np
import pytest

import agpt_b200 as A

pytestmark = pytest.mark.gpu


def _chain(cuda, n, heads, head_dim, wait):
    import torch
    torch.manual_seed(n)
    d = heads * head_dim
    plan = A.WalkerPlan(A.synth_tree(n, 64, 17, 0.35, 65, 1000, 3), 64, 0)
    q, k, v, g = [torch.randn(plan.n, d, device=cuda) for _ in range(4)]
    out = []
    for _ in range(4):                  # each pass reads what the one before wrote
        o, lse = A.attn_forward(plan, q, k, v, heads)
        if wait:
            torch.cuda.synchronize()
        dq, dk, dv = A.attn_backward(plan, q, k, v, o, lse, g, heads)
        if wait:
            torch.cuda.synchronize()
        out += [o, lse, dq, dk, dv]
        q, k, v = o, dk, dv
        if wait:
            torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("n,heads,head_dim", [(1, 4, 16), (63, 4, 32), (700, 8, 64), (9000, 4, 32), (70_000, 8, 64)])
def test_attention_chain(cuda, n, heads, head_dim):
    for a, b in zip(_chain(cuda, n, heads, head_dim, False), _chain(cuda, n, heads, head_dim, True)):
        np.testing.assert_array_equal(a, b)


def test_attention_chain_in_a_graph(cuda):
    """The early launches are captured, and a replay gives what the calls give."""
    import torch
    plan = A.WalkerPlan(A.synth_tree(3000, 64, 17, 0.35, 65, 1000, 3), 64, 0)
    q, k, v, g = [torch.randn(plan.n, 128, device=cuda) for _ in range(4)]

    def step():
        o, lse = A.attn_forward(plan, q, k, v, 4)
        return (o, lse) + tuple(A.attn_backward(plan, q, k, v, o, lse, g, 4))
    want = [t.clone() for t in step()]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for _ in range(3):
        for t in got:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
