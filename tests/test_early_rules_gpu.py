"""Which calls place their kernels while the kernel in front still works: read off the edges of a captured graph."""
import numpy as np
import pytest

import agpt_b200 as A

pytestmark = pytest.mark.gpu


def _early(call):
    """Edges of the graph of two calls in a row that let the second kernel be placed early, and all of its edges."""
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
        call()
    handle = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, _, _, n = rt.cudaGraphGetEdges_v2(handle)
    assert err == 0
    err, _, _, data, n = rt.cudaGraphGetEdges_v2(handle, n)
    assert err == 0 and len(data) == n > 0
    return sum(int(e.type) == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for e in data), n


@pytest.mark.parametrize("n,early", [(1 << 19, True), ((1 << 19) + 64, False)])
def test_attention_entry_points_follow_one_rule(cuda, n, early):
    """Up to 32 Mi row elements, in every form of the call."""
    import torch
    plan = A.WalkerPlan(np.full(n, -1, np.int32), 64, 0)          # no chains: the backward without a workspace takes it
    q, k, v, g = [torch.randn(n, 64, device=cuda) for _ in range(4)]
    o, lse = A.attn_forward(plan, q, k, v, 4)
    d = [torch.empty_like(q) for _ in range(3)]
    ws = torch.empty(max(plan.workspace_bytes(64), 1), dtype=torch.uint8, device=cuda)
    for call in (lambda: A.attn_forward(plan, q, k, v, 4, out=o, lse=lse),
                 lambda: A.attn_backward(plan, q, k, v, o, lse, g, 4, workspace=ws, dq=d[0], dk=d[1], dv=d[2]),
                 lambda: A.attn_backward_static(plan, q, k, v, o, lse, g, 4, *d)):
        got, edges = _early(call)
        assert got == (edges if early else 0)
