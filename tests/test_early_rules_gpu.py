"""Which calls place their kernels while the kernel in front still works: read off the edges of a captured graph."""
import ctypes as C

import numpy as np
import pytest

import agpt_b200 as A

pytestmark = pytest.mark.gpu


def _early(call):
    """Edges of the graph of two calls in a row that let the second kernel be placed early, and all of its edges."""
    import torch
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
        call()
    driver, handle, n = C.CDLL("libcuda.so.1"), C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    assert driver.cuGraphGetEdges_v2(handle, None, None, None, C.byref(n)) == 0 and n.value > 0
    ends, data = [(C.c_void_p * n.value)() for _ in range(2)], (C.c_uint8 * (8 * n.value))()       # data: {from port, to port, type, 5 bytes} per edge
    assert driver.cuGraphGetEdges_v2(handle, ends[0], ends[1], data, C.byref(n)) == 0
    return sum(data[8 * i + 2] == 1 for i in range(n.value)), n.value                              # 1: programmatic


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


@pytest.mark.parametrize("n", [1000, 1 << 20])
def test_optimizer_launches_in_the_ordinary_way(cuda, n):
    import torch
    p, g, m, v = [torch.rand(n, device=cuda) for _ in range(4)]
    got, edges = _early(lambda: A.optimizer_step("adam", p, g, m, v, lr=1e-4, t=3, clip_norm=1.0))
    assert got == 0 and edges == 3
