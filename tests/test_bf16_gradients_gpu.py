"""Attention gradients on a bfloat16 K/V store against float64 attention over the rounded rows, for each pair of kernels that a forward and a
backward of one plan can be: whole tiles in both directions; the whole-tile forward, whose lse comes of 16 bits of Q, before the chunked
backward, which rounds Q, P and dS to 11 (its P then sum to one but for that difference); chunked in both directions (even tiles)."""
import numpy as np
import pytest

import agpt_b200 as A
from tests.helpers import chain_tree, random_qkv, random_tree

pytestmark = pytest.mark.gpu


def _want(parent, q, k, v, go, H):
    import torch
    n, D = q.shape
    hd = D // H
    mask = torch.zeros(n, n, dtype=torch.bool)
    for i in range(n):
        a = i
        while a >= 0:
            mask[i, a] = True
            a = int(parent[a])
    q, k, v = [torch.from_numpy(x).double().view(n, H, hd).requires_grad_(True) for x in (q, k, v)]
    s = torch.einsum("ihd,jhd->hij", q, k) / np.sqrt(hd)
    p = torch.softmax(s.masked_fill(~mask[None], float("-inf")), dim=-1)
    torch.einsum("hij,jhd->ihd", p, v).backward(torch.from_numpy(go).double().view(n, H, hd))
    return [x.grad.reshape(n, D).numpy() for x in (q, k, v)]


def errors(parent, H, hd, even):
    """Relative 2-norm errors of dq, dk, dv."""
    import torch
    plan = A.WalkerPlan(parent, 64, 0, even=even)
    n = len(parent)
    q, k, v, go = random_qkv(n, H * hd, n)
    k, v = [torch.from_numpy(x).bfloat16() for x in (k, v)]
    tq, tg = torch.from_numpy(q).cuda(), torch.from_numpy(go).cuda()
    out, lse = A.attn_forward(plan, tq, k.cuda(), v.cuda(), H)
    got = A.attn_backward(plan, tq, k.cuda(), v.cuda(), out, lse, tg, H)
    want = _want(plan.parent_dfs, q, k.float().numpy(), v.float().numpy(), go, H)
    return [float(np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b)) for a, b in zip(got, want)]


# K and V are exact; each factor rounded to 11 bits adds at most 2^-12 relative to a product, 2^-12 / sqrt(3) in the mean, and a gradient is a
# sum of products of one to three of them (S once more in the exponent, scaled by |S| of about one here): 5e-4.  With 16 bits 2^-5 of that.
@pytest.mark.parametrize("parent,H,hd,even,tol", [
    (random_tree(333, 30, 2), 2, 16, False, 2e-5), (random_tree(333, 30, 2), 2, 32, False, 2e-5), (random_tree(333, 30, 2), 2, 64, False, 2e-5),
    (chain_tree(230), 1, 64, False, 5e-4), (random_tree(600, 120, 3, 0.1), 3, 64, False, 5e-4),
    (chain_tree(230), 1, 64, True, 5e-4), (random_tree(600, 120, 3, 0.1), 3, 64, True, 5e-4), (random_tree(333, 30, 2), 2, 32, True, 5e-4),
    (random_tree(333, 30, 2), 2, 16, True, 5e-4),
])
def test_bf16_store_gradients(parent, H, hd, even, tol):
    got = errors(parent, H, hd, even)
    print(got)
    assert max(got) < tol
