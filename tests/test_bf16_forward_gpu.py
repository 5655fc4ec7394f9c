"""Attention forward on a bfloat16 K/V store: float64 attention over the rounded rows, at the edges of the 64-row tiles and of the 16-key
blocks, and on both sides of the rule that sends deep plans to the chunked kernel."""
import numpy as np
import pytest

import agpt_b200 as A
from tests.helpers import chain_tree, random_qkv, random_tree, rel_err

pytestmark = pytest.mark.gpu


def _want(parent, q, k, v, H):
    n, D = q.shape
    hd = D // H
    out, lse = np.zeros((n, D)), np.zeros((n, H))
    for i in range(n):
        keys, a = [], i
        while a >= 0:
            keys.append(a)
            a = parent[a]
        for h in range(H):
            c = slice(h * hd, (h + 1) * hd)
            s = k[keys, c].astype(np.float64) @ q[i, c] / np.sqrt(hd)
            m = s.max()
            e = np.exp(s - m)
            out[i, c], lse[i, h] = e @ v[keys, c] / e.sum(), m + np.log(e.sum())
    return out, lse


@pytest.mark.parametrize("parent,H,hd,tol", [
    (chain_tree(1), 1, 16, 5e-5), (chain_tree(15), 2, 32, 5e-5), (chain_tree(65), 1, 64, 5e-5),
    (random_tree(64, 9, 1), 3, 16, 5e-5), (random_tree(333, 32, 2), 2, 32, 5e-5), (random_tree(400, 100, 3, 0.1), 2, 64, 5e-5),
    (chain_tree(440), 1, 16, 5e-5), (chain_tree(448), 1, 32, 5e-5), (chain_tree(432), 1, 64, 5e-5),
    (chain_tree(440), 1, 64, 2e-3),                      # chunked: one TF32 product
])
def test_bf16_store_forward(parent, H, hd, tol):
    import torch
    n = len(parent)
    plan = A.WalkerPlan(parent, 64, 0)
    q, k, v, _ = [torch.from_numpy(x).cuda() for x in random_qkv(n, H * hd, n)]
    q *= 3.0
    out, lse = A.attn_forward(plan, q, k.bfloat16(), v.bfloat16(), H)
    want_o, want_l = _want(np.asarray(plan.parent_dfs), q.cpu().numpy(), k.bfloat16().float().cpu().numpy(), v.bfloat16().float().cpu().numpy(), H)
    assert rel_err(out.cpu().numpy(), want_o) < tol and rel_err(lse.cpu().numpy(), want_l) < tol
