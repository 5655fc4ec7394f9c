"""Tiles over chains without branches (pruned tries with long repeats): forward and backward against a dense float64 reference, with chain lengths around the
tile sizes and what is left of them, and launch groups made per radix edge against the char-level path."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import trainer as T
from tests.helpers import TOL_F32, rel_err
from tests.test_run_groups_gpu import _same

pytestmark = pytest.mark.gpu


def _comb(lengths, stem):
    """A stem of `stem` rows, and on its last row a chain of each length."""
    parent = list(range(-1, stem - 1))
    for n in lengths:
        at = len(parent)
        parent += [stem - 1] + list(range(at, at + n - 1))
    return np.array(parent, np.int32)


def _dense(plan, q, k, v, do, heads):
    import torch
    n, d = q.shape
    hd = d // heads
    sub = torch.from_numpy(np.asarray(plan.sub_end).astype(np.int64)).to(q.device)
    i = torch.arange(n, device=q.device)
    mask = (i[None, :] <= i[:, None]) & (i[:, None] < sub[None, :])
    t = [x.double().view(n, heads, hd).transpose(0, 1).requires_grad_() for x in (q, k, v)]
    s = (t[0] @ t[1].transpose(1, 2) / hd ** 0.5).masked_fill(~mask, -np.inf)
    o = torch.softmax(s, -1) @ t[2]
    o.backward(do.double().view(n, heads, hd).transpose(0, 1))
    return [x.transpose(0, 1).reshape(n, d).cpu().numpy() for x in (o.detach(), t[0].grad, t[1].grad, t[2].grad)]


@pytest.mark.parametrize("lengths,stem", [([64, 64, 1], 1), ([65, 65, 2], 1), ([95, 96, 97], 3), ([127, 128, 129, 5], 2), ([160, 33, 191, 193], 40), ([300], 7), ([66, 31, 32, 66, 64], 31)])
def test_chains_against_dense_attention(cuda, lengths, stem):
    import torch
    plan = A.WalkerPlan(_comb(lengths, stem), 64, 0)
    g = torch.Generator(device="cuda").manual_seed(sum(lengths))
    for heads, hd in ((2, 16), (1, 32), (1, 64)):
        q, k, v, do = [torch.randn(plan.n, heads * hd, device=cuda, generator=g) for _ in range(4)]
        o, lse = A.attn_forward(plan, q, k, v, heads)
        got = (o,) + tuple(A.attn_backward(plan, q, k, v, o, lse, do, heads))
        for name, a, b in zip(("out", "dq", "dk", "dv"), got, _dense(plan, q, k, v, do, heads)):
            assert rel_err(a.cpu().numpy(), b) < TOL_F32, (name, heads, hd)


@pytest.mark.parametrize("chars,depth,rows", [(1500, 128, 1 << 30), (1500, 70, 9000)])
def test_groups_over_chains_equal_the_char_level_path(chars, depth, rows):
    import torch
    trie = A.RadixTrie.build(A.synth_markov_corpus(chars, 96, 4, 0, 10), depth, 1, 2, 4)
    got, _ = T.build_groups(trie, 0, 1, rows, "log", 128, torch.device("cuda", 0))
    want, _ = T.build_groups(trie, 0, 1, rows, "log", 128, torch.device("cpu"))
    assert len(got) == len(want) and max(g.plan.max_depth for g in got) > 60
    for a, b in zip(got, want):
        _same(a, b)
