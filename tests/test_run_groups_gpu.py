"""Launch groups made per radix edge on the GPU against the char-level path (char_tree, WalkerPlan, launch_groups): every array
the training step or the attention reads, for both unit levels, cut units, several ranks, pruned tries and sampled units."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import trainer as T

pytestmark = pytest.mark.gpu
NAMES = ("tokens", "tokens32", "pos", "unit_of_row", "unit_off", "q2n", "qoff", "rid", "edge_first", "mass_w", "trained")
PLAN = ("dfs_to_node", "node_to_dfs", "parent_dfs", "depth", "sub_end")
SIZES = ("n", "n_tiles", "chain_rows", "max_depth", "sum_depth", "sum_group_prefix", "n_groups", "bwd_launches")


def _same(got, want):
    assert (got.n, got.n_units, got.n_pos, got.n_trained_rows) == (want.n, want.n_units, want.n_pos, want.n_trained_rows)
    for k in NAMES:
        a, b = getattr(got, k), getattr(want, k)
        assert (a is None) == (b is None), k
        if a is not None:
            assert a.dtype == b.dtype and np.array_equal(a.cpu().numpy(), b.cpu().numpy()), k
    for k in PLAN:
        assert np.array_equal(getattr(got.plan, k), getattr(want.plan, k)), k
    # the device's chains and reduction list, through an attention backward
    import torch
    g = torch.Generator(device="cuda").manual_seed(got.n)
    q, k, v, do = [torch.randn(got.n, 64, device="cuda", generator=g) for _ in range(4)]
    dev = A.WalkerPlan(want.plan.parent_dfs, want.plan.tile_m, 0)
    for name in SIZES:
        assert getattr(got.plan, name) == getattr(dev, name), name
    for name in ("n_reduce_items", "n_reduce_nodes", "n_reduce_multi"):
        assert getattr(got.plan.info, name) == getattr(dev.info, name), name
    res = []
    for p in (got.plan, dev):
        o, lse = A.attn_forward(p, q, k, v, 4)
        res.append((o, lse) + A.attn_backward(p, q, k, v, o, lse, do, 4))
    assert all(torch.equal(x, y) for x, y in zip(*res))


@pytest.mark.parametrize("chars,vocab,depth,prune,level,cap,world,rows", [
    (40, 3, 5, (1, 4), 1, None, 1, 1000),                # one small group
    (3000, 12, 9, (1, 4), 1, None, 1, 2000),             # several groups
    (3000, 12, 9, (1, 4), 2, None, 3, 900),              # bigram units with context rows over three ranks
    (3000, 12, 9, (1, 4), 2, 40, 2, 700),                # units cut deeper
    (4000, 6, 24, (3, 2), 1, 100, 1, 5000),              # pruned: unary chains run over several edges
    (20000, 20, 16, (1, 4), 1, None, 1, 1 << 30),        # reductions cut into several segments
])
def test_groups_equal_the_char_level_path(chars, vocab, depth, prune, level, cap, world, rows):
    import torch
    trie = A.RadixTrie.build(A.synth_markov_corpus(chars, vocab, 2, 7), depth, level, *prune)
    for rank in range(world):
        got, n = T.build_groups(trie, rank, world, rows, "log", 16, torch.device("cuda", 0), level=level, unit_cap=cap)
        want, m = T.build_groups(trie, rank, world, rows, "log", 16, torch.device("cpu"), level=level, unit_cap=cap)
        assert n == m and len(got) == len(want)
        for a, b in zip(got, want):
            _same(a, b)


def test_sampled_groups_equal_the_char_level_path():
    import torch
    trie = A.RadixTrie.build(A.synth_markov_corpus(2500, 9, 2, 3), 10)
    space = T.SampleSpace(trie)
    for sampler in (1, 2, 3, 4):
        _, na, off, _, nodes, _ = trie.lightning_sample(sampler, 4, 77 + sampler)
        for s in range(4):
            ids = nodes[off[s]:off[s + 1]]
            for ctx in ([], ids[:1]):
                _same(space.group(ids, ctx, "linear", 32, torch.device("cuda", 0)), space.group(ids, ctx, "linear", 32, torch.device("cpu")))
    with pytest.raises(ValueError):
        space.group(nodes[off[3] + 1:off[4]], [], "off", 32, torch.device("cuda", 0))
