"""Plans with even tiles: tiles, reduction over more than 128 tiles of a node, both stores and every head_dim against the float32 kernels over
the same (rounded) rows; the embedding gradient in its serial order."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import trainer as T
from tests.helpers import chain_tree, random_tree, rel_err

pytestmark = pytest.mark.gpu


def _wide(n):
    """Two rows with all the others below the second: a subtree of every tile."""
    p = np.full(n, 1, np.int32)
    p[0], p[1] = -1, 0
    return p


@pytest.mark.parametrize("parent,H,hd", [(chain_tree(1), 1, 16), (chain_tree(65), 3, 32), (random_tree(700, 24, 1), 2, 64), (_wide(64 * 129 + 2), 2, 16),
                                         (_wide(64 * 260), 5, 32), (random_tree(5000, 90, 4, 0.2), 6, 64)])
@pytest.mark.parametrize("bf16,tol", [(False, 1e-5), (True, 2e-3)])        # float32 sums; products of operands rounded to 11 bits (2^-12 each, four of them)
def test_even_plan_attention(parent, H, hd, bf16, tol):
    import torch
    plan, even = A.WalkerPlan(parent, 64, 0), A.WalkerPlan(parent, 64, 0, even=True)
    n = len(parent)
    assert even.n_tiles == (n + 63) // 64 and even.info.n_reduce_multi == 0
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, do = [torch.randn(n, H * hd, device="cuda", generator=g) for _ in range(4)]
    ks, vs = (k.bfloat16(), v.bfloat16()) if bf16 else (k, v)
    got, want = [], []
    for p, kk, vv, res in ((even, ks, vs, got), (plan, ks.float(), vs.float(), want)):
        o, lse = A.attn_forward(p, q, kk, vv, H)
        res += [o, lse, *A.attn_backward(p, q, kk, vv, o, lse, do, H)]
    # floor 1: with a single key dq and dk are exactly zero, and what is left of dP - delta is the rounding of a sum of 16 products of
    # N(0, 1) values, 16 x 2^-12 at most, times scale and a row of K
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        assert rel_err(a.cpu().numpy(), b.cpu().numpy(), floor=1.0) < tol, name


def test_sampled_groups_with_even_tiles():
    import torch
    trie = A.RadixTrie.build(A.synth_markov_corpus(2000, 12, 2, 3), 12)
    ids = trie.lightning_sample(2, 1, 7)[4]
    space = T.SampleSpace(trie)
    for ranked in (True, False):                          # by runs, and over char positions
        if not ranked:
            space.rank = None
        for even in (False, True):
            s = space.group(ids, [], "off", 32, torch.device("cuda", 0), even=even)
            assert s.even == even and (s.plan.n_tiles == (s.n + 63) // 64) == even


@pytest.mark.parametrize("bf16", [False, True])
def test_even_plan_from_host_buffers(bf16):
    """The chunked host-buffer step reduces a node when the last of its tiles is done, whole: several chunks, a subtree over all of them."""
    import torch
    parent, H, hd = _wide(64 * 260), 5, 32
    plan = A.WalkerPlan(parent, 64, 0, even=True)
    rng = np.random.default_rng(2)
    q, k, v, do = [rng.standard_normal((len(parent), H * hd)).astype(np.float32) for _ in range(4)]
    got = A.attn_fwd_bwd_host(plan, q, k, v, do, H, A.KV_BF16 if bf16 else A.KV_F32)
    tq, tk, tv, td = [torch.from_numpy(x).cuda() for x in (q, k, v, do)]
    ks, vs = (A.kv_store_write_bf16(tk), A.kv_store_write_bf16(tv)) if bf16 else (tk, tv)
    o, lse = A.attn_forward(plan, tq, ks, vs, H)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, (o, lse, *A.attn_backward(plan, tq, ks, vs, o, lse, td, H))):
        assert np.array_equal(a, b.cpu().numpy()), name


@pytest.mark.parametrize("n,d,vocab", [(1, 32, 3), (2048, 64, 65), (2049, 36, 7), (20_000, 384, 96)])
def test_serial_embedding_gradient(n, d, vocab):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, d, device="cuda", generator=g)
    ids = torch.randint(0, vocab, (n,), device="cuda", generator=g, dtype=torch.int32)
    want = torch.zeros(vocab, d, dtype=torch.float64, device="cuda").index_add_(0, ids.long(), x.double())
    got = A.embedding_grad(x, ids, vocab, serial=True)
    # at most 2048 additions one after the other per block, then the blocks: (2048 + 10) half-ulps of sums of about 50
    assert rel_err(got.cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert torch.equal(got, A.embedding_grad(x, ids, vocab, serial=True))
