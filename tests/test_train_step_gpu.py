"""The native training step (agpt_b200_train_step: tcgen05 projections with the row work in their prologues and epilogues)
against the tape path of the trainer with torch's float32 GEMMs and the separate layer-norm, RoPE and bias kernels: loss
and every parameter gradient, at the edges of its tiles (128 rows, 128 columns, 64 k) and for both sides of its rules
(a row inside one accumulator tile or not, a RoPE table in shared memory or not)."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T
from tests.helpers import TOL_BF16, TOL_F32, random_tree, rel_err

pytestmark = pytest.mark.gpu


def _group(n, depth, vocab, seed, seq_len, dev, context=False):
    """A launch group over a random tree: every node its own edge, two units, counts for each node."""
    rng = np.random.default_rng(seed)
    plan = A.WalkerPlan(random_tree(n, depth, seed, roots=min(3, n)), 64, -1)
    tokens = rng.integers(0, vocab, n).astype(np.int32)
    radix = np.arange(1, n + 1, dtype=np.int32)
    mass = rng.integers(1, 9, n + 1).astype(np.int32)
    trained = None
    if context:
        trained = rng.random(n) > 0.1
        trained[0] = True
    unit = (np.arange(n) >= n // 2).astype(np.int64)
    g = T.LaunchGroup(plan.parent_dfs, tokens, plan.depth, radix, mass, "log", seq_len, dev, 64, trained, unit)
    counts = (np.arange(n + 2, dtype=np.int32), rng.integers(0, vocab, n + 1).astype(np.int32), np.ones(n + 1, np.int32))
    return g, counts


def _step(mf, g, counts, dev, impl, **kw):
    import torch
    opts = {k: kw.pop(k) for k in ("grad_mode", "ffn_recompute") if k in kw}
    model = T.TrieWalkModel(mf, dev)
    model.dense_impl = impl
    for k, v in opts.items():
        setattr(model, k, v)
    model.flat_grad.fill_(0.25)                   # gradients are added to what is there
    ls, nq = model.group_step(g, [torch.from_numpy(c).to(dev) for c in counts], entropy_lambda=0.3, intermediate_weight=0.8, **kw)
    return ls, nq, {k: (p.grad - 0.25).cpu().numpy() for k, p in model.params.items()}


@pytest.mark.parametrize("n,depth,d,heads,ff,vocab,kw", [
    (1, 1, 32, 2, 32, 5, {}),                                            # one row, one 32-column chunk
    (127, 9, 64, 4, 256, 65, {}),                                        # one row short of a tile; padded vocabulary
    (129, 9, 96, 3, 160, 12, dict(context=True)),                        # one row over; half a k block
    (700, 40, 128, 4, 512, 96, dict(grad_mode="local_depth")),           # the widest row of one accumulator tile
    (700, 20, 160, 5, 320, 129, {}),                                     # a row over two tiles, vocabulary over one
    (900, 70, 256, 4, 1024, 96, dict(bf16_store=True)),                  # head_dim 64: RoPE table beyond shared memory
    (40_000, 12, 64, 4, 256, 65, dict(ffn_recompute=True)),              # two row tiles per unit
])
def test_native_step_matches_the_tape(n, depth, d, heads, ff, vocab, kw):
    import torch
    dev = torch.device("cuda", 0)
    kw = dict(kw)
    g, counts = _group(n, depth, vocab, n + d, 128, dev, kw.pop("context", False))
    mf = MF.random_init(d, heads, 2, vocab, 128, d_ff=ff, seed=3, std=0.1)
    rng = np.random.default_rng(7)
    mf.mats = [(k, (a + 0.1 * rng.standard_normal(a.shape)).astype(np.float32)) for k, a in mf.mats]      # gains, shifts and biases too
    # feed-forward units well away from the kink of the ReLU (the same float32 sum in another order may fall on its other side)
    mf.mats = [(k, a * 0.1 if k.endswith("l1.w") else (np.where(np.arange(a.size) % 3, 0.5, -0.5).astype(np.float32)[None] if k.endswith("l1.b") else a))
               for k, a in mf.mats]
    want_l, want_n, want = _step(mf, g, counts, dev, "torch", **kw)
    got_l, got_n, got = _step(mf, g, counts, dev, "tensor", **kw)
    tol = TOL_BF16 if kw.get("bf16_store") else TOL_F32
    assert got_n == want_n and abs(got_l - want_l) <= tol * abs(want_l)
    for k in want:
        assert rel_err(got[k], want[k]) < tol, k
    again = _step(mf, g, counts, dev, "tensor", **kw)
    assert again[0] == got_l and all(np.array_equal(again[2][k], got[k]) for k in got)          # repeatable bit for bit
    assert A.device_status() == 0
