"""Both layouts of the native training step against the tape with torch's float32 GEMMs.  The gradients of the rows are kept layer by layer, or (many rows, or
recomputed feed-forward activations) pass through buffers that all layers share; then the residual gradient is updated in place and q, k, v, the feed-forward's
gradient and the logits take turns in one region.  Sizes lie where the projections' schedules change as well."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from tests.helpers import TOL_BF16, TOL_F32, rel_err
from tests.test_train_step_gpu import _group, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,d,heads,ff,vocab,layers,kw", [
    # shared buffers by the recompute switch, at sizes of every kind
    (127, 9, 64, 4, 256, 65, 3, dict(ffn_recompute=True)),
    (700, 40, 128, 4, 512, 96, 2, dict(ffn_recompute=True, grad_mode="own_edge", context=True)),
    (700, 20, 160, 5, 320, 129, 2, dict(ffn_recompute=True, grad_mode="local_depth")),       # layer-norm backward as a pass of its own, in place
    (900, 70, 256, 4, 1024, 96, 3, dict(ffn_recompute=True, bf16_store=True)),               # keys and values rotated and rounded in passes of their own
    # shared buffers by the row count
    (49_153, 20, 128, 4, 512, 65, 2, {}),                                                    # 385 row tiles; one row in the last
    (49_281, 20, 128, 4, 512, 65, 2, dict(bf16_store=True, context=True)),                   # 386
    (49_281, 20, 128, 4, 512, 65, 2, dict(ffn_recompute=True, grad_mode="own_edge")),
    (24_700, 40, 256, 4, 1024, 96, 2, dict(bf16_store=True)),                                # rotation beyond shared memory, streamed weights
    # weights that stream while two row tiles share a pass, 99 and 100 row tiles: the last pass has one tile, or two
    (12_600, 12, 256, 4, 1024, 65, 1, {}),
    (12_700, 12, 256, 4, 1024, 65, 2, {}),
    # weights that stream through the clusters of whole rows
    (300, 9, 128, 4, 2048, 65, 1, {}),
])
def test_layouts_match_the_tape(n, depth, d, heads, ff, vocab, layers, kw):
    import torch
    dev = torch.device("cuda", 0)
    kw = dict(kw)
    g, counts = _group(n, depth, vocab, n + d, 128, dev, kw.pop("context", False))
    mf = MF.random_init(d, heads, layers, vocab, 128, d_ff=ff, seed=3, std=0.1)
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
