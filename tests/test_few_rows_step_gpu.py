"""The native training step on both sides of the rule that tells few rows from many (rows x d_model against 6 Mi): few rows keep the gradients
of the rows layer by layer and form all weight gradients in launches of up to 40 contractions.  Against the tape with torch's float32 GEMMs."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from tests.helpers import TOL_F32, rel_err
from tests.test_train_step_gpu import _group, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,d,heads,ff,layers,kw", [
    (63, 9, 64, 4, 256, 2, {}),                                              # one row block, one slice
    (65, 9, 128, 4, 512, 1, dict(grad_mode="local_depth")),                  # two
    (500, 12, 96, 3, 160, 1, {}),                                            # whole rows over clusters of three blocks
    (4736, 12, 128, 4, 512, 1, {}),                                          # the last row count whose row tiles have a cluster each on 148 SMs,
    (4737, 12, 128, 4, 512, 1, {}),                                          # the first without
    (1344, 12, 32, 2, 64, 11, {}),                                           # 45 contractions: two launches, several row blocks a slice
    ((6 << 20) // 64, 10, 64, 4, 96, 1, {}),                                 # the last row count with kept gradients and early placement,
    ((6 << 20) // 64 + 1, 10, 64, 4, 96, 1, {}),                             # the first without
    ((6 << 20) // 64, 10, 64, 4, 96, 1, dict(ffn_recompute=True)),           # early placement with shared buffers,
    ((6 << 20) // 64 + 1, 10, 64, 4, 96, 1, dict(ffn_recompute=True)),       # neither
])
def test_few_and_many_rows_match_the_tape(n, depth, d, heads, ff, layers, kw):
    import torch
    dev = torch.device("cuda", 0)
    g, counts = _group(n, depth, 65, n + d, 128, dev)
    mf = MF.random_init(d, heads, layers, 65, 128, d_ff=ff, seed=3, std=0.1)
    # feed-forward units well away from the kink of the ReLU (the same float32 sum in another order may fall on its other side)
    mf.mats = [(k, a * 0.1 if k.endswith("l1.w") else (np.where(np.arange(a.size) % 3, 0.5, -0.5).astype(np.float32)[None] if k.endswith("l1.b") else a))
               for k, a in mf.mats]
    want_l, want_n, want = _step(mf, g, counts, dev, "torch", **kw)
    got_l, got_n, got = _step(mf, g, counts, dev, "tensor", **kw)
    assert got_n == want_n and abs(got_l - want_l) <= TOL_F32 * abs(want_l)
    for k in want:
        assert rel_err(got[k], want[k]) < TOL_F32, k
    again = _step(mf, g, counts, dev, "tensor", **kw)
    assert again[0] == got_l and all(np.array_equal(again[2][k], got[k]) for k in got)          # repeatable bit for bit
    assert A.device_status() == 0
