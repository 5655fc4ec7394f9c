"""A training step repeats bit for bit whatever its workspace held before, in shapes whose output rows are an odd number of 32-column chunks (the vocabulary's 68
columns, feed-forwards of 96 and 32): the staging buffers of such tiles do not alternate from tile to tile."""
import numpy as np
import pytest

from agpt_b200 import model_file as MF
from tests.test_train_step_gpu import _group, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,heads,ff,vocab,kw", [
    (98_304, 64, 4, 96, 65, {}),                              # three chunks in the head and the feed-forward; the last row count with kept gradients,
    (98_305, 64, 4, 96, 65, {}),                              # the first without
    (60_000, 96, 3, 32, 20, dict(bf16_store=True)),           # one chunk; q, k and v end with one
    (66_000, 96, 3, 32, 20, dict(bf16_store=True)),           # the same without kept gradients
])
def test_step_repeats(n, d, heads, ff, vocab, kw):
    import torch
    dev = torch.device("cuda", 0)
    g, counts = _group(n, 10, vocab, n + d, 128, dev)
    mf = MF.random_init(d, heads, 1, vocab, 128, d_ff=ff, seed=3, std=0.1)
    first = None
    for _ in range(8):
        junk = [torch.full((1 << 28,), float("nan"), device=dev) for _ in range(2)]      # what the step's buffers hold, and a cold cache
        torch.cuda.synchronize()
        del junk
        got = _step(mf, g, counts, dev, "tensor", **kw)
        first = first or got
        assert got[:2] == first[:2] and all(np.array_equal(got[2][k], first[2][k]) for k in got[2])
