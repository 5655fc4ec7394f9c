"""Device memory of the native training step, by the size it asks for (nothing is launched)."""
import ctypes as C

import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200._lib import TrainStepArgs

pytestmark = pytest.mark.gpu
KEPT = 1 << 30


def _bytes(n, d, heads, layers, ff, recompute=False, vocab=65):
    plan = A.WalkerPlan(np.full(n, -1, np.int32), 64, 0)          # no chains: the attention's share does not depend on the tree
    a = TrainStepArgs()
    a.plan, a.n, a.n_units, a.n_pos, a.seq_len = plan._h, n, 1, 1, 128
    a.d_model, a.n_heads, a.n_layers, a.d_ff, a.vocab, a.ffn_recompute = d, heads, layers, ff, vocab, int(recompute)
    a.params = a.grads = 256                                      # not read
    return A.check(A.lib().agpt_b200_train_step_workspace_bytes(C.byref(a)), "workspace")


@pytest.mark.parametrize("n,d,heads,layers,ff", [(200, 128, 4, 4, 512), (20_000, 64, 4, 8, 256), (49_152, 128, 4, 8, 512), (60_000, 128, 4, 4, 512)])
def test_recompute_saves_the_activations_of_all_layers_but_one(cuda, n, d, heads, layers, ff):
    assert _bytes(n, d, heads, layers, ff) - _bytes(n, d, heads, layers, ff, True) >= (layers - 1) * n * ff * 4


@pytest.mark.parametrize("n,d,heads,layers,ff", [(98_304, 64, 4, 12, 4096), (49_152, 128, 4, 8, 512), (6144, 1024, 16, 24, 4096)])
def test_kept_gradients_have_a_limit(cuda, n, d, heads, layers, ff):
    """Beside what the activations take: wide or deep models of few rows share their buffers."""
    shared = _bytes(n, d, heads, layers, ff, True) + (layers - 1) * n * ff * 4
    assert _bytes(n, d, heads, layers, ff) <= shared + KEPT + 4096 * layers


@pytest.mark.parametrize("d,heads,layers,ff", [(128, 4, 4, 512), (64, 4, 12, 4096), (1024, 16, 1, 4096)])
@pytest.mark.parametrize("recompute", [False, True])
def test_the_largest_group_s_workspace_serves_the_smaller_ones(cuda, d, heads, layers, ff, recompute):
    """Across the row counts at which gradients are no longer kept and the slices of their launch become fewer."""
    kept = min((6 << 20) // d, KEPT // (4 * layers * (ff + 5 * d)))
    rows = sorted({1, 64, 128, 192, 256, 257, 512, 513, 1280, 1281, 4096, 4097, kept - 1, kept, kept + 1, kept + 65, 2 * kept})
    sizes = [_bytes(n, d, heads, layers, ff, recompute) for n in rows if n > 0]
    assert sizes == sorted(sizes)
