"""The training step in a workspace the caller cut from an arena of its own."""
import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from tests.test_train_step_gpu import _group, _step


class _Arena:
    """torch.empty whose byte buffers (the step's workspace) start `offset` bytes behind an allocation's first address."""

    def __init__(self, torch, offset):
        self.empty, self.uint8, self.offset, self.seen = torch.empty, torch.uint8, offset, []

    def __call__(self, *size, **kw):
        if kw.get("dtype") is not self.uint8:
            return self.empty(*size, **kw)
        t = self.empty(size[0] + 256, **kw)[self.offset:self.offset + size[0]]
        self.seen.append(t.data_ptr())
        return t


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,heads,ff,vocab", [(150, 128, 4, 512, 65), (9000, 64, 4, 96, 12)])
def test_workspace_on_a_16_byte_boundary(monkeypatch, n, d, heads, ff, vocab):
    """Nothing of the step needs more than 16 bytes: the same bits at every such offset (partial sums leave by 32-byte stores where they can)."""
    import torch
    dev = torch.device("cuda", 0)
    g, counts = _group(n, 9, vocab, n + d, 128, dev)
    mf = MF.random_init(d, heads, 2, vocab, 128, d_ff=ff, seed=3, std=0.1)
    want = _step(mf, g, counts, dev, "tensor")
    for offset in (16, 48, 64):
        with monkeypatch.context() as m:
            arena = _Arena(torch, offset)
            m.setattr(torch, "empty", arena)
            got = _step(mf, g, counts, dev, "tensor")
        assert arena.seen and arena.seen[0] % 64 == offset % 64
        assert got[:2] == want[:2] and all(np.array_equal(got[2][k], want[2][k]) for k in want[2])
    assert A.device_status() == 0


def test_other_boundaries_are_refused():
    """Without a look at anything else: no kernel has been launched."""
    import ctypes as C
    from agpt_b200._lib import TrainStepArgs
    args = TrainStepArgs()
    for at in (0x1001, 0x1004, 0x1008):
        assert A.lib().agpt_b200_train_step(C.byref(args), C.c_void_p(at), 1 << 30, None) == -1
        assert "16-byte boundary" in A.lib().agpt_b200_last_error().decode()
