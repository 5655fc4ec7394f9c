"""A wait that ran out in a kernel reaches whoever trains: the status word is read with an epoch's statistics, on every rank.  The word itself is
planted on the host."""
import os
import socket

import numpy as np
import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

import agpt_b200 as A
from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T
from tests.test_dist_cpu import _FakeGroup, _FakeModel, _FakeOpt


class _FailingModel(_FakeModel):
    word = 2.0

    def group_step(self, g, counts, sync=True, **kw):
        self.flat_grad[self.n_flat + 3] = self.word
        return super().group_step(g, counts, sync, **kw)


def test_epoch_raises():
    groups = [_FakeGroup(torch.ones(10), 1.0, 3)]
    model = _FailingModel(10)
    with pytest.raises(A.AgptError, match="status 2"):
        T.train_epoch(model, groups, None, _FakeOpt(model))
    model.word = 0.0
    assert T.train_epoch(model, groups, None, _FakeOpt(model)) == (1.0, 3)


def _worker(rank, world, port, ret):
    os.environ["MASTER_ADDR"], os.environ["MASTER_PORT"] = "127.0.0.1", str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    model = _FailingModel(10)
    model.word = float(rank)                              # rank 1's kernels failed
    try:
        T.train_epoch(model, [_FakeGroup(torch.ones(10), 1.0, 3)], None, _FakeOpt(model), world=world)
        ret[rank] = "went on"
    except A.AgptError:
        ret[rank] = "raised"
    dist.barrier()
    dist.destroy_process_group()


def test_every_rank_raises():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    ret = mp.Manager().dict()
    mp.spawn(_worker, args=(2, port, ret), nprocs=2, join=True)
    assert dict(ret) == {0: "raised", 1: "raised"}


@pytest.mark.gpu
@pytest.mark.parametrize("dense,bf16", [("tensor", False), ("torch", False), ("tensor", True)])
def test_epochs_on_the_gpu(cuda, monkeypatch, dense, bf16):
    word = torch.full((1,), 0.5, device=cuda)
    A.device_status_add(word)
    assert float(word) == 0.5 and A.device_status() == 0
    trie = A.RadixTrie.build(A.synth_markov_corpus(600, 8, 2, 3), 6)
    counts = [torch.tensor(np.asarray(c), dtype=torch.int32, device=cuda) for c in (trie.cnt_off, trie.cnt_tok, trie.cnt_val)]
    model = T.TrieWalkModel(MF.random_init(32, 2, 1, 8, 16, seed=1), cuda)
    model.dense_impl = dense
    opt = T.make_optimizer("momentum", model, 1e-3)
    groups, _ = T.build_groups(trie, 0, 1, 1 << 20, "off", 16, cuda)

    def epochs():
        yield lambda: T.train_epoch(model, groups, counts, opt, bf16_store=bf16)
        yield lambda: T.train_lightning_epoch(model, T.SampleSpace(trie), counts, opt, 1, 2, 9, bf16_store=bf16)
    for run in epochs():
        run()
    monkeypatch.setattr(A.api, "device_status_add", lambda out: out.add_(2.0))
    for run in epochs():
        with pytest.raises(A.AgptError, match="status 2"):
            run()
