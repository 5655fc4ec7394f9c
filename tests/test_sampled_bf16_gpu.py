"""Sampled training on a bfloat16 K/V store gives the outputs it always gave.

A few optimizer steps on units of some ten rows amplify every rounding: a K or V row that falls to the other bfloat16 neighbour moves a
unit of the feed-forward over the kink of its ReLU, and the momentum of a model of eight layers by 1e-2 (one float32 GEMM in the place
of another of the same accuracy does that).  So the vectors are those of the steps by single operations before there was a native step
(commit 03f603c, on a B200), every 3,449th element of weights and momentum, and the tolerance is what bfloat16 training states: 3e-3
relative, 0.2 root mean squares for a single element.  tests/golden/sampled_bf16.npz is written by
`python -m tests.test_sampled_bf16_gpu OUT` run with that commit's package."""
import os
import sys

import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "sampled_bf16.npz")
# sampler, steps, characters, vocabulary, order, depth: uniform units of ten rows; walks that stop at subtrees of up to two thousand rows
# (many tiles, blocks of the embedding gradient); short walks to the leaves
CASES = [(1, 5, 4000, 96, 3, 22), (3, 6, 5000, 96, 2, 9), (4, 5, 3000, 70, 3, 19)]
STRIDE = 3449


def _run(sampler, steps, chars, vocab, order, depth):
    import torch
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(0)
    trie = A.RadixTrie.build(A.synth_markov_corpus(chars, vocab, order, 5), depth)
    counts = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in (trie.cnt_off.astype(np.int32), trie.cnt_tok, trie.cnt_val)]
    model = T.TrieWalkModel(MF.random_init(384, 6, 8, vocab, 128, seed=11), dev)
    opt = T.make_optimizer("momentum", model, 1e-4)
    loss, queries, nodes, _ = T.train_lightning_epoch(model, T.SampleSpace(trie), counts, opt, sampler, steps, 0x5C115E1, mass_mode="linear", bf16_store=True)
    return dict(loss=loss, queries=queries, nodes=nodes, weights=model.flat.detach()[::STRIDE].cpu().numpy(), momentum=opt.m[::STRIDE].cpu().numpy())


@pytest.mark.parametrize("i", range(len(CASES)))
def test_sampled_bf16_outputs_stay(i, cuda):
    want = np.load(GOLDEN)
    got = _run(*CASES[i])
    for k, v in got.items():
        a, b = np.asarray(want[f"{i}.{k}"], np.float64), np.asarray(v, np.float64)
        if k in ("queries", "nodes"):
            assert int(a) == int(b), k
            continue
        d, rms = np.abs(a - b), np.sqrt((a * a).mean())
        assert np.sqrt((d * d).mean()) <= 3e-3 * rms and (d / np.maximum(np.abs(a), rms)).max() <= 0.2, k


if __name__ == "__main__":
    np.savez(sys.argv[1], **{f"{i}.{k}": v for i, c in enumerate(CASES) for k, v in _run(*c).items()})
