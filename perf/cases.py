"""Performance cases: the work a user of agpt_b200 has it do, through the package's public entry points.

Six kinds of work, in the order a training run meets them:

  build      a corpus becomes launch groups: RadixTrie.build_gpu, then trainer.build_groups (the start-up of a run)
  attention  attn_forward (and attn_backward) over one launch of a trie, inputs resident on the GPU
  loss       loss_per_query over the logits of one launch, mass weights on
  train      trainer.train_epoch: every position of the trie once, gradients summed, one optimizer step
  sampled    trainer.train_lightning_epoch: stochastic training units, one gradient and one optimizer step each
  host       attn_fwd_bwd_host: the same attention step for a caller whose rows live in pinned host memory

The shapes are those of the repository's own configurations (bench.py: c1, c2, the microbenchmark tree, c4, c5), with
shorter corpora so that one pass takes milliseconds: 65 or 96 symbols, tries of depth 8, 32 or 128 (pruned at count < 2),
head layouts 4 x 16, 4 x 32, 8 x 32, 8 x 64 and 6 x 64, float32 and bfloat16 KV stores.
"""
import functools
import math

import numpy as np
import torch

import agpt_b200 as A
from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T

# tree: "trie" = radix trie of a Markov corpus (chars, vocab, order, depth; prune: count < 2 from depth 4, with injected
# repeats); "random" = the microbenchmark's geometric-children tree (nodes)
LISTED = [
    # the smallest configuration's whole forest in one launch: 66k positions, latency and launches count
    dict(name="attention-depth8-4x16", kind="attention", tree="trie", chars=20_000, vocab=65, order=2, depth=8, prune=False,
         heads=4, head_dim=16, kv="f32", backward=True),
    # the headline workload (depth-32 trie, 4 x 32, float32) at a twentieth of its corpus: 1.4M positions
    dict(name="attention-depth32-4x32", kind="attention", tree="trie", chars=50_000, vocab=65, order=3, depth=32, prune=False,
         heads=4, head_dim=32, kv="f32", backward=True),
    # the attention microbenchmark's wide rows: 600k nodes, 8 x 64, float32
    dict(name="attention-random-8x64", kind="attention", tree="random", nodes=600_000, heads=8, head_dim=64, kv="f32", backward=True),
    # the deep pruned configuration: chains of up to 128 keys, 6 x 64, bfloat16 store
    dict(name="attention-deep-6x64-bf16", kind="attention", tree="trie", chars=12_000, vocab=96, order=4, depth=128, prune=True,
         heads=6, head_dim=64, kv="bf16", backward=True),
    # forward alone, as when a model is scored: 8 x 32, bfloat16 store
    dict(name="forward-depth32-8x32-bf16", kind="attention", tree="trie", chars=20_000, vocab=96, order=3, depth=32, prune=False,
         heads=8, head_dim=32, kv="bf16", backward=False),
    # the loss of one launch of the headline workload, rows of 65 logits
    dict(name="loss-v65", kind="loss", chars=50_000, vocab=65, order=3, depth=32, mass="linear", entropy=0.0),
    # one epoch of the smallest configuration: 66k positions, d_model 64, two layers
    dict(name="train-d64-depth8", kind="train", chars=20_000, vocab=65, order=2, depth=8, d_model=64, heads=4, layers=2, kv="f32",
         group_rows=1_000_000),
    # one epoch of the headline model on a 1.1M-position trie (two launch groups)
    dict(name="train-d128-depth32", kind="train", chars=40_000, vocab=65, order=3, depth=32, d_model=128, heads=4, layers=4, kv="f32",
         group_rows=1_000_000),
    # one epoch of the 5M-char configuration's model (d_model 256, six layers, 96 symbols) on a short corpus
    dict(name="train-d256-depth32", kind="train", chars=8_000, vocab=96, order=3, depth=32, d_model=256, heads=8, layers=6, kv="f32",
         group_rows=1_000_000),
    # the headline model trained on units drawn by the uniform sampler: tens of rows a step, so the host counts
    dict(name="sampled-l1-d128", kind="sampled", sampler=1, steps=16, chars=20_000, vocab=65, order=3, depth=32, d_model=128, heads=4,
         layers=4, kv="f32"),
    # a caller with its rows in pinned host memory: 170k positions up and back down
    dict(name="host-depth32-4x32", kind="host", chars=6_000, vocab=65, order=3, depth=32, heads=4, head_dim=32, kv="f32"),
    # from a 60k-token corpus to its launch group (1.7M positions)
    dict(name="build-depth32", kind="build", chars=60_000, vocab=65, order=3, depth=32),
]

LAYOUTS = [(4, 16), (4, 32), (3, 32), (8, 32), (8, 64), (6, 64)]
# d_model, heads, layers, vocabulary, KV store and the cost of a position relative to the headline model
MODELS = [(64, 4, 2, 65, "f32", 0.2), (128, 4, 4, 65, "f32", 1.0), (256, 8, 6, 96, "f32", 5.0), (384, 6, 8, 96, "bf16", 14.0)]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "attention", "loss", "train", "train", "train", "sampled", "host", "build"])
    if kind == "attention":
        heads, head_dim = rng.choice(LAYOUTS)
        c = dict(kind=kind, heads=heads, head_dim=head_dim, kv=rng.choice(["f32", "bf16"]), backward=rng.random() < 0.75)
        wide = heads * head_dim / 128.0
        shape = rng.choice(["shallow", "deep", "pruned", "random"])
        if shape == "random":
            return dict(c, tree="random", nodes=_log(rng, 3_000, 1_200_000 / wide))
        if shape == "pruned":
            return dict(c, tree="trie", chars=_log(rng, 2_000, 16_000 / max(wide, 1.0)), vocab=96, order=4, depth=rng.randint(64, 128), prune=True)
        if shape == "shallow":
            return dict(c, tree="trie", chars=_log(rng, 2_000, 100_000 / max(wide, 1.0)), vocab=rng.choice([65, 96]), order=2,
                        depth=rng.randint(4, 12), prune=False)
        return dict(c, tree="trie", chars=_log(rng, 1_000, 50_000 / max(wide, 1.0)), vocab=rng.choice([65, 96]), order=3,
                    depth=rng.randint(16, 48), prune=False)
    if kind == "loss":
        return dict(kind=kind, chars=_log(rng, 1_000, 50_000), vocab=rng.randint(40, 128), order=rng.choice([2, 3]), depth=rng.randint(8, 32),
                    mass=rng.choice(["linear", "log", "off"]), entropy=rng.choice([0.0, 0.5]))
    if kind in ("train", "sampled"):
        d_model, heads, layers, vocab, kv, cost = rng.choice(MODELS)
        deep = rng.random() < 0.6
        c = dict(kind=kind, vocab=vocab if rng.random() < 0.5 else rng.randint(40, 120), order=3 if deep else 2,
                 depth=rng.randint(16, 32) if deep else rng.randint(6, 12), d_model=d_model, heads=heads, layers=layers, kv=kv)
        if kind == "train":
            return dict(c, chars=_log(rng, 1_000, max(2_000, (40_000 if deep else 120_000) / max(cost, 1.0))),
                        group_rows=rng.choice([200_000, 1_000_000]))
        wide = cost > 1.0
        return dict(c, chars=_log(rng, 2_000, 8_000 if wide else 20_000), sampler=rng.choice([1, 1, 3, 4]),
                    steps=rng.randint(4, 8 if wide else 16))
    if kind == "host":
        heads, head_dim = rng.choice([(4, 16), (4, 32), (8, 32)])
        return dict(kind=kind, chars=_log(rng, 1_000, 8_000 * 128 // (heads * head_dim)), vocab=65, order=3, depth=rng.randint(16, 32), heads=heads,
                    head_dim=head_dim, kv=rng.choice(["f32", "f32", "bf16"]))
    return dict(kind=kind, chars=_log(rng, 4_000, 60_000), vocab=rng.choice([65, 96]), order=3, depth=rng.randint(12, 32))


# ---- trees ------------------------------------------------------------------------------------------------------------
def _corpus(case, seed):
    """One Markov corpus per case with its symbols renamed by the seed: other tokens, another order of the trie's branches and
    so other launch tiles, but the same number of positions, nodes and counts, so that the outputs of all seeds have one size."""
    base = A.synth_markov_corpus(case["chars"], case["vocab"], case["order"], 0, 10 if case.get("prune") else 0)
    return np.random.default_rng(seed).permutation(case["vocab"]).astype(np.int32)[base]


def _trie(case, seed):
    prune = (2, 4) if case.get("prune") else (1, 4)
    build = A.RadixTrie.build_gpu if torch.cuda.is_available() else A.RadixTrie.build
    return build(_corpus(case, seed), case["depth"], 1, *prune)


def _parent(case, seed):
    if case.get("tree") == "random":
        return A.synth_tree(case["nodes"], 64, 65, 0.35, 65, 75_000, seed)
    return _trie(case, seed).char_tree()[0]


@functools.lru_cache(maxsize=64)
def _sizes(key):
    """(positions, sum of depths, radix nodes, count entries) of a case's tree."""
    case = dict(key)
    if case.get("tree") == "random":
        plan = A.WalkerPlan(_parent(case, 0), 64, -1)
        return plan.n, plan.sum_depth, plan.n, 0
    trie = _trie(case, 0)
    plan = A.WalkerPlan(trie.char_tree()[0], 64, -1)
    return plan.n, plan.sum_depth, trie.radix_count, int(trie.cnt_tok.size)


def _tree_sizes(case):
    keys = ("tree", "chars", "vocab", "order", "depth", "prune", "nodes")
    return _sizes(tuple(sorted((k, case[k]) for k in keys if k in case)))


# ---- preparation ------------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _randn(gen, *shape):
    return torch.randn(shape, device=gen.device, generator=gen)


def _counts(trie, dev):
    return [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in (trie.cnt_off.astype(np.int32), trie.cnt_tok, trie.cnt_val)]


def _model(case, seed, dev):
    """The model with its optimizer: N(0, 0.02) weights and unit gains, as a run starts."""
    mf = MF.random_init(case["d_model"], case["heads"], case["layers"], case["vocab"], 128, seed=seed)
    model = T.TrieWalkModel(mf, dev)
    return model, T.make_optimizer("momentum", model, 1e-4)


def prepare(case, seed):
    kind, dev = case["kind"], _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    s = dict(case=case)
    if kind == "build":
        s["corpus"] = _corpus(case, seed)
    elif kind == "attention":
        s["plan"] = A.WalkerPlan(_parent(case, seed), 64, dev.index)
        n, d = s["plan"].n, case["heads"] * case["head_dim"]
        s["q"], s["k"], s["v"], s["dout"] = [_randn(gen, n, d) for _ in range(4)]
        if case["kv"] == "bf16":
            s["k"], s["v"] = A.kv_store_write_bf16(s["k"]), A.kv_store_write_bf16(s["v"])
    elif kind == "loss":
        trie = _trie(case, seed)
        groups, _ = T.build_groups(trie, 0, 1, 1 << 30, case["mass"], 128, dev)
        s["group"], s["counts"] = groups[0], _counts(trie, dev)
        s["logits"] = _randn(gen, groups[0].n, case["vocab"])
    elif kind == "train":
        trie = _trie(case, seed)
        s["groups"], _ = T.build_groups(trie, 0, 1, case["group_rows"], "linear", 128, dev)
        s["counts"] = _counts(trie, dev)
        s["model"], s["opt"] = _model(case, seed, dev)
    elif kind == "sampled":
        trie = _trie(case, seed)
        s["space"], s["counts"], s["seed"] = T.SampleSpace(trie), _counts(trie, dev), 0x5C115E1 + 7919 * seed & 0xFFFFFFFF
        s["model"], s["opt"] = _model(case, seed, dev)
    elif kind == "host":
        s["plan"] = A.WalkerPlan(_parent(case, seed), 64, dev.index)
        n, h, d = s["plan"].n, case["heads"], case["heads"] * case["head_dim"]
        pinned = lambda cols: torch.empty((n, cols), dtype=torch.float32, pin_memory=True)  # noqa: E731
        s["in"] = [pinned(d) for _ in range(4)]
        for t in s["in"]:
            t.copy_(_randn(gen, n, d))
        s["out"] = [pinned(c) for c in (d, h, d, d, d)]
    else:
        raise ValueError(kind)
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "build":
        trie = A.RadixTrie.build_gpu(s["corpus"], case["depth"])
        groups, total = T.build_groups(trie, 0, 1, 2_000_000, "linear", 128, _device())
        # the trie's arrays, and of the launch group what the kernels read
        g = groups[0]
        names = ("parent", "first_char_depth", "edge_len", "edge_mass", "endpoint_depth", "edge_start", "edge_tok", "cnt_off", "cnt_tok", "cnt_val")
        out = {n: getattr(trie, n) for n in names}
        return dict(out, positions=total, tokens=g.tokens32, pos=g.pos, q2n=g.q2n, qoff=g.qoff, rid=g.rid, mass=g.mass_w,
                    edge_first=g.edge_first, sub_end=g.plan.sub_end)
    if kind == "attention":
        out, lse = A.attn_forward(s["plan"], s["q"], s["k"], s["v"], case["heads"])
        if not case["backward"]:
            return out, lse
        return (out, lse) + A.attn_backward(s["plan"], s["q"], s["k"], s["v"], out, lse, s["dout"], case["heads"])
    if kind == "loss":
        g = s["group"]
        return A.loss_per_query(s["logits"], g.q2n, g.qoff, g.rid, g.tokens32, *s["counts"], g.mass_w, case["entropy"])
    if kind == "train":
        loss, n = T.train_epoch(s["model"], s["groups"], s["counts"], s["opt"], bf16_store=case["kv"] == "bf16")
        return dict(loss=loss, queries=n, weights=s["model"].flat, momentum=s["opt"].m)
    if kind == "sampled":
        loss, n, nodes, _ = T.train_lightning_epoch(s["model"], s["space"], s["counts"], s["opt"], case["sampler"], case["steps"], s["seed"],
                                                    mass_mode="linear", bf16_store=case["kv"] == "bf16")
        return dict(loss=loss, queries=n, nodes=nodes, weights=s["model"].flat, momentum=s["opt"].m)
    store = A.KV_BF16 if case["kv"] == "bf16" else A.KV_F32
    return A.attn_fwd_bwd_host(s["plan"], *[t.numpy() for t in s["in"]], case["heads"], store, outs=[t.numpy() for t in s["out"]])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _attention_work(n, depths, heads, head_dim, kv_bytes, forward=True, backward=True):
    d = heads * head_dim
    b = f = 0.0
    if forward:         # q, k, v -> out, lse;  two products per attended key
        b += n * (2 * 4 * d + 2 * kv_bytes * d + 4 * heads)
        f += 4.0 * d * depths
    if backward:        # q, k, v, out, dout, lse -> dq, dk, dv;  five products per attended key
        b += n * (6 * 4 * d + 2 * kv_bytes * d + 4 * heads)
        f += 10.0 * d * depths
    return b, f


def work(case):
    kind = case["kind"]
    n, depths, nodes, entries = _tree_sizes(case)
    kv_bytes = 2 if case.get("kv") == "bf16" else 4
    if kind == "attention":
        b, f = _attention_work(n, depths, case["heads"], case["head_dim"], kv_bytes, True, case["backward"])
        return dict(bytes=b, flops=f)
    if kind == "loss":
        return dict(bytes=n * (8.0 * case["vocab"] + 16) + 8 * entries + 8 * nodes, flops=n * 6.0 * case["vocab"])
    if kind == "host":
        d = case["heads"] * case["head_dim"]
        return dict(bytes=n * (8 * 4.0 * d + 4 * case["heads"]), flops=_attention_work(n, depths, case["heads"], case["head_dim"], kv_bytes)[1])
    if kind == "build":
        return dict(bytes=4.0 * case["chars"] + n * 4.0 * 8 + nodes * 4.0 * 12 + entries * 8.0, flops=2.0 * case["chars"] * case["depth"])
    d, layers = case["d_model"], case["layers"]
    if kind == "sampled":
        # rows of a step: the mean over the sampled units of seed 0
        trie = _trie(case, 0)
        _, _, _, _, ids, _ = trie.lightning_sample(case["sampler"], case["steps"], 0x5C115E1)
        rows = float(trie.edge_len[ids].sum())
        n, depths, steps = rows, rows * 0.5 * case["depth"], case["steps"]
    else:
        steps = 1
    params = 2.0 * case["vocab"] * d + layers * (12.0 * d * d + 13 * d)
    ab, af = _attention_work(n, depths, case["heads"], d // case["heads"], kv_bytes)
    # per layer beside the attention: the residual stream once each way, q/k/v, the attention output and the feed-forward
    # activation written for the backward and read there; per step the parameters, gradients and momenta
    b = layers * (ab + n * d * 4.0 * 16) + n * 12.0 * case["vocab"] + steps * params * 4.0 * 5
    f = layers * (af + 3 * 24.0 * n * d * d) + 6.0 * n * d * case["vocab"]
    return dict(bytes=b, flops=f)


def tolerance(case):
    kind = case["kind"]
    if kind == "build":            # index arrays are equal; the mass weights are float32 quotients
        return dict(rel=1e-6)
    if kind == "loss":             # float32 exponentials and logarithms
        return dict(rel=1e-5)
    if kind in ("train", "sampled"):
        # float32 GEMMs and reductions through every layer; a bfloat16 store may round a row the other way
        return dict(rel=1e-4 if case["kv"] == "f32" else 3e-3, max=0.02 if case["kv"] == "f32" else 0.2)
    # float32 store: sums of float32-accurate products; bfloat16 store: products of bfloat16 rows at reduced precision
    return dict(rel=2e-5 if case["kv"] == "f32" else 5e-3, max=1e-3 if case["kv"] == "f32" else 0.2)
