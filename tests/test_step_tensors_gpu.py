"""A training step reads the parameters and adds to the gradients as they are when it is called: storage replaced between two steps, a
parameter or a gradient that the native step does not read by address (it then runs on the tape)."""
import numpy as np
import pytest

from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T
from tests.helpers import rel_err
from tests.test_train_step_gpu import _group

pytestmark = pytest.mark.gpu


def _setup(dev, twice=None):
    import torch
    g, counts = _group(200, 9, 12, 1, 32, dev)
    mf = MF.random_init(64, 2, 1, 12, 32, seed=3, std=0.1)
    if twice:
        mf.mats = [(k, a * 2 if k == twice else a) for k, a in mf.mats]
    return T.TrieWalkModel(mf, dev), g, [torch.from_numpy(c).to(dev) for c in counts]


def _grads(model):
    return {k: p.grad.detach().clone().cpu().numpy() for k, p in model.params.items()}


def _check(got, want):
    assert np.isclose(got[0], want[0], rtol=1e-5)
    for k in want[1]:
        assert rel_err(got[1][k], want[1][k]) < 1e-4, k


def _want(dev, name):
    model, g, counts = _setup(dev, name)
    return model.group_step(g, counts)[0], _grads(model)


@pytest.mark.parametrize("name", ["token_emb", "layer0.wk.w", "layer0.ln2.gamma", "out.b"])
def test_replaced_parameter_storage(cuda, name):
    model, g, counts = _setup(cuda)
    model.group_step(g, counts)
    model.flat_grad.zero_()
    p = model.params[name]
    p.data = p.data * 2                                  # the gradient tensors stay
    _check((model.group_step(g, counts)[0], _grads(model)), _want(cuda, name))


def test_replaced_gradient_storage(cuda):
    import torch
    model, g, counts = _setup(cuda)
    model.group_step(g, counts)
    old = model.params["layer0.wq.w"].grad.data
    kept = old.clone()
    model.flat_grad[:].zero_()
    old.copy_(kept)
    model.params["layer0.wq.w"].grad.data = torch.zeros_like(old)
    _check((model.group_step(g, counts)[0], _grads(model)), _want(cuda, None))
    assert torch.equal(old, kept)


def test_what_the_native_step_reads_by_address(cuda):
    import torch
    model, _, _ = _setup(cuda)
    n = len(model.params)
    at = model._step_addresses()
    assert at[:n] == [p.data_ptr() for p in model.params.values()] and at[n:] == [p.grad.data_ptr() for p in model.params.values()]
    p = model.params["layer0.wo.w"]
    plain = p.data
    for other in (torch.zeros(plain.numel() + 1, device=cuda)[1:].view(plain.shape), plain.t(), plain.double(), plain.cpu(), plain[:32]):
        p.grad = None
        p.data = other
        p.grad = None if other.device != plain.device else torch.zeros_like(other)
        assert model._step_addresses() is None
    p.grad = None
    p.data = plain
    assert model._step_addresses()[:n] == at[:n]


def test_strided_gradient_and_missing_gradient(cuda):
    import torch
    model, g, counts = _setup(cuda)
    w = model.params["layer0.l1.w"]
    w.grad = torch.zeros(w.shape[1], w.shape[0], device=cuda).t()
    model.params["out.w"].grad = None
    loss = model.group_step(g, counts)[0]
    _check((loss, _grads(model)), _want(cuda, None))
    # the statistics of a step without a host read are laid out alike on either path
    got = [T._step_stats(model.group_step(g, counts, sync=None, tape=t).cpu()) for t in (False, True)]
    assert got[0][0][1] == got[1][0][1] > 0 and np.allclose([x[0][0] for x in got], loss, rtol=1e-5)
