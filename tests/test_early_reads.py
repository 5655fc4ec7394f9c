"""Kernels that may be placed while the kernel in front still works read nothing from device memory before they wait for it."""
import glob
import os
import re

import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200 import model_file as MF
from agpt_b200 import trainer as T
from tests.test_train_step_gpu import _group

CSRC = os.path.join(os.path.dirname(A.__file__), "csrc")
# what touches device memory: cached and bulk loads, atomics, and any subscript of a kernel parameter
ACCESS = re.compile(r"__ld\w+\s*\(|bulk_load|tma_(load|store)|\b(ld|st|red|atom)\.global|atomic\w+\s*\(")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(([^{;]*)\)\s*\{", text):
            body = text[m.end():text.index("\n}\n", m.end())] if "\n}\n" in text[m.end():] else text[m.end():]
            yield os.path.basename(path), m.group(1), m.group(2), body


def test_nothing_is_read_before_the_wait():
    seen = set()
    for path, name, params, body in _kernels():
        if "pdl_wait();" not in body:
            continue
        seen.add(name)
        front = re.sub(r"//[^\n]*", "", body[:body.index("pdl_wait();")])
        assert body.count("pdl_wait();") == 1 and not re.search(r"if\s*\([^()]*\)\s*\{?\s*$", front), (path, name)       # on every path
        assert not ACCESS.search(front), (path, name)
        for p in re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params):
            assert not re.search(rf"\b{p}\b", front), (path, name, p)
    assert {"row_gemm_kernel", "contract_kernel", "reduce_items_kernel", "step_kernel"} <= seen


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,heads,ff,layers", [(60, 128, 4, 512, 2), (700, 256, 4, 1024, 1)])
def test_steps_read_the_weights_of_the_update_before_them(n, d, heads, ff, layers):
    """Training steps and updates back to back, every weight moved far by each update: the same bits as with a device-wide wait after each call."""
    import torch
    dev = torch.device("cuda", 0)
    g, counts = _group(n, 9, 65, n + d, 128, dev)
    counts = [torch.from_numpy(c).to(dev) for c in counts]
    got = []
    for wait in (False, True):
        model = T.TrieWalkModel(MF.random_init(d, heads, layers, 65, 128, d_ff=ff, seed=3, std=0.1), dev)
        model.dense_impl = "tensor"
        opt = T.make_optimizer("adam", model, 0.05)
        for _ in range(12):
            model.group_step(g, counts, sync=None)
            if wait:
                torch.cuda.synchronize()
            opt.step()
            if wait:
                torch.cuda.synchronize()
        got.append({k: p.detach().cpu().numpy() for k, p in model.params.items()})
    for k in got[0]:
        assert np.isfinite(got[0][k]).all() and np.array_equal(got[0][k], got[1][k]), k
    assert A.device_status() == 0
