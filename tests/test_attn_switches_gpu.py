"""The switches between the attention kernels.  On a single tile the chunked kernels are those of an
even plan, bit for bit; the whole-tile ones keep more bits of Q and P.  whole_tile 0 leaves a bfloat16 store's forward as it is."""
import os
import subprocess
import sys

import pytest

import agpt_b200 as A
from tests.helpers import random_tree

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _outputs(even, hd, bf16, n=60):
    import torch
    plan = A.WalkerPlan(random_tree(n, 20, 3), 64, 0, even=even)
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = [torch.randn(n, 2 * hd, device="cuda", generator=g) for _ in range(4)]
    if bf16:
        k, v = k.bfloat16(), v.bfloat16()
    out, lse = A.attn_forward(plan, q, k, v, 2)
    return (out, lse) + A.attn_backward(plan, q, k, v, out, lse, do, 2)


def _same(x, y):
    import torch
    return [torch.equal(a, b) for a, b in zip(x, y)]


@pytest.mark.parametrize("hd", [16, 32, 64])
@pytest.mark.parametrize("bf16", [False, True])
def test_whole_tile_0_is_the_chunked_kernels(hd, bf16):
    want, whole = _outputs(True, hd, bf16), _outputs(False, hd, bf16)
    assert not any(_same(whole, want))
    A.set_attn_variant(False, 4)
    try:
        got = _outputs(False, hd, bf16)
        if bf16:                                         # the backward from the forward's out and lse, whichever kernel they are of
            assert all(_same(got[:2], whole[:2])) and not any(_same(got[2:], whole[2:]))
        else:
            assert all(_same(got, want))
    finally:
        A.set_attn_variant(True, 4)


@pytest.mark.parametrize("env,want", [({"AGPT_B200_ATTN_TILE_BF16": "0"}, "TTTTT FFFFF"), ({"AGPT_B200_ATTN_TILE": "0"}, "FFFFF TTTTT"), ({}, "FFFFF FFFFF")])
def test_environment(env, want):
    """Per output (out, lse, dq, dk, dv): is it the chunked kernel's?  Bfloat16 store, then float32."""
    code = ("from tests.test_attn_switches_gpu import _outputs, _same; print(' '.join(''.join('TF'[not x] for x in "
            "_same(_outputs(False, 32, b), _outputs(True, 32, b))) for b in (True, False)))")
    got = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0, got.stderr[-2000:]
    assert got.stdout.split("\n")[-2] == want


def test_five_blocks_per_sm():
    code = ("import torch; from tests.test_attn_switches_gpu import _outputs; torch.save([x.cpu() for x in _outputs(False, 32, False)], __import__('sys').argv[1])")
    import tempfile

    import torch
    res = []
    with tempfile.TemporaryDirectory() as d:
        for env in ({}, {"AGPT_B200_FWD_BLOCKS": "5"}):
            f = os.path.join(d, "o.pt")
            subprocess.run([sys.executable, "-c", code, f], cwd=ROOT, env={**os.environ, **env}, check=True, timeout=300)
            res.append(torch.load(f))
    assert all(torch.allclose(a, b, rtol=1e-5, atol=1e-6) for a, b in zip(*res))      # another register allocation of the same program
