"""The GPU trie builder in the caller's device memory: the same trie as in its own, at both digit widths' edges of the key length, and a refusal
of a workspace that is too small."""
import ctypes as C

import numpy as np
import pytest

import agpt_b200 as A
from agpt_b200._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chars,vocab,depth", [(12, 3, 2), (2000, 7, 20), (3000, 65, 8), (3000, 300, 15)])
def test_build_in_a_workspace(chars, vocab, depth):
    import torch
    corpus = np.ascontiguousarray(np.random.default_rng(chars + vocab).integers(0, vocab, chars), np.int32)
    corpus[0] = vocab - 1
    vp = corpus.ctypes.data_as(C.c_void_p)
    need = lib().agpt_b200_trie_build_workspace_bytes(chars)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    tries = []
    for own in (False, True):
        h = C.c_void_p()
        if own:
            check(lib().agpt_b200_trie_build_gpu(vp, chars, depth, 1, 1, 4, 0, C.byref(h)), "build")
        else:
            check(lib().agpt_b200_trie_build_gpu_ws(vp, chars, depth, 1, 1, 4, 0, C.c_void_p(ws.data_ptr()), need, None, C.byref(h)), "build")
        tries.append(A.RadixTrie(h))
    a, b = [t.char_tree() for t in tries]
    assert all(np.array_equal(x, y) for x, y in zip(a, b) if isinstance(x, np.ndarray))
    h = C.c_void_p()
    with pytest.raises(A.AgptError, match="workspace"):
        check(lib().agpt_b200_trie_build_gpu_ws(vp, chars, depth, 1, 1, 4, 0, C.c_void_p(ws.data_ptr()), 64, None, C.byref(h)), "build")
