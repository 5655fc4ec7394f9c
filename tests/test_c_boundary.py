"""Limits and failures at the C boundary come back as codes: rows of a sampled set counted beyond 32 bits, and memory that runs out."""
import subprocess
import sys
import os

import numpy as np
import pytest

import agpt_b200 as A

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEPTH = 30_000


def _one_edge():
    """A trie of one radix edge of 30,000 characters."""
    trie = A.RadixTrie.build(np.zeros(DEPTH + 50, np.int32), DEPTH)
    assert trie.radix_count == 2 and trie.total_edge_chars == DEPTH
    return trie


@pytest.mark.parametrize("times", [2 ** 31 // DEPTH + 1, 2 ** 32 // DEPTH + 1, 2 ** 33 // DEPTH + 3])     # beyond 2^31, and where a 32-bit sum is positive again
def test_sampled_rows_beyond_32_bits(times):
    trie = _one_edge()
    with pytest.raises(ValueError, match="2\\^31"):
        A.RunGroups.of_sample(trie, A.trie_ranks(trie), np.ones(times, np.int32), [])
    assert len(A.RunGroups.of_sample(trie, A.trie_ranks(trie), np.ones(3, np.int32), [])) == 1


def test_out_of_memory_is_a_code():
    """A group of 1.8 billion rows (tiles and token staging of gigabytes) in a process that may take 512 MB more."""
    code = (
        "import resource, ctypes as C, numpy as np, agpt_b200 as A\n"
        "from agpt_b200._lib import RunGroupInfo, lib\n"
        "from tests.test_c_boundary import _one_edge\n"
        "trie = _one_edge(); g = A.RunGroups.of_sample(trie, A.trie_ranks(trie), np.ones(60_000, np.int32), [])\n"
        "used = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()\n"
        "hard = resource.getrlimit(resource.RLIMIT_AS)[1]\n"
        "resource.setrlimit(resource.RLIMIT_AS, (used + (512 << 20), hard))\n"
        "rc = lib().agpt_b200_trie_group_prepare(g._h, 0, 64, 0, 128, C.byref(RunGroupInfo()))\n"
        "msg = lib().agpt_b200_last_error().decode()\n"
        "up = lib().agpt_b200_trie_group_upload(g._h, 0, 16, None, C.byref(C.c_void_p()))\n"
        "resource.setrlimit(resource.RLIMIT_AS, (hard, hard))\n"
        "print(rc, '|', msg, '|', up)\n")
    got = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0, got.stderr[-2000:]
    rc, msg, up = got.stdout.strip().split("\n")[-1].split(" | ")
    assert int(rc) == -5 and "out of host memory" in msg and int(up) == -1          # and nothing is left that upload would take
