"""The arrays of a RadixTrie are the native trie's own memory, read-only: they outlive close() and the RadixTrie, below and above the
size from which they lie in huge pages (262,144 characters)."""
import gc

import numpy as np
import pytest

import agpt_b200 as A

NAMES = ("parent", "edge_len", "edge_mass", "edge_start", "edge_off", "edge_tok", "cnt_off", "cnt_tok", "cnt_val")


def _suffix_order(c, key_len):
    n = c.size
    pad = np.full(n + key_len, -1, np.int32)
    pad[:n] = c
    rows = np.lib.stride_tricks.sliding_window_view(pad, key_len)[:n - 1]
    sa = np.lexsort(rows.T[::-1]).astype(np.int32)
    a, b = rows[sa[:-1]], rows[sa[1:]]
    same = (a == b) & (a >= 0)
    return sa, np.concatenate([[0], np.where(same.all(1), key_len, same.argmin(1))]).astype(np.int32)


@pytest.mark.parametrize("chars", [200, 12_000])
def test_arrays_outlive_the_trie(chars):
    corpus, depth = A.synth_markov_corpus(chars, 65, 3), 32
    trie = A.RadixTrie.from_suffix_order(corpus, depth, *_suffix_order(corpus, depth + 1))
    assert (trie.total_edge_chars > 262_144) == (chars == 12_000)
    got = {n: getattr(trie, n) for n in NAMES}
    trie.close()
    del trie
    gc.collect()
    other = A.RadixTrie.build(corpus, depth)
    for n in NAMES:
        assert np.array_equal(got[n], getattr(other, n)), n


def test_arrays_are_read_only():
    """Writing into one would change what the native calls on the trie see."""
    corpus = A.synth_markov_corpus(300, 12, 2)
    trie = A.RadixTrie.build(corpus, 6)
    for n in NAMES:
        a = getattr(trie, n)
        with pytest.raises(ValueError):
            a[0] = 7
        with pytest.raises(ValueError):
            a.setflags(write=True)
        b = a.copy()
        b[0] = 7                                        # a copy is the caller's
    assert np.array_equal(trie.edge_mass, A.RadixTrie.build(corpus, 6).edge_mass)
