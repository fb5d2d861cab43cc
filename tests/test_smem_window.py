"""The window / forward / next search that the SMEM kernels run, restated over a plain
"does this string occur" predicate, finds the oracle's find_smems and find_mems, whole or cut
into segments, on texts with ambiguity codes and sentinels."""
from __future__ import annotations

import random

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from tests.helpers import concat, enc, naive_positions, seqs_codes


def window_search(occurs, n, min_len, start=0, stop=None):
    """Results of q[0, n) that start in [start, stop): occurs(s, e) tells whether q[s, e) does."""
    stop = n if stop is None else stop
    i, first, out = start, start > 0, []
    while i < stop and n - i >= min_len:
        k = i + min_len
        while k > i and occurs(k - 1, i + min_len):
            k -= 1
        if k > i:
            i, first = k, False
            continue
        e = i + min_len
        while e < n and occurs(i, e + 1):
            e += 1
        if not (first and occurs(i - 1, e)):
            out.append((i, e))
        first = False
        if e == n:
            break
        k = e + 1
        while k > i + 1 and occurs(k - 1, e + 1):
            k -= 1
        i = k
    return out


@pytest.mark.parametrize("seed", range(6))
def test_window_search_finds_the_oracles_mems(oracle, seed):
    rng = random.Random(seed)
    letters = ["ACGT", "ACGTN", "ACGTACGTACGTRYSWKMBDHVN"][seed % 3]
    seqs = ["".join(rng.choice(letters) for _ in range(rng.randint(20, 150))) for _ in range(rng.randint(1, 4))]
    tag = 1 if seed == 3 else 0
    text, _ = concat(seqs)
    b = oracle.build_index_bytes(seqs_codes(seqs), rate=4, tag=tag, kind=1)
    o = oracle.OracleIndex(b, 1)
    for _ in range(12):
        n = rng.randint(1, 40)
        src = rng.choice(seqs)
        a = rng.randrange(len(src))
        q = (list(enc(src[a:a + n])) + [rng.randint(1, 15) for _ in range(n)])[:n]
        for k in range(n):
            if rng.random() < 0.08:
                q[k] = rng.randint(1, 15)
        q = np.array(q, np.uint8)
        memo = {}

        def occurs(s, e):
            if (s, e) not in memo:
                memo[s, e] = len(naive_positions(text, q[s:e], tag)) > 0
            return memo[s, e]

        for min_len in (1, 3, 7):
            got = window_search(occurs, n, min_len)
            for mode in (0, 1):
                hit_off, hits, _ = o.mems_packed(q, np.array([0, n], np.uint64), min_len, mode, [], 8)
                want = sorted({(int(h[0]), int(h[1])) for h in hits})
                assert got == want
            for seg in (3, 8, 16):
                cut = [r for a in range(0, n, seg) for r in window_search(occurs, n, min_len, a, min(n, a + seg))]
                assert cut == got
