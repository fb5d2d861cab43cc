"""Counts of patterns longer than what the comparison with the text takes at a time, on ACGT
texts: every length around its words, matches that reach the start of the text or of a sequence
and patterns that would go past it, mismatches and codes of several symbols at every place."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import FmIndex, FmIndexConfig, KIND_FM, _build

pytestmark = pytest.mark.gpu


def _index(tag, seed=3):
    rng = np.random.default_rng(seed)
    seqs = [rng.integers(1, 5, size=n).astype(np.uint8) for n in (30_000, 400, 9000)]
    return seqs, _build([al.DnaSequence(s) for s in seqs], FmIndexConfig(sa_sample_rate=16, lookup_depth=4), tag, KIND_FM)


@pytest.mark.parametrize("tag", [0, 1])
def test_long_counts_match_oracle(oracle, tag):
    seqs, b = _index(tag)
    rng = np.random.default_rng(4)
    text = seqs[0]
    pats = []
    for n in list(range(30, 36)) + list(range(44, 50)) + list(range(76, 82)) + [128, 150, 320, 399, 400]:
        a = int(rng.integers(0, len(text) - n))
        pats.append(text[a:a + n].copy())
        for s in seqs:                                   # from the first code of a sequence on, and past it
            if n <= len(s):
                pats.append(s[:n].copy())
                pats.append(np.concatenate([rng.integers(1, 5, size=3).astype(np.uint8), s[:n - 3]]))
        for at in {0, 1, 7, n // 2, n - 33, n - 32, n - 31, n - 14, n - 1}:
            if 0 <= at < n:
                for code in (5, 6, 14, 0, 16, int(text[a + at]) % 4 + 1):
                    p = text[a:a + n].copy()
                    p[at] = code
                    pats.append(p)
        p = text[a:a + n].copy()                         # many of them, and one that does not match
        p[rng.random(n) < 0.3] = 5
        pats.append(p)
        q = p.copy()
        q[3] = text[a + 3] % 4 + 1
        pats.append(q)
    flat, off = pack_queries(pats)
    got = FmIndex.from_bytes(b).handle.count_packed(flat, off)
    assert np.array_equal(got, oracle.OracleIndex(b, KIND_FM).count_packed(flat, off, threads=8))
    assert (got == 1).any() and (got == 0).any()


@pytest.mark.parametrize("at", [8, 1000, 1950])
def test_work_is_linear_in_the_pattern(at):
    """A code of several symbols does not make the codes around it be looked at again."""
    seqs, b = _index(0)
    n, m = 200, 2000
    pats = [seqs[0][k * 100:k * 100 + m].copy() for k in range(n)]
    for p in pats:
        p[at] = 5
    flat, off = pack_queries(pats)
    h = FmIndex.from_bytes(b).handle
    h.set_counters(True)
    assert (h.count_packed(flat, off) == 1).all()
    assert h.stats().occ_touches <= n * 2 * m            # two records a code at most
