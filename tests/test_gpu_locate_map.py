"""Locate without deduplication, at the edges of the resolve's blocks of 256 positions: queries
of one position, of exactly a block, of several blocks and of none (the last ones included), so
that a block begins inside, at the start and at the end of a query's interval."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import _lib as L
from haystackfm_b200.fm_index import KIND_FM, _Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [0, 1, 255, 256, 257])
@pytest.mark.parametrize("codes", [4, 15])
def test_blocks_of_positions(oracle, cap, codes):
    rng = np.random.default_rng(cap + codes)
    seqs = [rng.integers(1, codes + 1, size=n).astype(np.uint8) for n in (6000, 41)]
    b = oracle.build_index_bytes(seqs, rate=4, kind=KIND_FM)
    o, h = oracle.OracleIndex(b, KIND_FM), _Handle(b, KIND_FM, 0, L.HFM_FLAG_DEDUP_NEVER)
    one = [seqs[0][a:a + 20] for a in rng.integers(0, 5900, size=300)]
    many = [np.array([c], np.uint8) for c in range(1, 5)]
    none = [np.array([1, 2, 3, 4] * 12, np.uint8)]
    for qs in (one[:1], many[:1], none, one[:255] + many + one[255:], one[:256] + none + many, many * 3 + none * 2,
               none + one[:257] + none):
        flat, off = L.pack_queries(qs)
        for g, w in zip(h.locate_packed(flat, off, cap), o.locate_packed(flat, off, cap)):
            assert np.array_equal(g, w)
