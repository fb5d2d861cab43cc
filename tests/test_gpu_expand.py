"""Positions of deduplicated hits at the edges of the copy's blocks: segments of one position,
more segments in a block than it stages, and segments longer than several blocks, mixed."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import _lib as L
from haystackfm_b200.fm_index import KIND_FM, _Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", ["short", "long", "mixed"])
def test_dedup_copy(oracle, lens):
    rng = np.random.default_rng(5)
    seqs = [rng.integers(1, 5, size=n).astype(np.uint8) for n in (40_000, 37, 9000)]
    b = oracle.build_index_bytes(seqs, rate=8, kind=KIND_FM)
    o, h = oracle.OracleIndex(b, KIND_FM), _Handle(b, KIND_FM, 0, L.HFM_FLAG_DEDUP_ALWAYS)
    short = [seqs[0][a:a + 12] for a in rng.integers(0, 39_000, size=9_000)]          # one position each
    long_ = [np.array([c], np.uint8) for c in (1, 2, 3, 4)] * 6                       # ~12,000 positions each
    qs = {"short": short, "long": long_, "mixed": short[:3000] + long_[:5] + short[3000:6000] + long_[5:9] + short[:1]}[lens]
    flat, off = L.pack_queries(qs)
    for cap in (0, 1, 700):
        for g, w in zip(h.locate_packed(flat, off, cap), o.locate_packed(flat, off, cap, threads=8)):
            assert np.array_equal(g, w)
