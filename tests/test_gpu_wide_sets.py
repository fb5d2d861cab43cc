"""Backward search whose interval sets run from one to thousands of intervals, in the thread
and the warp tier: the same hits in the same order as the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import KIND_FM, _Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("codes", [(1, 2, 3, 4), (1, 2, 3, 4, 15), (1, 4, 5, 9, 12), tuple(range(1, 16))])
@pytest.mark.parametrize("size", [40, 700, 20_000])
def test_wide_sets(oracle, codes, size):
    rng = np.random.default_rng(size + len(codes))
    seqs = [rng.choice(codes, size=n).astype(np.uint8) for n in (size, size // 3, 1)]
    b = oracle.build_index_bytes(seqs, rate=4, kind=KIND_FM)
    o, h = oracle.OracleIndex(b, KIND_FM), _Handle(b, KIND_FM)
    qs = [rng.integers(1, 16, size=int(n)).astype(np.uint8) for n in rng.integers(1, 12, size=300)]
    qs += [np.full(n, 15, np.uint8) for n in range(1, 14)]                 # N: matches everything
    qs += [np.array([15, c] * 4, np.uint8) for c in range(1, 16)] + [np.array([c, 15, 15], np.uint8) for c in range(1, 16)]
    flat, off = pack_queries(qs)
    assert np.array_equal(h.count_packed(flat, off), o.count_packed(flat, off))
    for g, w in zip(h.locate_packed(flat, off, 0), o.locate_packed(flat, off, 0)):
        assert np.array_equal(g, w)
