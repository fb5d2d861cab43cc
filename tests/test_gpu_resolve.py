"""Every row of the index resolves to the oracle's position, whether the handle keeps the
whole suffix array or walks (a sample rate above its limit), sentinel rows and the ends of
short sequences included."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import KIND_FM, _Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [1, 3, 64, 1024, 1025])
@pytest.mark.parametrize("codes", [4, 15])
def test_every_row_resolves(oracle, rate, codes):
    rng = np.random.default_rng(rate * 100 + codes)
    lens = [1, 2, 63, 64, 65, 700, 1, 3000, 5]
    seqs = [rng.integers(1, codes + 1, size=n).astype(np.uint8) for n in lens]
    b = oracle.build_index_bytes(seqs, rate=rate, kind=KIND_FM)
    o, h = oracle.OracleIndex(b, KIND_FM), _Handle(b, KIND_FM)
    qs = [np.zeros(0, np.uint8)] + [np.array([c], np.uint8) for c in range(1, codes + 1)] + [s[-3:] for s in seqs]
    flat, off = pack_queries(qs)
    for cap in (0, 2):
        for g, w in zip(h.locate_packed(flat, off, cap), o.locate_packed(flat, off, cap)):
            assert np.array_equal(g, w)
