"""Results of the host-buffer calls: large ones are views of the library's block, which stays
valid while any of them lives and is given back afterwards; small ones and everything past the
bound are copies.  The values are the same either way."""
from __future__ import annotations

import gc

import numpy as np
import pytest

from haystackfm_b200 import fm_index as fi
from haystackfm_b200 import synth
from haystackfm_b200 import alphabet as al
from haystackfm_b200._lib import pack_queries

pytestmark = pytest.mark.gpu


def test_views_live_and_are_given_back(monkeypatch):
    rng = np.random.default_rng(3)
    seqs = [rng.integers(1, 5, size=60_000).astype(np.uint8) for _ in range(2)]
    b = fi._build([al.DnaSequence(s) for s in seqs], fi.FmIndexConfig(sa_sample_rate=8), 1, fi.KIND_BIDIR)
    h = fi._Handle(b, fi.KIND_BIDIR)
    flat, off = pack_queries([np.array([c], np.uint8) for c in (1, 2, 3, 4)] * 4)     # ~480,000 positions
    gc.collect()
    before = dict(fi._viewed)
    counts, offsets, pairs = h.locate_packed(flat, off)
    assert sum(fi._viewed.values()) > sum(before.values())
    kept = [a.copy() for a in (counts, offsets, pairs)]
    for _ in range(3):                                     # later calls leave a held result alone
        h.locate_packed(flat[:4], off[:5])
        h.mems_packed(flat, off, 1, 0, [120_002], 1000)
    for a, k in zip((counts, offsets, pairs), kept):
        assert np.array_equal(a, k)
    tail = pairs[-5:]
    del counts, offsets, pairs, a
    gc.collect()
    assert np.array_equal(tail, kept[2][-5:])              # any view keeps the block
    del tail
    gc.collect()
    assert fi._viewed == before
    monkeypatch.setattr(fi, "RESULT_VIEW_MAX", 0)          # past the bound: copies of the same values
    again = h.locate_packed(flat, off)
    assert fi._viewed == before
    for a, k in zip(again, kept):
        assert np.array_equal(a, k)
    empty = h.locate_packed(np.zeros(1, np.uint8), np.zeros(1, np.uint64))
    assert [len(x) for x in empty] == [0, 1, 0] and empty[2].shape == (0, 2)
