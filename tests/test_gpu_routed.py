"""A first call on a fresh handle that routes most of a batch to the warp kernel: the areas of
the shared first sweep are sized for the reads that it takes, whichever reads those are."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import BidirFmIndex, FmIndexConfig, KIND_BIDIR, _build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("routed", [0.95, 0.5, 0.0])
def test_mostly_routed_first_call(oracle, routed):
    ref = synth.iupac_reference(total=300_000, n_contigs=3, n_run_mean=60, seed=21)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), 0, KIND_BIDIR)
    reads = list(synth.sample_reads(ref, n_reads=4000, read_len=60, seed=22))
    truth = max(ref.truth, key=len)
    for k in range(8):                                   # segments in front of the reads in one piece
        reads[500 * k + 3] = truth[1000 * k:1000 * k + 1500].copy()
    flat, off = pack_queries(reads)
    nq = len(reads)
    # the reads that the sweep takes are the batch's last ones: the highest read numbers
    n_warp = int(nq * routed)
    idx = BidirFmIndex.from_bytes(b)
    bounds = idx.seq_boundaries()
    got = idx.handle.mems_sched_packed(flat, off, 19, 0, bounds, 16, order=np.arange(nq), n_warp=n_warp)
    want = oracle.OracleIndex(b, KIND_BIDIR).mems_packed(flat, off, 19, 0, bounds, 16, threads=8)
    for g, w in zip(got[:3], want):
        assert np.array_equal(g, w)
