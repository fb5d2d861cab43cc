"""The work areas of small ACGT batches follow the batch, not the threads that it is spread over,
and hit lists as long as a job's positions are enough."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, _Handle, _build, _header_fields
from haystackfm_b200._lib import pack_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tag", [0, 1])
@pytest.mark.parametrize("nq", [1, 32, 250])
def test_small_batch_on_a_fresh_handle(oracle, nq, tag):
    ref = synth.repeat_reference(total=400_000, n_contigs=3, seed=9)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), tag, KIND_BIDIR)
    flat, off, lens = synth.sample_mixed_reads(ref, n_reads=nq, seed=6, n_rate=0.002 if tag == 0 else 0.0)
    bounds = _header_fields(b, 4)[2]
    h = _Handle(b, KIND_BIDIR)
    got = h.mems_packed(flat, off, 19, 0, bounds, 16)
    want = oracle.OracleIndex(b, KIND_BIDIR).mems_packed(flat, off, 19, 0, bounds, 16, threads=8)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    # lists of 128 hits a segment of 64 codes are 64 bytes a code; with codes of several symbols
    # the jobs that hold one have 1,024 hits and two sets of 768 intervals
    jobs = int(np.sum(np.maximum(1, -(-lens // 64))))
    room = 200e6 if tag == 0 else 16e6 + 8192 * jobs
    assert h.device_bytes()["work"] <= room


def test_a_hit_at_every_position(oracle):
    """Jobs of 128 codes with a result at each place where one can start."""
    rng = np.random.default_rng(3)
    a = rng.integers(1, 5, size=40_000).astype(np.uint8)
    b = _build([al.DnaSequence(a)], FmIndexConfig(sa_sample_rate=16), 1, KIND_BIDIR)
    h = _Handle(b, KIND_BIDIR)
    o = oracle.OracleIndex(b, KIND_BIDIR)
    reads = [rng.integers(1, 5, size=n).astype(np.uint8) for n in (64, 127, 128, 129, 640)]
    flat, off = pack_queries(reads)
    for min_len in (1, 2, 5):
        for mode in (0, 1):
            for g, w in zip(h.mems_packed(flat, off, min_len, mode, None, 4), o.mems_packed(flat, off, min_len, mode, None, 4)):
                assert np.array_equal(g, w)
