"""The per-read work log on texts with ambiguity codes: the call takes the same path as one without
a log, and what a read is charged does not depend on the reads that share its sweep."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import BidirFmIndex, FmIndexConfig, KIND_BIDIR, _build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["few_codes", "n_runs"])
def case(request):
    kw = dict(n_frac=0.0, iupac_frac=0.002) if request.param == "few_codes" else dict(n_run_mean=60)
    ref = synth.iupac_reference(total=300_000, n_contigs=3, seed=8, **kw)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), 0, KIND_BIDIR)
    reads = list(synth.sample_reads(ref, n_reads=3000, read_len=100, sub_rate=0.02, n_rate=0.0, seed=2))
    return BidirFmIndex.from_bytes(b), reads


def test_log_takes_the_path_of_other_calls(case):
    idx, reads = case
    h = idx.handle
    flat, off = pack_queries(reads)
    bounds = idx.seq_boundaries()
    h.set_counters(True)
    want = h.mems_packed(flat, off, 19, 0, bounds, 8)
    touches = h.stats().occ_touches
    h.set_counters(False)
    got = h.mems_sched_packed(flat, off, 19, 0, bounds, 8, work_log=True)
    for g, w in zip(got[:3], want):
        assert np.array_equal(g, w)
    assert h.stats().occ_touches == touches
    # shared nodes are charged to every read that holds them
    assert got[3][:, 0].sum(dtype=np.uint64) >= touches
    assert (got[3][:, 0] > 0).all()


def test_log_does_not_depend_on_the_group(case):
    idx, reads = case
    h = idx.handle
    bounds = idx.seq_boundaries()
    flat, off = pack_queries(reads)
    rng = np.random.default_rng(0)
    logs = [h.mems_sched_packed(flat, off, 19, 0, bounds, 8, order=order, work_log=True)[3]
            for order in (None, rng.permutation(len(reads)), np.arange(len(reads))[::-1])]
    few = reads[:40]                                     # a block each
    flat, off = pack_queries(few)
    alone = h.mems_sched_packed(flat, off, 19, 0, bounds, 8, work_log=True)[3]
    stayed = (alone[:, 3] & 1) == 0
    assert stayed.any()
    for log in logs:
        same = stayed & ((log[:40, 3] & 1) == 0)
        assert same.any()
        assert np.array_equal(log[:40][same], alone[same])
    both = ((logs[0][:, 3] | logs[1][:, 3] | logs[2][:, 3]) & 1) == 0
    assert np.array_equal(logs[0][both], logs[1][both]) and np.array_equal(logs[0][both], logs[2][both])
