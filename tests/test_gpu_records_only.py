"""An index loaded without the arrays kept beside its records: the memory is not taken, and
every search and resolve gives the same results by steps and walks."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200._lib import HFM_FLAG_RECORDS_ONLY, pack_queries
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, KIND_FM, _Handle, _build, _header_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["acgt", "acgt_iupac", "n_runs"])
def test_records_only(oracle, kind):
    if kind == "n_runs":
        ref, tag = synth.iupac_reference(total=300_000, n_contigs=3, n_run_mean=60, seed=8), 0
    else:
        ref, tag = synth.repeat_reference(total=300_000, n_contigs=3, seed=5), 1 if kind == "acgt" else 0
    seqs = [al.DnaSequence(c) for c in ref.contigs]
    cfg = FmIndexConfig(sa_sample_rate=16, lookup_depth=6)
    b = _build(seqs, cfg, tag, KIND_BIDIR)
    o = oracle.OracleIndex(b, KIND_BIDIR)
    reads = list(synth.sample_reads(ref, n_reads=80, read_len=150, n_rate=0.003, seed=2))
    reads += [r[:k] for k, r in enumerate(reads[:40])]
    truth = max(ref.truth, key=len)
    reads += [truth[:1500].copy(), truth[700:1000].copy()]
    flat, off = pack_queries(reads)
    cut, cut_off = pack_queries([r[:28] for r in reads])
    bounds = _header_fields(b, 4)[2]
    full = _Handle(b, KIND_BIDIR)
    blob = full.export_layout()
    handles = [_Handle(b, KIND_BIDIR, 0, HFM_FLAG_RECORDS_ONLY), _Handle.from_layout(blob, 0, HFM_FLAG_RECORDS_ONLY)]
    handles.append(handles[0].share())
    for h in handles:
        for min_len, mode in ((19, 0), (12, 1)):
            want = o.mems_packed(flat, off, min_len, mode, bounds, 64, threads=8)
            for variant in (3, 2):
                h.set_tuning(variant, 64)
                for g, w in zip(h.mems_packed(flat, off, min_len, mode, bounds, 64), want):
                    assert np.array_equal(g, w)
        for g, w in zip(h.locate_packed(cut, cut_off, 64), o.locate_packed(cut, cut_off, 64)):
            assert np.array_equal(g, w)
        assert np.array_equal(h.count_packed(cut, cut_off), o.count_packed(cut, cut_off))
    assert handles[0].export_layout() == blob
    # 4 bytes a row less at least
    assert handles[0].device_bytes()["index"] + 4 * o.text_len <= full.device_bytes()["index"]


def test_records_only_forward_index(oracle):
    ref = synth.repeat_reference(total=200_000, n_contigs=2, seed=6)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=32), 1, KIND_FM)
    o = oracle.OracleIndex(b, KIND_FM)
    h = _Handle(b, KIND_FM, 0, HFM_FLAG_RECORDS_ONLY)
    flat, off = pack_queries([r[:40] for r in synth.sample_reads(ref, n_reads=200, read_len=60, seed=3)])
    for g, w in zip(h.locate_packed(flat, off, 0), o.locate_packed(flat, off, 0)):
        assert np.array_equal(g, w)
    assert np.array_equal(h.count_packed(flat, off), o.count_packed(flat, off))


def test_arrays_beside_the_records_have_no_slack():
    """They never grow: 4 bytes a row, and on an ACGT text what its length says."""
    ref = synth.repeat_reference(total=3_000_000, n_contigs=2, seed=6)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=32), 1, KIND_BIDIR)
    full, bare = _Handle(b, KIND_BIDIR), _Handle(b, KIND_BIDIR, 0, HFM_FLAG_RECORDS_ONLY)
    n = 3_000_002
    k = max(k for k in range(2, 14) if 16 << 2 * k <= 2 * n)
    seen = min(4 ** k for k in range(3, 18) if 4 ** k >= 4 * n) // 8
    beside = (4 * n + 16) + (n // 32 + 2) * 16 + (16 << 2 * k) + seen
    assert full.device_bytes()["index"] - bare.device_bytes()["index"] == beside
