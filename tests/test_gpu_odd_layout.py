"""Device-layout blobs of consistent sizes with damaged contents: loading reads and writes only
its own buffers, and what does not depend on the damage is answered as before."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, _Handle, _build, _header_fields

pytestmark = pytest.mark.gpu

DEV_FM = 16                       # the first direction's scalars: 6 pointers, then u32 fields
SAMPLE_RATE, C_ARRAY = DEV_FM + 56, DEV_FM + 80


def _index(kind):
    if kind == "acgt":
        ref, tag = synth.repeat_reference(total=200_000, n_contigs=3, seed=5), 1
    else:
        ref, tag = synth.iupac_reference(total=200_000, n_contigs=3, n_run_mean=60, seed=8), 0
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), tag, KIND_BIDIR)
    return ref, b


def _sections(blob, n, size):
    """Offsets of the first direction's buffers."""
    nblk = (n + 63) // 64
    at = bytes(blob).index(np.uint64(nblk * size).tobytes(), 16)
    sizes = blob[at:at + 56].copy().view(np.uint64).astype(int)
    return at + 56 + np.concatenate([[0], np.cumsum(sizes)])


@pytest.mark.parametrize("kind", ["acgt", "n_runs"])
@pytest.mark.parametrize("damage", ["marks_past_text", "value_places", "sample_rate", "record_counts", "code_counts"])
def test_damaged_blob_loads(oracle, kind, damage):
    ref, b = _index(kind)
    o = oracle.OracleIndex(b, KIND_BIDIR)
    n = o.text_len
    assert n % 64                                        # the last word has room past the text
    blob = np.frombuffer(_Handle(b, KIND_BIDIR).export_layout(), np.uint8).copy()
    sec = _sections(blob, n, 32 if kind == "acgt" else 96)
    ssa = blob[sec[2]:sec[3]].view(np.uint32).reshape(-1, 4)
    if damage == "marks_past_text":
        word = (1 << 64) - (1 << (n % 64))
        ssa[-1, 0] |= word & 0xFFFFFFFF
        ssa[-1, 1] |= word >> 32
    elif damage == "value_places":
        ssa[3::7, 2] = 0xFFFFFF00
    elif damage == "sample_rate":
        blob[SAMPLE_RATE:SAMPLE_RATE + 4].view(np.uint32)[0] = 0x7FFFFFFF
    elif damage == "record_counts":
        rec = blob[sec[0]:sec[1]].reshape(-1, 32 if kind == "acgt" else 96)
        rec[5::3, :8 if kind == "acgt" else 64] = 0xF0
    else:
        blob[C_ARRAY:C_ARRAY + 64].view(np.uint32)[3:] = 0xFFFFFFF0
    h = _Handle.from_layout(blob.tobytes())
    reads = list(synth.sample_reads(ref, n_reads=60, read_len=100, seed=11))
    flat, off = pack_queries(reads)
    bounds = _header_fields(b, 4)[2]
    cut, cut_off = pack_queries([r[:32] for r in reads])
    if damage in ("marks_past_text", "value_places", "sample_rate"):     # searches use none of it
        for g, w in zip(h.mems_packed(flat, off, 19, 0, None, 64), o.mems_packed(flat, off, 19, 0, None, 64, threads=8)):
            assert np.array_equal(g, w)
        assert np.array_equal(h.count_packed(cut, cut_off), o.count_packed(cut, cut_off))
    if damage == "marks_past_text":
        for g, w in zip(h.locate_packed(cut, cut_off, 64), o.locate_packed(cut, cut_off, 64)):
            assert np.array_equal(g, w)
    del h
    good = _Handle(b, KIND_BIDIR)
    for g, w in zip(good.mems_packed(flat, off, 19, 0, bounds, 64), o.mems_packed(flat, off, 19, 0, bounds, 64, threads=8)):
        assert np.array_equal(g, w)
