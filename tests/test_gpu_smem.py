"""The SMEM / MEM kernels at the sizes where they can go wrong: reads around min_len, groups
of reads that one warp shares, reads that leave the shared sweep early, late and never,
segment edges, and interval sets that outgrow every area.  Bytes equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, _Handle, _build, _header_fields
from haystackfm_b200._lib import pack_queries

pytestmark = pytest.mark.gpu


def _index(kind):
    if kind == "acgt":               # narrow records
        ref = synth.repeat_reference(total=300_000, n_contigs=3, seed=5)
        tag = 1
    elif kind == "acgt_iupac":       # narrow records, query codes that match several symbols
        ref = synth.repeat_reference(total=300_000, n_contigs=3, seed=6)
        tag = 0
    elif kind == "few_codes":        # wide records, no N runs: reads leave the shared sweep
        ref = synth.iupac_reference(total=300_000, n_contigs=3, n_frac=0.0, iupac_frac=0.002, seed=7)
        tag = 0
    else:                            # wide records, N runs longer than the reads
        ref = synth.iupac_reference(total=300_000, n_contigs=3, n_run_mean=120, seed=8)
        tag = 0
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), tag, KIND_BIDIR)
    return ref, b


def _check(oracle, b, h, reads, min_len, mode, cap=64):
    flat, off = pack_queries(reads)
    bounds = _header_fields(b, 4)[2]
    want = oracle.OracleIndex(b, KIND_BIDIR).mems_packed(flat, off, min_len, mode, bounds, cap, threads=8)
    got = h.mems_packed(flat, off, min_len, mode, bounds, cap)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("kind", ["acgt", "acgt_iupac", "few_codes", "n_runs"])
def test_read_lengths_and_group_sizes(oracle, kind):
    ref, b = _index(kind)
    h = _Handle(b, KIND_BIDIR)
    rng = np.random.default_rng(1)
    rows = synth.sample_reads(ref, n_reads=400, read_len=150, n_rate=0.003, seed=2)
    lens = [0, 1, 18, 19, 20, 31, 32, 33, 63, 64, 65, 150]
    ragged = [r[:lens[k % len(lens)]] for k, r in enumerate(rows)]
    noise = [rng.integers(1, 5, size=60).astype(np.uint8) for _ in range(8)]
    odd = [np.array([0, 1, 2], np.uint8), np.full(40, 16, np.uint8), np.concatenate([rows[0][:70], [0], rows[0][70:]])]
    for n in (1, 2, 31, 32, 33):
        _check(oracle, b, h, ragged[:n], 19, 0)
    _check(oracle, b, h, ragged + noise + odd, 19, 0)
    _check(oracle, b, h, ragged[:60] + noise + odd, 1, 0, cap=4)
    _check(oracle, b, h, ragged[:40] + noise + odd, 12, 1)
    for min_len in (6, 7, 8):                                           # around the k-mer table's k (7 here)
        _check(oracle, b, h, ragged[:60] + noise + odd, min_len, 0, cap=4)
    _check(oracle, b, h, [r[:60] for r in rows[:24]], 61, 0)            # nothing is long enough
    _check(oracle, b, h, ragged[:24], 0, 0)                             # min_len 0: no results
    # a batch large enough for groups formed by prefix
    if kind in ("few_codes", "n_runs"):
        many = synth.sample_reads(ref, n_reads=12_000, read_len=90, seed=3)
        _check(oracle, b, h, list(many), 19, 0, cap=2)


@pytest.mark.parametrize("kind", ["acgt", "n_runs"])
def test_segment_edges(oracle, kind):
    """Reads of 2 * seg_len and around it, whole matches that span many segments, and errors
    right at segment boundaries, with short reads between them."""
    ref, b = _index(kind)
    h = _Handle(b, KIND_BIDIR)
    t = ref.truth[0]
    rng = np.random.default_rng(4)
    reads = []
    for n in (127, 128, 129, 191, 192, 193, 64 * 7, 64 * 7 + 1):
        a = int(rng.integers(0, len(t) - n))
        exact = t[a:a + n].copy()
        reads.append(exact)
        for at in (63, 64, 65, n - 20, n - 19):
            e = exact.copy()
            e[at] = e[at] % 4 + 1
            reads.append(e)
        reads.append(exact[:40])
    for seg in (64, 512):
        h.set_tuning(3, seg)
        _check(oracle, b, h, reads, 19, 0)
        _check(oracle, b, h, reads[:20], 25, 1)


def test_iupac_codes_of_one_symbol(oracle):
    """A text of two bases: query codes such as R match one symbol of it, others two or none,
    inside long one-row matches and next to sequence ends."""
    rng = np.random.default_rng(12)
    seqs = [rng.integers(1, 3, size=n).astype(np.uint8) for n in (40_000, 90, 3000)]
    b = _build([al.DnaSequence(c) for c in seqs], FmIndexConfig(sa_sample_rate=8), 0, KIND_BIDIR)
    h = _Handle(b, KIND_BIDIR)
    reads = []
    for k in range(160):
        s = seqs[k % 3]
        n = int(rng.integers(30, 90))
        a = int(rng.integers(0, len(s) - n + 1)) if k % 5 else len(s) - n
        r = np.concatenate([s[a:a + n], rng.integers(1, 3, size=k % 4).astype(np.uint8)])
        for at in rng.integers(0, len(r), size=k % 6):
            r[at] = rng.integers(1, 16)
        reads.append(r)
    for min_len in (1, 12, 25):
        _check(oracle, b, h, reads, min_len, 0)
    _check(oracle, b, h, reads, 20, 1)


def test_set_overflow_tiers(oracle):
    """N stretches in the reads grow interval sets past the shared node lists and the
    per-thread sets; the reads around them keep their results."""
    ref, b = _index("n_runs")
    h = _Handle(b, KIND_BIDIR)
    rows = synth.sample_reads(ref, n_reads=70, read_len=100, seed=9)
    reads = [r.copy() for r in rows]
    for k in range(0, 70, 7):
        reads[k][:7] = 5
        reads[k + 1][60:67] = 5
    _check(oracle, b, h, reads, 19, 0)
    _check(oracle, b, h, reads[:24], 19, 1, cap=4)


@pytest.mark.parametrize("kind", ["acgt", "few_codes", "n_runs"])
def test_layout_blob_keeps_its_form(oracle, kind):
    """The device-layout blob holds counts before each record's first row and whole planes,
    whatever form the device keeps: the counts of code 1 are the oracle's ranks, and a
    handle loaded from the blob exports the same bytes and gives the same results."""
    ref, b = _index(kind)
    h = _Handle(b, KIND_BIDIR)
    blob = h.export_layout()
    again = _Handle.from_layout(blob)
    assert again.export_layout() == blob
    o = oracle.OracleIndex(b, KIND_BIDIR)
    arr = np.frombuffer(blob, np.uint8)
    size = 32 if kind == "acgt" else 96
    nblk = (o.text_len + 63) // 64
    # the seven buffer sizes (the Occ records' first), then the records
    at = blob.index(np.uint64(nblk * size).tobytes(), 16)
    rec = arr[at + 56:at + 56 + nblk * size].reshape(nblk, size)
    for blk in (0, 1, nblk // 2, nblk - 1):
        if kind == "acgt":               # u16 counts of codes 1..4 from the superblock's start
            counts = rec[blk, :8].copy().view(np.uint16)
            first = blk // 1024 * 65536
            for c in (1, 2, 3, 4):
                assert counts[c - 1] == o.rank(c, blk * 64) - o.rank(c, first)
        else:                            # u32 counts of every code
            counts = rec[blk, :64].copy().view(np.uint32)
            for c in (0, 1, 4, 5, 9):
                assert counts[c] == o.rank(c, blk * 64)
    reads = list(synth.sample_reads(ref, n_reads=50, read_len=100, seed=11))
    _check(oracle, b, again, reads, 19, 0)
