"""Index bytes that pass the format checks without being an index of any text: the parts
disagree with one another.  Whatever such a handle answers, no search leaves its buffers: the
calls return, and a proper index is still searched correctly afterwards."""
from __future__ import annotations

import struct

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200._lib import pack_queries
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, KIND_FM, _Handle, _build

pytestmark = pytest.mark.gpu


def _two_texts(seed, p=(0.25, 0.25, 0.25, 0.25)):
    """A forward index of one text and a reverse index of another of the same length."""
    rng = np.random.default_rng(seed)
    a = rng.integers(1, 5, size=60_000).astype(np.uint8)
    c = rng.permutation(a) if p is None else rng.choice(np.arange(1, 5, dtype=np.uint8), size=len(a), p=p)
    cfg = FmIndexConfig(sa_sample_rate=16, lookup_depth=4)
    fwd = _build([al.DnaSequence(a)], cfg, 1, KIND_FM)
    rev = _build([al.DnaSequence(c[::-1].copy())], FmIndexConfig(sa_sample_rate=16), 1, KIND_FM)
    return a, c, struct.pack("<I", len(fwd)) + fwd + rev


def _search(h, reads):
    flat, off = pack_queries(reads)
    for variant, mode in ((3, 0), (2, 0), (3, 1)):
        h.set_tuning(variant, 64)
        hit_off, hits, pos = h.mems_packed(flat, off, 19, mode, None, 64)
        assert hit_off[-1] == len(hits)


def _proper(oracle, a, reads):
    b = _build([al.DnaSequence(a)], FmIndexConfig(sa_sample_rate=16, lookup_depth=4), 1, KIND_BIDIR)
    flat, off = pack_queries(reads)
    want = oracle.OracleIndex(b, KIND_BIDIR).mems_packed(flat, off, 19, 0, None, 64)
    for g, w in zip(_Handle(b, KIND_BIDIR).mems_packed(flat, off, 19, 0, None, 64), want):
        assert np.array_equal(g, w)


def test_directions_of_different_texts(oracle):
    """Same codes in another order: a match's forward row is that of some other string, and the
    text behind it may end long before the read does."""
    a, c, b = _two_texts(1, None)
    h = _Handle(b, KIND_BIDIR)
    reads = [a[k:k + 4000].copy() for k in range(0, 56_000, 3500)] + [c[k:k + 4000].copy() for k in range(0, 56_000, 3500)]
    reads += [a[-3000:].copy(), c[-3000:].copy(), a[-40:].copy(), c[-40:].copy()]
    _search(h, reads)
    _proper(oracle, a, reads)


@pytest.mark.parametrize("p", [(0.05, 0.05, 0.05, 0.85), (0.85, 0.05, 0.05, 0.05)])
def test_directions_of_different_code_counts(oracle, p):
    """A step of either direction counts from that direction's own rows of smaller codes."""
    a, c, b = _two_texts(2, p)
    h = _Handle(b, KIND_BIDIR)
    reads = [a[k:k + 300].copy() for k in range(0, 56_000, 3500)] + [c[k:k + 300].copy() for k in range(0, 56_000, 3500)]
    for codes in (1, 4):
        reads += [np.full(200, codes, np.uint8), np.concatenate([a[:100], np.full(100, codes, np.uint8)])]
    _search(h, reads)
    _proper(oracle, a, reads)


def test_directions_of_different_code_counts_wide(oracle):
    rng = np.random.default_rng(3)
    a = rng.integers(1, 16, size=20_000).astype(np.uint8)
    c = np.where(rng.random(len(a)) < 0.9, 15, a).astype(np.uint8)
    fwd = _build([al.DnaSequence(a)], FmIndexConfig(sa_sample_rate=16), 0, KIND_FM)
    rev = _build([al.DnaSequence(c[::-1].copy())], FmIndexConfig(sa_sample_rate=16), 0, KIND_FM)
    h = _Handle(struct.pack("<I", len(fwd)) + fwd + rev, KIND_BIDIR)
    reads = [a[k:k + 60].copy() for k in range(0, 18_000, 900)] + [c[k:k + 60].copy() for k in range(0, 18_000, 900)]
    flat, off = pack_queries(reads)
    for variant in (3, 2):
        h.set_tuning(variant, 64)
        hit_off, hits, pos = h.mems_packed(flat, off, 25, 0, None, 64)
        assert hit_off[-1] == len(hits)


def _fm_parts(b, at):
    """Offsets of the sampled values and of the marker words of the FmIndex at `at`."""
    o = at + 64 + 2 + 32
    o += 8 + 4 * struct.unpack_from("<Q", b, o)[0]
    o += 8 + struct.unpack_from("<Q", b, o)[0]
    o += 8 + 4 + 4
    n_ssa = struct.unpack_from("<Q", b, o)[0]
    ssa = o + 8
    n_vals = struct.unpack_from("<Q", b, ssa + n_ssa)[0]
    return ssa + n_ssa + 8, n_vals


@pytest.mark.parametrize("change", ["one_value", "swapped", "short_sequence_moved"])
def test_samples_that_disagree(oracle, change):
    """Sampled positions changed within the text: positions are those that walks to the samples
    give (the oracle's), searches do not depend on them."""
    rng = np.random.default_rng(5)
    seqs = [rng.integers(1, 5, size=n).astype(np.uint8) for n in (9000, 11, 13, 7000, 200)]
    b = bytearray(_build([al.DnaSequence(s) for s in seqs], FmIndexConfig(sa_sample_rate=32, lookup_depth=4), 1, KIND_BIDIR))
    at, n_vals = _fm_parts(b, 4)
    vals = np.frombuffer(b, "<u4", n_vals, at).copy()
    if change == "one_value":
        vals[vals == 3200] = 4800
    elif change == "swapped":
        i, k = np.flatnonzero(vals == 320)[0], np.flatnonzero(vals == 12_000 // 32 * 32)[0]
        vals[i], vals[k] = vals[k], vals[i]
    else:                                                # every sample of the second sequence
        start = len(seqs[0]) + 1
        inside = (vals >= start) & (vals < start + len(seqs[1]) + 1)
        assert inside.sum() >= 1
        vals[inside] += 3000
    b[at:at + 4 * n_vals] = vals.astype("<u4").tobytes()
    b = bytes(b)
    o = oracle.OracleIndex(b, KIND_BIDIR)
    h = _Handle(b, KIND_BIDIR)
    reads = [s[k:k + 120].copy() for s in seqs for k in range(0, max(1, len(s) - 120), 64)] + [s.copy() for s in seqs]
    flat, off = pack_queries(reads)
    bounds = np.cumsum([len(s) + 1 for s in seqs]).astype(np.uint32)
    for g, w in zip(h.mems_packed(flat, off, 11, 0, bounds, 64), o.mems_packed(flat, off, 11, 0, bounds, 64)):
        assert np.array_equal(g, w)
    assert np.array_equal(h.count_packed(flat, off), o.count_packed(flat, off))
    cut, cut_off = pack_queries([r[k:k + 9] for r in reads for k in range(0, len(r) - 8, 5)])
    for g, w in zip(h.locate_packed(cut, cut_off, 64), o.locate_packed(cut, cut_off, 64)):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("change", ["emptied", "exchanged"])
def test_lookup_table_is_the_answer(oracle, change):
    """What the index's lookup table holds for a pattern's last codes is the answer, also where the
    records say otherwise."""
    rng = np.random.default_rng(7)
    a = rng.integers(1, 5, size=60_000).astype(np.uint8)
    depth = 4
    b = bytearray(_build([al.DnaSequence(a)], FmIndexConfig(sa_sample_rate=16, lookup_depth=depth), 1, KIND_FM))
    lut = np.frombuffer(b, "<u4", 2 * 4 ** depth, len(b) - 1 - 8 * 4 ** depth).copy().reshape(-1, 2)
    assert (lut[:, 1] >= lut[:, 0]).all() and int((lut[:, 1] - lut[:, 0]).sum()) > 50_000
    if change == "emptied":
        lut[::3] = 0
    else:
        lut[[5, 77]] = lut[[77, 5]]
    b[len(b) - 1 - 8 * 4 ** depth:len(b) - 1] = lut.astype("<u4").tobytes()
    b = bytes(b)
    o = oracle.OracleIndex(b, KIND_FM)
    h = _Handle(b, KIND_FM)
    flat, off = pack_queries([a[k:k + n].copy() for n in (4, 6, 12, 40) for k in range(0, 50_000, 331)])
    assert np.array_equal(h.count_packed(flat, off), o.count_packed(flat, off))
    for g, w in zip(h.locate_packed(flat, off, 64), o.locate_packed(flat, off, 64)):
        assert np.array_equal(g, w)
    assert np.array_equal(h.share().count_packed(flat, off), o.count_packed(flat, off))


@pytest.mark.parametrize("wide_forward", [False, True])
def test_directions_of_different_record_formats(oracle, wide_forward):
    """One direction holds ambiguity codes, the other does not: their records have different sizes.
    MEM searches, which read both, are refused; the forward index alone is searched as ever."""
    import ctypes as C

    import torch
    from haystackfm_b200 import _lib as L
    from haystackfm_b200.errors import FmIndexError
    rng = np.random.default_rng(9)
    a = rng.integers(1, 5, size=20_000).astype(np.uint8)
    c = a.copy()
    c[::50] = 5
    if wide_forward:
        a, c = c, a
    fwd = _build([al.DnaSequence(a)], FmIndexConfig(sa_sample_rate=16, lookup_depth=4), 0, KIND_FM)
    rev = _build([al.DnaSequence(c[::-1].copy())], FmIndexConfig(sa_sample_rate=16), 0, KIND_FM)
    h = _Handle(struct.pack("<I", len(fwd)) + fwd + rev, KIND_BIDIR)
    flat, off = pack_queries([a[k:k + 40].copy() for k in range(0, 19_000, 500)])
    for variant, threads in ((3, 1), (2, 1), (4, 1), (3, 32)):
        h.set_tuning(variant, 64, threads_per_read=threads)
        with pytest.raises(FmIndexError):
            h.mems_packed(flat, off, 19, 0, None, 64)
    q, qo, g = torch.from_numpy(flat).cuda(), torch.from_numpy(off.astype(np.int64)).cuda(), C.c_void_p()
    assert L.lib().hfm_mems_graph_create(h.h, q.data_ptr(), qo.data_ptr(), len(off) - 1, len(flat), 19, 0, None, 0, 64, 10_000,
                                         C.byref(g)) != 0
    o = oracle.OracleIndex(fwd, KIND_FM)
    assert np.array_equal(h.count_packed(flat, off), o.count_packed(flat, off))
    for g, w in zip(h.locate_packed(flat, off, 64), o.locate_packed(flat, off, 64)):
        assert np.array_equal(g, w)
