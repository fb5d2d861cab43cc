"""SMEM windows that hold many codes of several symbols: the search starts at the window's longest
run of ACGT.  Runs of N at every place of the first windows, around errors and at the ends of
reads, other ambiguity codes, codes that match nothing; bytes equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, _Handle, _build, _header_fields
from haystackfm_b200._lib import pack_queries

pytestmark = pytest.mark.gpu


def _index(kind):
    if kind == "acgt":
        ref = synth.repeat_reference(total=200_000, n_contigs=3, seed=16)
    elif kind == "few_codes":
        ref = synth.iupac_reference(total=100_000, n_contigs=3, n_frac=0.0, iupac_frac=0.002, seed=17)
    else:
        ref = synth.iupac_reference(total=100_000, n_contigs=3, n_run_mean=40, seed=18)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), 0, KIND_BIDIR)
    return ref, b


def _reads(ref, n=60, seed=1):
    """Reads of 45..70 codes with a run of 1..7 N (or other codes) at every kind of place."""
    rng = np.random.default_rng(seed)
    reads = []
    for k in range(n):
        t = ref.truth[k % len(ref.truth)]
        m = int(rng.integers(45, 71))
        a = int(rng.integers(0, len(t) - m))
        r = t[a:a + m].copy()
        w = 1 + k % 7
        at = [0, 5, 10, 13, 18, 19, 25, m - w - 3, m - w][k % 9] if k % 3 else int(rng.integers(0, m - w))
        r[at:at + w] = 5 if k % 4 else rng.integers(5, 16, size=w)
        if k % 2:                                        # an error shortly before or behind the run
            e = int(np.clip(at + rng.integers(-12, w + 12), 0, m - 1))
            r[e] = r[e] % 4 + 1 if r[e] <= 4 else r[e]
        if k % 11 == 0:
            r[int(rng.integers(0, m))] = 0
        reads.append(r)
    return reads


@pytest.mark.parametrize("kind", ["acgt", "few_codes", "n_runs"])
def test_runs_of_ambiguous_codes(oracle, kind):
    ref, b = _index(kind)
    h = _Handle(b, KIND_BIDIR)
    bounds = _header_fields(b, 4)[2]
    flat, off = pack_queries(_reads(ref))
    o = oracle.OracleIndex(b, KIND_BIDIR)
    for min_len, mode in ((19, 0), (11, 0), (19, 1), (30, 0)):
        want = o.mems_packed(flat, off, min_len, mode, bounds, 4, threads=8)
        for variant, threads in ((3, 1), (2, 1), (3, 8), (3, 32)):
            h.set_tuning(variant, 64, threads_per_read=threads)
            for g, w in zip(h.mems_packed(flat, off, min_len, mode, bounds, 4), want):
                assert np.array_equal(g, w), (min_len, mode, variant, threads)


def test_sets_stay_small(oracle):
    """A match of the whole read is found without large sets wherever six N stand in it."""
    ref, b = _index("acgt")
    h = _Handle(b, KIND_BIDIR)
    rng = np.random.default_rng(2)
    reads = []
    for at in range(12, 60):
        t = ref.truth[at % len(ref.truth)]
        a = int(rng.integers(0, len(t) - 90))
        r = t[a:a + 90].copy()
        r[at:at + 6] = 5
        reads.append(r)
    flat, off = pack_queries(reads)
    want = oracle.OracleIndex(b, KIND_BIDIR).mems_packed(flat, off, 19, 0, None, 4, threads=8)
    for g, w in zip(h.mems_packed(flat, off, 19, 0, None, 4), want):
        assert np.array_equal(g, w)
    assert h.stats().fallback_reads == 0
