"""GPU index construction at the edges of its passes: texts around 32, 64 and 512 rows (a
ballot, a record, a superblock) and around 16 positions (a thread's share of the joined text),
one to sixteen lanes, both Occ encodings, empty sequences, and each sampling rate's count of
sampled rows.  The bytes equal the CPU builder's."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from haystackfm_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _bytes(fn, codes, lens, tail, opts, kind):
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    out, n = L.u8p(), C.c_size_t()
    L.check(fn(L.ptr(codes, L.u8p), L.ptr(off, L.u64p), len(lens), None, C.byref(opts), kind, *tail, C.byref(out),
               C.byref(n)))
    try:
        return np.ctypeslib.as_array(out, shape=(n.value,)).copy()
    finally:
        L.lib().hfm_free(out)


@pytest.mark.parametrize("codes", [1, 2, 3, 4, 8, 15])
@pytest.mark.parametrize("enc", [0, 1])
def test_gpu_builder_at_the_edges_of_its_passes(codes, enc):
    rng = np.random.default_rng(100 * codes + enc)
    texts = [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 511, 512, 513, 2047, 2048, 2049, 4 * 512 + 65, 40_000]
    for k, n in enumerate(texts):                     # n: positions with the sentinels
        for nseq in {1, min(n, 1 + int(rng.integers(0, 6)))}:
            cuts = np.sort(rng.integers(0, n - nseq + 1, size=nseq - 1))
            lens = np.diff(np.concatenate([[0], cuts, [n - nseq]]))          # empty ones among them
            q = rng.integers(1, codes + 1, size=max(n - nseq, 1), dtype=np.uint8)
            opts = L.HfmBuildOpts([0, 1, 3, 32, 64][k % 5], [0, 1, 2, 3, 6][(k + enc) % 5], 0, enc, 1)
            kind = k & 1
            want = _bytes(L.lib().hfm_build_index, q, lens, (), opts, kind)
            got = _bytes(L.lib().hfm_build_index_gpu, q, lens, (0,), opts, kind)
            assert np.array_equal(got, want), (n, lens.tolist(), opts.sa_sample_rate, opts.lookup_depth, kind)
