"""ACGT reads searched whole, as one job of many words: the packing pass takes 992 codes a turn,
an anchor may straddle two turns.  Reads whole by tuning and in a captured graph, which cuts at the
tuned segment length; errors and other codes around the turns' edges.  Bytes equal the oracle's."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from haystackfm_b200 import _lib as L
from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200.fm_index import FmIndexConfig, KIND_BIDIR, _Handle, _build, _header_fields
from haystackfm_b200._lib import pack_queries

pytestmark = pytest.mark.gpu

LENGTHS = (960, 991, 992, 993, 1023, 1024, 1025, 1984, 1985, 2977, 4500)


@pytest.fixture(scope="module", params=[0, 1])
def case(request, oracle):
    tag = request.param
    ref = synth.repeat_reference(total=300_000, n_contigs=2, seed=15)
    b = _build([al.DnaSequence(c) for c in ref.contigs], FmIndexConfig(sa_sample_rate=16, lookup_depth=6), tag, KIND_BIDIR)
    t = max(ref.truth, key=len)
    rng = np.random.default_rng(6)
    reads = []
    for n in LENGTHS:
        a = int(rng.integers(0, len(t) - n))
        reads.append(t[a:a + n].copy())
        for edge in (992, 1984, 2976):
            for at in (edge - 20, edge - 1, edge, edge + 1, edge + 18):
                if at < n:
                    r = t[a:a + n].copy()
                    r[at] = r[at] % 4 + 1
                    r[max(0, at - 25)] = 5 if at % 3 == 0 else r[max(0, at - 25)] % 4 + 1
                    reads.append(r)
        noisy = t[a:a + n].copy()
        hit = rng.random(n) < 0.06
        noisy[hit] = noisy[hit] % 4 + 1
        reads += [noisy, t[a:a + 90].copy()]
    return b, reads, _header_fields(b, 4)[2], oracle.OracleIndex(b, KIND_BIDIR)


@pytest.mark.parametrize("min_len", [15, 19, 33, 64])
def test_whole_reads(case, min_len):
    b, reads, bounds, o = case
    h = _Handle(b, KIND_BIDIR)
    flat, off = pack_queries(reads)
    for mode in (0, 1):
        want = o.mems_packed(flat, off, min_len, mode, bounds, 32, threads=8)
        for variant in (2, 3):
            h.set_tuning(variant, 512)
            for g, w in zip(h.mems_packed(flat, off, min_len, mode, bounds, 32), want):
                assert np.array_equal(g, w), (mode, variant)


@pytest.mark.parametrize("seg_len", [512, 1024, 4096])
def test_captured_chain(case, seg_len):
    import torch
    b, reads, bounds, o = case
    h = _Handle(b, KIND_BIDIR)
    h.set_tuning(3, seg_len)
    flat, off = pack_queries(reads)
    want = o.mems_packed(flat, off, 19, 0, bounds, 32, threads=8)
    q = torch.from_numpy(flat).cuda()
    qo = torch.from_numpy(off.astype(np.int64)).cuda()
    torch.cuda.synchronize()
    g = C.c_void_p()
    rb = np.ascontiguousarray(bounds, dtype=np.uint32)
    L.check(L.lib().hfm_mems_graph_create(h.h, q.data_ptr(), qo.data_ptr(), len(reads), int(off[-1]), 19, 0,
                                          L.ptr(rb, L.u32p), len(rb), 32, 2_000_000, C.byref(g)))
    try:
        for _ in range(2):
            d, replayed = L.HfmDevMems(), C.c_uint32()
            L.check(L.lib().hfm_mems_graph_launch(g, C.byref(d), C.byref(replayed)))
            assert d.n_hits == want[0][-1] and d.n_positions == len(want[2])

            def host(p, n, dt):
                class A:
                    __cuda_array_interface__ = {"shape": (int(n),), "typestr": dt, "data": (int(p), False), "version": 3}
                return torch.as_tensor(A(), device="cuda").cpu().numpy()
            assert np.array_equal(host(d.d_hit_offsets, len(reads) + 1, "<i8").astype(np.uint64), want[0])
            assert np.array_equal(host(d.d_hits, 8 * d.n_hits, "<i4").view(np.uint32).reshape(-1, 8), want[1])
            assert np.array_equal(host(d.d_positions, 2 * d.n_positions, "<i4").view(np.uint32).reshape(-1, 2), want[2])
        assert replayed.value == 1
    finally:
        L.lib().hfm_mems_graph_free(g)
