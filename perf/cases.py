"""Performance cases of the query path and of index construction.

Each case is one call that a program makes: a batch of queries against an index that it
loaded once and keeps.  Three references stand for what is indexed:

  exact   1 Mbp uniform ACGT, ExactDna, no lookup table (a small genome, cache-resident)
  iupac   100 Mbp IupacDna, 200 contigs, 2% in N runs (mean 500), 0.5% ambiguity codes
  genome  256 Mbp repeat-rich ACGT, ExactDna, 24 contigs (a large chromosome)

all with suffix-array sample rate 32 (iupac and genome: lookup depth 10, bidirectional).
The references are the same for every seed, as an index is for a program's many batches.
The size of a result depends on the reads, so a batch whose result is data-dependent is a
fixed sample of reads in an order that the seed gives (every output changes with it, no
size does); queries of the exact reference, counted queries and built sequences are new for
every seed.  Outputs are whole numbers: positions, counts, hit records and index bytes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from haystackfm_b200 import _lib as L
from haystackfm_b200 import alphabet as al
from haystackfm_b200 import synth
from haystackfm_b200 import synth_gpu
from haystackfm_b200.fm_index import BidirFmIndex, FmIndex

N = 5
IUPAC_LEN = 100_000_000
GENOME_LEN = 256_000_000
EXACT_LEN = 1_000_000


def listed():
    return [
        # one interactive lookup: the latency of a whole host call
        dict(name="locate_1_host", op="locate_host", ref="exact", reads=1, length=24, ragged=False, max_hits=0),
        # the reference's own batch-locate shape: 10,000 32-mers through host buffers
        dict(name="locate_10k_host", op="locate_host", ref="exact", reads=10_000, length=32, ragged=False, max_hits=0),
        # k-mer counting, ragged 20..40-mers already on the device
        dict(name="count_1m_genome", op="count", ref="genome", reads=1_000_003, length=40, ragged=True),
        # seed lookup on an IUPAC assembly: first 32 bases of each read, hits capped
        dict(name="locate_500k_iupac", op="locate", ref="iupac", reads=500_000, length=32, ragged=False,
             max_hits=1024),
        # a small serving batch of short reads, host buffers in and out
        dict(name="smem_64_host", op="mems_host", ref="iupac", reads=64, length=150, ragged=False, min_len=19,
             max_hits=1024, mode=0, order=0),
        # an ordinary batch through host buffers: the result copy is part of the call
        dict(name="smem_4k_host", op="mems_host", ref="iupac", reads=4_099, length=150, ragged=False, min_len=19,
             max_hits=1024, mode=0, order=0),
        # the headline workload: short reads on an IUPAC assembly, device-resident, with the
        # read order that the autotuner picks there
        dict(name="smem_200k_iupac", op="mems", ref="iupac", reads=200_000, length=150, ragged=False, min_len=19,
             max_hits=1024, mode=0, order=1),
        # resequencing: a large batch of short reads on a chromosome
        dict(name="smem_1m_genome", op="mems", ref="genome", reads=1_000_000, length=150, ragged=False, min_len=19,
             max_hits=1024, mode=0, order=0),
        # short and long noisy reads together (20% up to 10 kbp, 8% errors)
        dict(name="smem_mixed_60k", op="mixed", ref="genome", reads=60_000, min_len=19, max_hits=1024, mode=0,
             order=0),
        # the same mix as a serving loop's small batch: bound by its longest read
        dict(name="smem_mixed_250", op="mixed", ref="genome", reads=250, min_len=19, max_hits=1024, mode=0, order=0),
        # all MEMs of ragged reads (find_mems)
        dict(name="mem_20k_genome", op="mems", ref="genome", reads=20_000, length=200, ragged=True, min_len=21,
             max_hits=256, mode=1, order=0),
        # construction of a bidirectional IUPAC index on the GPU (a bacterial genome)
        dict(name="build_5m", op="build", bases=5_000_000, contigs=12, tag=0, lookup=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["locate_host", "count", "locate", "locate", "mems_host", "mems", "mems", "mems", "mixed",
                     "mem_mode", "build"])
    if op == "build":
        return dict(op=op, bases=_log(rng, 200_000, 5_000_000), contigs=rng.randint(1, 40), tag=rng.randint(0, 1),
                    lookup=rng.choice([0, 4, 8, 10]))
    if op == "locate_host":
        return dict(op=op, ref="exact", reads=_log(rng, 1, 20_000), length=rng.randint(24, 64),
                    ragged=rng.random() < 0.5, max_hits=rng.choice([0, 64]))
    if op in ("count", "locate"):
        ref = rng.choice(["exact", "iupac", "genome"] if op == "count" else ["iupac", "genome"])
        c = dict(op=op, ref=ref, reads=_log(rng, 32, 1_000_000 if ref != "iupac" else 500_000),
                 length=rng.randint(20, 64), ragged=rng.random() < 0.5)
        if op == "locate":
            c["max_hits"] = rng.choice([0, 64, 1024]) if ref == "genome" else rng.choice([64, 1024])
        return c
    c = dict(op=op, ref=rng.choice(["iupac", "genome"]), min_len=rng.randint(15, 31),
             max_hits=rng.choice([64, 256, 1024]), mode=0, order=rng.randint(0, 1))
    if op == "mixed":
        return dict(c, ref="genome", reads=_log(rng, 32, 50_000))
    c.update(length=rng.randint(60, 250), ragged=rng.random() < 0.5)
    if op == "mem_mode":
        return dict(c, op="mems", mode=1, reads=_log(rng, 32, 15_000 if c["ref"] == "genome" else 100))
    if op == "mems_host":
        return dict(c, reads=_log(rng, 32, 4_000))
    return dict(c, reads=_log(rng, 32, 150_000 if c["ref"] == "iupac" else 500_000))


# ---- references and indices: made once per process, kept as a program keeps them --------

_refs: dict = {}
_handles: dict = {}


def _build_bytes(codes: np.ndarray, ends: np.ndarray, tag: int, lookup: int, kind: int):
    """hfm_build_index_gpu on concatenated sequences (host codes) -> index bytes."""
    off = np.concatenate([[0], np.asarray(ends)]).astype(np.uint64)
    opts = L.HfmBuildOpts(32, lookup, tag, 0, 1)
    out, n = L.u8p(), C.c_size_t()
    L.check(L.lib().hfm_build_index_gpu(L.ptr(codes, L.u8p), L.ptr(off, L.u64p), len(off) - 1, None, C.byref(opts),
                                        kind, 0, C.byref(out), C.byref(n)))
    try:
        return np.ctypeslib.as_array(out, shape=(n.value,)).copy()
    finally:
        L.lib().hfm_free(out)


def _mask_reference(truth: torch.Tensor, gen: torch.Generator, n_frac=0.02, run_mean=500, code_frac=0.005):
    """N runs (geometric lengths) and single ambiguity codes laid over an ACGT sequence."""
    total = truth.numel()
    runs = max(1, int(total * n_frac) // run_mean)
    dev = truth.device
    u = torch.rand(runs, generator=gen, device=dev, dtype=torch.float64)
    length = (torch.log1p(-u) / math.log1p(-1.0 / run_mean)).long() + 1
    start = torch.randint(0, total, (runs,), generator=gen, device=dev)
    edge = torch.zeros(total + 1, dtype=torch.int32, device=dev)
    one = torch.ones(runs, dtype=torch.int32, device=dev)
    edge.index_add_(0, start, one)
    edge.index_add_(0, (start + length).clamp(max=total), -one)
    covered = torch.cumsum(edge[:total], 0, dtype=torch.int32) > 0
    out = truth.clone()
    for a in range(0, total, 1 << 24):
        m = min(1 << 24, total - a)
        hit = torch.rand(m, generator=gen, device=dev) < code_frac
        code = torch.randint(6, 16, (m,), generator=gen, device=dev, dtype=torch.uint8)
        out[a:a + m] = torch.where(hit, code, out[a:a + m])
    out[covered] = N
    return out


def _reference(ref: str):
    """(unmasked codes on the GPU, exclusive sequence ends, index)."""
    if ref in _refs:
        return _refs[ref]
    gen = _gen(101)
    if ref == "genome":
        truth, ends = synth_gpu.repeat_genome(total=GENOME_LEN, n_contigs=24, seed=11)
        data = _build_bytes(truth.cpu().numpy(), ends, 1, 10, 1)
        index = BidirFmIndex.from_bytes(data)
    elif ref == "iupac":
        truth = torch.randint(1, 5, (IUPAC_LEN,), generator=gen, device="cuda", dtype=torch.uint8)
        w = np.random.default_rng(7).lognormal(13.0, 1.0, size=200)
        ends = np.maximum(np.floor(w / w.sum() * IUPAC_LEN), 2000).astype(np.int64)
        ends[int(np.argmax(ends))] += IUPAC_LEN - int(ends.sum())
        ends = np.cumsum(ends)
        data = _build_bytes(_mask_reference(truth, gen).cpu().numpy(), ends, 0, 10, 1)
        index = BidirFmIndex.from_bytes(data)
    else:
        truth = torch.randint(1, 5, (EXACT_LEN,), generator=gen, device="cuda", dtype=torch.uint8)
        ends = np.array([EXACT_LEN])
        data = _build_bytes(truth.cpu().numpy(), ends, 1, 0, 0)
        index = FmIndex.from_bytes(data)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _refs[ref] = (truth, ends, index)
    return _refs[ref]


def _handle(ref: str, order: int):
    """The handle that a program keeps for this index and read order."""
    if (ref, order) not in _handles:
        h = _reference(ref)[2].handle
        if order:
            h = h.share()
            t = h.tuning()
            h.set_tuning(t["mems_variant"], t["seg_len"], read_order=order)
        _handles[(ref, order)] = h
    return _handles[(ref, order)]


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ragged(rows: torch.Tensor, seed: int):
    """Rows cut to lengths between half and all of the row."""
    n, w = rows.shape
    lens = torch.randint((w + 1) // 2, w + 1, (n,), generator=_gen(seed), device="cuda")
    keep = torch.arange(w, device="cuda")[None, :] < lens[:, None]
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    return rows[keep], off


def _shuffled(q: torch.Tensor, off: torch.Tensor, seed: int):
    """The reads of a batch in the order that the seed gives."""
    perm = torch.randperm(len(off) - 1, generator=_gen(seed), device="cuda")
    lens = torch.diff(off)[perm]
    out = torch.zeros_like(off)
    out[1:] = torch.cumsum(lens, 0)
    src = torch.repeat_interleave(off[:-1][perm] - out[:-1], lens) + torch.arange(len(q), device="cuda")
    return q[src], out


def _reads(case, seed):
    """Query codes and offsets on the GPU."""
    truth, ends, _ = _reference(case["ref"])
    n = case["reads"]
    if case["op"] == "mixed":
        return _shuffled(*synth_gpu.sample_mixed_reads(truth, ends, n, seed=5), seed)
    w = case["length"]
    if case["ref"] == "exact":           # nine queries in ten are substrings of the reference
        g = _gen(seed + 1)
        start = torch.randint(0, EXACT_LEN - w + 1, (n,), generator=g, device="cuda")
        rows = truth[start[:, None] + torch.arange(w, device="cuda")[None, :]]
        other = torch.randperm(n, generator=g, device="cuda")[: n // 10]
        rows[other] = torch.randint(1, 5, (len(other), w), generator=g, device="cuda", dtype=torch.uint8)
        sample = seed
    else:
        sample = seed if case["op"] == "count" else 3
        rows = synth_gpu.sample_reads(truth, ends, n, read_len=w, sub_rate=0.01,
                                      n_rate=0.001 if case["ref"] == "iupac" else 0.0, seed=sample)
    if case["ragged"]:
        q, off = _ragged(rows, sample + 2)
    else:
        q, off = rows.reshape(-1).contiguous(), torch.arange(n + 1, dtype=torch.int64, device="cuda") * w
    return (q, off) if sample == seed else _shuffled(q, off, seed)


def prepare(case, seed):
    op = case["op"]
    if op == "build":
        total = case["bases"]
        if case["tag"] == 0:
            codes = synth.iupac_reference(total=total, n_contigs=1, seed=seed).contigs[0]
        else:
            codes = np.random.default_rng(seed).integers(1, 5, size=total, dtype=np.uint8)
        cuts = np.random.default_rng(case["contigs"]).integers(1, total, size=case["contigs"] - 1)
        return dict(op=op, codes=codes, ends=np.unique(np.append(cuts, total)), tag=case["tag"],
                    lookup=case["lookup"])
    q, off = _reads(case, seed)
    index = _reference(case["ref"])[2]
    s = dict(op=op, handle=_handle(case["ref"], case.get("order", 0)), reads=len(off) - 1,
             max_hits=case.get("max_hits", 0), min_len=case.get("min_len", 0), mode=case.get("mode", 0),
             bounds=np.ascontiguousarray(index.seq_boundaries(), dtype=np.uint32))
    if op.endswith("_host"):
        s.update(q=q.cpu().numpy(), off=off.cpu().numpy().view(np.uint64))
    else:
        s.update(q=q, off=off, counts=torch.zeros(len(off) - 1, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return s


class _Device:
    """A device array of the library, for torch."""

    def __init__(self, p, n, kind):
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": kind, "data": (int(p), False), "version": 3}


def _tensor(p, n, kind):
    if not n:
        return torch.zeros(0, dtype=torch.int32 if kind == "<i4" else torch.int64, device="cuda")
    return torch.as_tensor(_Device(p, n, kind), device="cuda")


def run(s):
    op, n = s["op"], s.get("reads")
    if op == "build":
        return _build_bytes(s["codes"], s["ends"], s["tag"], s["lookup"], 1)
    h, lib = s["handle"], L.lib()
    if op == "locate_host":
        return h.locate_packed(s["q"], s["off"], s["max_hits"])
    if op == "mems_host":
        return h.mems_packed(s["q"], s["off"], s["min_len"], s["mode"], s["bounds"], s["max_hits"])
    q, off = s["q"].data_ptr(), s["off"].data_ptr()
    if op == "count":
        L.check(lib.hfm_count_batch_device(h.h, q, off, n, s["counts"].data_ptr()))
        return s["counts"]
    if op == "locate":
        d = L.HfmDevHits()
        L.check(lib.hfm_locate_batch_device(h.h, q, off, n, s["max_hits"], C.byref(d)))
        return (_tensor(d.d_offsets, n + 1, "<i8"), _tensor(d.d_counts, n, "<i4"),
                _tensor(d.d_pairs, 2 * d.total, "<i4"))
    d = L.HfmDevMems()
    L.check(lib.hfm_mems_batch_device(h.h, q, off, n, s["min_len"], s["mode"], L.ptr(s["bounds"], L.u32p),
                                      len(s["bounds"]), s["max_hits"], C.byref(d)))
    return (_tensor(d.d_hit_offsets, n + 1, "<i8"), _tensor(d.d_hits, 8 * d.n_hits, "<i4"),
            _tensor(d.d_positions, 2 * d.n_positions, "<i4"))


def work(case):
    """Expected bytes of one pass: codes in, one 32-byte Occ sector for every base that is
    searched (those a lookup table answers left out), results out (hits per read as these
    references give them)."""
    if case["op"] == "build":            # both directions: the codes once, about 1.5 bytes of index per base
        return dict(bytes=case["bases"] * (1 + 3), flops=0)
    n = case["reads"]
    if case["op"] == "mixed":            # 80% of 150 bp, 20% of a mean near 3.5 kbp
        return dict(bytes=n * (820 * 33 + 20 * 40), flops=0)
    m = case["length"] * (0.75 if case["ragged"] else 1.0)
    iupac = case["ref"] == "iupac"
    if case["op"] in ("count", "locate", "locate_host"):
        seeded = 0 if case["ref"] == "exact" else min(10, m)
        out = 4 if case["op"] == "count" else 12 + 8 * (40 if iupac else 2)
        return dict(bytes=n * (m + 32 * (m - seeded) + 8 + out), flops=0)
    hits, positions = (38, 3000) if iupac else (4, 6)
    if case["max_hits"] < 1024:
        positions = min(positions, hits * case["max_hits"] // 4)
    return dict(bytes=n * (33 * m + 8 + 32 * hits + 8 * positions), flops=0)


def exact(case, seed):
    return None                          # every output is a whole number
