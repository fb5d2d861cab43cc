// search.cuh — per-read search kernels: IUPAC backward search (count / locate
// intervals) and the bidirectional SMEM / MEM candidate search.
//
// Execution model: persistent grids (one wave of resident threads) pull reads from a
// device work queue; one thread owns one read at a time.  A read's path is a chain of
// ~|read| dependent rank steps, so throughput comes from keeping ~10^5 reads in flight,
// not from spreading one read over a warp.  Interval sets live in per-thread slices of a
// global work area, interleaved across the 32 lanes of a warp (element i of every lane is
// one contiguous run: 128 B per u32 plane of the SMEM sets, 256 B per uint2 of the backward
// search sets) with a fixed capacity; a read whose set, hit list or output outgrows it is
// queued for a fallback pass with much larger slices (a per-thread rerun for long hit
// lists, then one warp per read).  There is therefore no cap on interval-set size, as in
// the reference CPU (src/fm_index/query.rs:248-274, src/fm_index/smem.rs:332-357).  The
// per-thread SMEM kernel is in smem.cuh; this file has the sets, the plain launch and the
// lane-group kernels.
#pragma once
#include <type_traits>
#include "dev_index.cuh"

namespace hfm {

// Interval-set capacity of the per-thread SMEM kernels (warp-interleaved sets, STRIDE 32).
constexpr uint32_t FAST_SET_CAP = 768;

// Results are bump-allocated in pools; per-read (offset, count) record where they went.
struct Pool {
  void* base;
  unsigned long long* used;   // device counter (elements)
  uint64_t cap;               // elements
};

__device__ __forceinline__ uint64_t thread_reserve(Pool& p, uint32_t n) {
  if (n == 0) return 0;
  unsigned long long off = atomicAdd(p.used, (unsigned long long)n);
  return (off + n <= p.cap) ? off : ~0ull;
}

// Status bits per read.
enum : uint32_t { ST_OK = 0, ST_SET_OVF = 1, ST_CAND_OVF = 2, ST_POOL_OVF = 4 };

// A thread's interval set: element i at p[i * STRIDE].
template <class T, int STRIDE>
struct SetRef {
  T* p;
  __device__ __forceinline__ T& operator[](uint32_t i) const { return p[(size_t)i * STRIDE]; }
};

// Interval sets of the SMEM path store a bidirectional interval as three u32 planes
// (flo, rlo, size): fhi - flo == rhi - rlo always holds, so 12 bytes carry the 16 of a BIv
// and the sets' traffic (most DRAM writes of the search) drops by a quarter.  Single-row
// intervals (the front list of a TwoList) store only (flo, rlo): their size is 1.
template <int STRIDE>
struct SetRef<BIv, STRIDE> {
  uint32_t* p;          // this thread's slot: field f of element i at p[(f * cap + i) * STRIDE]
  uint32_t plane_;      // cap * STRIDE (warp-interleaved sets: always FAST_SET_CAP * 32)
  __device__ __forceinline__ uint32_t pl() const { return STRIDE == 32 ? FAST_SET_CAP * 32 : plane_; }
  struct Ref {
    uint32_t* a; uint32_t plane;
    __device__ __forceinline__ operator BIv() const {
      uint32_t f = a[0], r = a[plane], z = a[2 * plane];
      return BIv{f, f + z, r, r + z};
    }
    __device__ __forceinline__ Ref& operator=(const BIv& v) {
      a[0] = v.flo; a[plane] = v.rlo; a[2 * plane] = v.fhi - v.flo;
      return *this;
    }
  };
  __device__ __forceinline__ Ref operator[](uint32_t i) const { return Ref{p + (size_t)i * STRIDE, pl()}; }
  __device__ __forceinline__ BIv single(uint32_t i) const {
    const uint32_t* a = p + (size_t)i * STRIDE;
    uint32_t f = a[0], r = a[pl()];
    return BIv{f, f + 1, r, r + 1};
  }
  __device__ __forceinline__ void set_single(uint32_t i, uint32_t flo, uint32_t rlo) const {
    uint32_t* a = p + (size_t)i * STRIDE;
    a[0] = flo; a[pl()] = rlo;
  }
};

// Set s (of NS) of the calling thread inside `work`, `cap` elements each.
// STRIDE 32: warp-interleaved slices (fast path); STRIDE 1: contiguous per-thread slices.
template <class T, int STRIDE>
__device__ __forceinline__ SetRef<T, STRIDE> thread_set(T* work, uint32_t cap, int NS, int s) {
  uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (std::is_same<T, BIv>::value) {
    uint32_t* w = reinterpret_cast<uint32_t*>(work);           // 3 planes of cap u32 per set
    if (STRIDE == 32) {
      uint64_t warp = tid >> 5, lane = tid & 31;
      return SetRef<T, STRIDE>{w + ((warp * NS + s) * cap * 3) * 32 + lane, cap * STRIDE};
    }
    return SetRef<T, STRIDE>{w + (tid * NS + s) * cap * 3, cap * STRIDE};
  } else {
    if (STRIDE == 32) {
      uint64_t warp = tid >> 5, lane = tid & 31;
      return SetRef<T, STRIDE>{work + ((warp * NS + s) * cap) * 32 + lane};
    }
    return SetRef<T, STRIDE>{work + (tid * NS + s) * cap};
  }
}

// Next read from the device queue: reads are ids[k] (or k itself when ids is null).
__device__ __forceinline__ bool next_read(unsigned int* ctr, uint32_t n, const uint32_t* ids, uint32_t& i) {
  uint32_t k = atomicAdd(ctr, 1u);
  if (k >= n) return false;
  i = ids ? ids[k] : k;
  return true;
}

// The same queue taken `chunk` consecutive entries per atomic: the thread works through its
// chunk before it takes the next one (a tunable; 1 = one entry per atomic).
struct QueueCursor { uint32_t next = 0, end = 0; };
__device__ __forceinline__ bool next_read_chunked(unsigned int* ctr, uint32_t n, const uint32_t* ids, uint32_t chunk,
                                                  QueueCursor& c, uint32_t& i) {
  if (c.next >= c.end) {
    const uint32_t k = atomicAdd(ctr, chunk);
    if (k >= n) return false;
    c.next = k;
    c.end = min(n, k + chunk);
  }
  const uint32_t k = c.next++;
  i = ids ? ids[k] : k;
  return true;
}

// =====================================================================================
// Backward search (FmIndex::backward_search, src/fm_index/query.rs:219-277)
// =====================================================================================

struct BsOut {
  uint32_t* counts;      // exact count per query
  uint64_t* nhits;       // sum of min(size, cap) per query (nullptr: count only)
  uint32_t* niv;         // intervals per query
  uint64_t* ivoff;       // pool offset of the intervals
  uint32_t* status;      // per-query status bits
  uint32_t* ovf_list;    // queries to re-run with large sets
  uint32_t* n_ovf;
  unsigned long long* touches;  // Occ record touches (counted only with COUNT_TOUCH)
};

// What a handle keeps for queries besides the records, made on the device when an index is
// loaded: sa is the position of every forward row (resolve.cuh); the others exist for ACGT
// texts only:
//   kmer  for every ACGT string of k codes its forward start, reverse start and rows: a search
//         starts k steps on, with one load;
//   text  the text as bit planes (with sa): the rest of a one-row match is read off them;
//   seen  a bit for every string of seen_k codes, set when it occurs in the text.
// A string's place in kmer and seen: the second bits of its symbols - 1, then their first
// bits, the string's first code in the lowest bit of either (plane_key).
// Any may be absent (no memory for it): the searches then take the steps.
struct DevAux {
  const uint4* kmer;
  const uint32_t* sa;
  const uint4* text;              // 32 codes a word (k_text_planes); only with sa
  const uint32_t* seen;           // only with text
  uint32_t k, seen_k;
};

__device__ __forceinline__ uint64_t plane_key(uint32_t b0, uint32_t b1, uint32_t k) {
  const uint32_t m = (1u << k) - 1u;        // k < 32
  return (uint64_t)(b1 & m) << k | (b0 & m);
}

// Query code -> the one symbol of the text that it matches, 0 for none, SYM_MANY for several
// (256 entries, every code a byte can hold).
constexpr uint32_t SYM_MANY = 0xFF;
__device__ __forceinline__ void sym_table_init(uint8_t* t, const uint16_t* compat, uint32_t sym_mask) {
  for (uint32_t c = threadIdx.x; c < 256; c += blockDim.x) {
    const uint32_t m = c < 16 ? (uint32_t)compat[c] & sym_mask : 0u;
    t[c] = (uint8_t)(!m ? 0u : m & (m - 1) ? SYM_MANY : 31u - (uint32_t)__clz(m));
  }
}

// Rows [lo, lo + n) narrowed to those preceded by code s (1..4) of an ACGT text; false, and
// nothing changed, when there are none.
template <bool COUNT_TOUCH>
__device__ __forceinline__ bool acgt_rows(const DevFm& F, const uint32_t* C, uint32_t s, uint32_t& lo, uint32_t& n,
                                          uint64_t& touches) {
  const uint32_t last = lo + n - 1, bl = lo >> 6, bh = last >> 6, sh = 16u * (s - 1u);
  const uint4* pl = F.occ + (size_t)bl * OCC_NARROW_U4;
  const uint4 u = __ldg(pl), v = __ldg(pl + 1);
  const uint32_t sbl = __ldg(F.sb + (size_t)(bl >> SB_BLOCK_SHIFT) * 16 + s);
  uint4 u2 = u, v2 = v;
  uint32_t sbh = sbl;
  if (bh != bl) {
    const uint4* ph = F.occ + (size_t)bh * OCC_NARROW_U4;
    u2 = __ldg(ph); v2 = __ldg(ph + 1);
    sbh = __ldg(F.sb + (size_t)(bh >> SB_BLOCK_SHIFT) * 16 + s);
  }
  if (COUNT_TOUCH) touches += bh != bl ? 2 : 1;
  Border<OCC_NARROW> L, H;
  L.take(u, v, lo & 63);
  H.take(u2, v2, (last & 63) + 1u);
  const uint32_t k0 = 0u - ((s - 1u) & 1u), k1 = 0u - ((s - 1u) >> 1);
  auto rank = [&](const Border<OCC_NARROW>& B) {
    return ((uint32_t)((((uint64_t)B.c34 << 32) | B.c12) >> sh) & 0xFFFFu) +
           (uint32_t)__popc(B.m & ~B.z & ~((B.b0 ^ k0) | (B.b1 ^ k1))) * B.sg;
  };
  const uint32_t rl = sbl + rank(L), d = sbh + rank(H) - rl;
  if (!d) return false;
  lo = C[s] + rl;
  n = d;
  return true;
}

// The borders of rows [lo, lo + n), n >= 1, of a wide index.  The records are those of the first
// and the last row, one when they are the same.
__device__ __forceinline__ void wide_borders(const uint4* __restrict__ occ, uint32_t lo, uint32_t n, Border<OCC_WIDE>& L,
                                             Border<OCC_WIDE>& H) {
  const uint32_t last = lo + n - 1, bl = lo >> 6, bh = last >> 6, xl = lo & 63, xh = (last & 63) + 1;
  const uint4* pl = occ + (size_t)bl * OCC_WIDE_U4;
  const uint4* ph = occ + (size_t)bh * OCC_WIDE_U4;
  L.a = __ldg(pl); L.b = __ldg(pl + 1); L.c = __ldg(pl + 2); L.d = __ldg(pl + 3);
  L.w = __ldg(pl + (xl >= 32 ? 5 : 4));
  H.w = __ldg(ph + (xh >= 32 ? 5 : 4));
  H.a = L.a; H.b = L.b; H.c = L.c; H.d = L.d;
  if (bh != bl) { H.a = __ldg(ph); H.b = __ldg(ph + 1); H.c = __ldg(ph + 2); H.d = __ldg(ph + 3); }
  L.select(xl); H.select(xh);
}

// 16 counts at those borders: r[s] = rank of s at lo, d[s] = rows of code s.
__device__ __forceinline__ void wide_split(const uint4* __restrict__ occ, uint32_t lo, uint32_t n, uint32_t r[16],
                                           uint32_t d[16]) {
  Border<OCC_WIDE> L, H;
  wide_borders(occ, lo, n, L, H);
  wide_ranks(L, r);
  wide_ranks(H, d);
#pragma unroll
  for (int s = 0; s < 16; s++) d[s] -= r[s];
}

// Ranks at lo and rows of every code in [lo, hi), hi > lo, for either record format.
template <uint32_t FMT>
__device__ __forceinline__ void rows_by_code(const DevFm& F, uint32_t lo, uint32_t hi, uint32_t r[16], uint32_t d[16]) {
  if constexpr (FMT == OCC_WIDE) {
    wide_split(F.occ, lo, hi - lo, r, d);
  } else {
    sym_ranks_t<FMT>(F, lo, r);
    sym_ranks_t<FMT>(F, hi, d);
#pragma unroll
    for (int s = 0; s < 16; s++) d[s] -= r[s];
  }
}

// Calls f(code, rank at lo, rows) for each code of `mask` (the same in all lanes that call it)
// in ascending order; rows may be 0.
template <uint32_t FMT, class FN>
__device__ __forceinline__ void each_code(const DevFm& F, uint32_t lo, uint32_t hi, uint32_t mask, FN f) {
  if constexpr (FMT == OCC_WIDE) {
    Border<OCC_WIDE> L, H;
    wide_borders(F.occ, lo, hi - lo, L, H);
#pragma unroll
    for (int s = 0; s < 16; s++) {
      if (!(mask >> s & 1)) continue;
      const uint32_t r = L.local(s);
      f(s, r, H.local(s) - r);
    }
  } else {
    uint32_t r[16], d[16];
    rows_by_code<FMT>(F, lo, hi, r, d);
#pragma unroll
    for (int s = 1; s < 5; s++)
      if (mask >> s & 1) f(s, r[s], d[s]);
  }
}

// Entries of a lookup table over ACGT (last code in the top digit) that are not the rows of their
// string, empty for none: the k-mer table stands in for one that has no such entry.
__global__ void k_lookup_differs(DevFm F, uint32_t* __restrict__ differ) {
  const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >> (2 * F.lut_depth)) return;
  uint32_t C[5], lo = 0, n = F.text_len;
  for (int c = 0; c < 5; c++) C[c] = F.C[c];
  uint64_t touches = 0;
  for (int k = (int)F.lut_depth - 1; k >= 0 && n; k--) {
    if (!acgt_rows<false>(F, C, 1u + ((uint32_t)(idx >> (2 * k)) & 3u), lo, n, touches) || (uint64_t)lo + n > F.text_len) n = 0;
  }
  const uint2 iv = F.lut[idx];
  const uint32_t rows = iv.y > iv.x ? iv.y - iv.x : 0u;
  if (rows != n || (n && iv.x != lo)) atomicAdd(differ, 1u);
}

// The last codes of a pattern at once: the index's own lookup table (LookupTable::get,
// src/fm_index/lookup.rs:101-111: only when all of them are ACGT, and whatever it holds is
// the answer, which on IUPAC texts leaves out strings with other codes), or the k-mer table
// of an ACGT text when that reaches further.  Sets [lo, lo + n) and the codes still to search;
// n = 0 when there is no match, start = m when nothing was looked up.
template <bool COUNT_TOUCH>
__device__ __forceinline__ void seed_pattern(const DevFm& F, const DevAux& A, const uint8_t* dig, const uint8_t* p, uint32_t m,
                                             uint32_t& lo, uint32_t& n, uint32_t& start, uint64_t& touches) {
  lo = 0; n = F.text_len; start = m;
  if (A.kmer && m >= A.k && A.k >= F.lut_depth) {
    uint32_t b0 = 0, b1 = 0, bad = 0;
    const uint8_t* b = p + (m - A.k);
    for (uint32_t k = 0; k < A.k; k++) { const uint32_t c = b[k] - 1u; bad |= c; b0 |= (c & 1u) << k; b1 |= (c >> 1 & 1u) << k; }
    if (bad < 4) {
      const uint4 v = __ldg(A.kmer + plane_key(b0, b1, A.k));
      if (COUNT_TOUCH) touches++;
      lo = v.x; n = v.z; start = m - A.k;
      return;
    }
  }
  if (F.lut && m >= F.lut_depth) {
    uint64_t idx = 0;
    for (int k = (int)F.lut_depth - 1; k >= 0; --k) {
      const uint8_t c = p[m - F.lut_depth + k];
      const uint32_t d = c < 16 ? dig[c] : 0xFF;
      if (d == 0xFF) return;
      idx = idx * F.lut_radix + d;
    }
    const uint2 iv = __ldg(F.lut + idx);
    if (COUNT_TOUCH) touches++;
    lo = iv.x; n = iv.y > iv.x ? iv.y - iv.x : 0u; start = m - F.lut_depth;
  }
}

// Codes left from which on a counted one-row match of an ACGT text is compared with the text.
constexpr uint32_t COUNT_TEXT_LEFT = 4;

// Do the codes p[0..k) stand before the suffix of row `row`, each matching the text's symbol?  A
// code of several symbols is looked up on its own.  (Left to a step of the search, after which
// the rest was compared anew, 1,000 patterns of 2,000 codes with an N among the first took 192 ms.)
template <bool COUNT_TOUCH>
__device__ __forceinline__ bool text_before(const DevAux& A, const SmemFm& S, const uint8_t* sym, const uint8_t* p, uint32_t k,
                                            uint32_t row, uint64_t& touches) {
  const uint32_t at = __ldg(A.sa + row);
  if (COUNT_TOUCH) touches += 1;
  for (uint32_t e = k; e > 0;) {                       // up to 32 codes at a time, the last ones first
    const uint32_t len = min(e, 32u), from = at - (k - e) - len;       // text place of the first of them
    if (at < k - e + len) return false;
    uint32_t b0 = 0, b1 = 0, many = 0, odd = 0;
    for (uint32_t t = 0; t < len; t++) {
      const uint32_t s = sym[p[e - len + t]];
      odd |= s == 0;
      many |= (s == SYM_MANY ? 1u : 0u) << t;
      b0 |= ((s - 1u) & 1u) << t; b1 |= ((s - 1u) >> 1 & 1u) << t;
    }
    if (odd) return false;
    const uint4 x = __ldg(A.text + (from >> 5)), y = __ldg(A.text + (from >> 5) + 1);
    if (COUNT_TOUCH) touches += 1;
    const uint32_t sh = from & 31, part = len == 32 ? ~0u : (1u << len) - 1u;
    const uint32_t t0 = __funnelshift_r(x.x, y.x, sh), t1 = __funnelshift_r(x.y, y.y, sh), z = __funnelshift_r(x.z, y.z, sh);
    if (((((t0 ^ b0) | (t1 ^ b1)) & ~many) | z) & part) return false;
    for (; many; many &= many - 1) {
      const uint32_t t = (uint32_t)__ffs(many) - 1u, symbol = 1u + (t0 >> t & 1u) + 2u * (t1 >> t & 1u);
      if (!(S.compat_mask[p[e - len + t]] >> symbol & 1)) return false;
    }
    e -= len;
  }
  return true;
}

// Backward search of one pattern (FmIndex::backward_search, src/fm_index/query.rs:219-277).
// One interval stays in registers (lo, rows); more are in cur, sorted and coalesced.  Returns
// their number (0 = no match), or ~0u on set overflow.
template <bool COUNT_TOUCH, uint32_t FMT, class SR>
__device__ __forceinline__ uint32_t backward_search_one(const DevFm& F, const SmemFm& S, const DevAux& A, const uint8_t* sym,
                                                        bool count_only, const uint8_t* p, uint32_t m, SR& cur, SR& nxt,
                                                        uint32_t cap, uint32_t& lo, uint32_t& rows, uint64_t& touches) {
  uint32_t n = 1, k;
  seed_pattern<COUNT_TOUCH>(F, A, S.dig, p, m, lo, rows, k, touches);
  if (!rows) return 0;
  while (k > 0) {
    if (FMT == OCC_NARROW && n == 1) {
      if (count_only && A.text && rows == 1 && k >= COUNT_TEXT_LEFT)
        return text_before<COUNT_TOUCH>(A, S, sym, p, k, lo, touches) ? 1u : 0u;
      const uint32_t s = sym[p[k - 1]];
      if (!s) return 0;
      if (s != SYM_MANY) {
        if (!acgt_rows<COUNT_TOUCH>(F, S.C, s, lo, rows, touches)) return 0;
        k--;
        continue;
      }
    }
    const uint8_t c = p[--k];
    const uint32_t mask = (c < 16 ? S.compat_mask[c] : 0u) & F.sym_mask;   // symbol_count(r) == 0 -> skipped
    if (!mask) return 0;
    if (FMT == OCC_WIDE && n == 1 && rows == 1) {
      uint32_t s, rk;
      row_code_rank<FMT>(F, lo, s, rk);
      if (COUNT_TOUCH) touches += 1;
      if (!((mask >> s) & 1)) return 0;
      lo = S.C[s] + rk;
      continue;
    }
    uint32_t nn = 0, f0 = 0, f1 = 0;                   // the last interval is held back: it may still grow
    bool ovf = false;
    auto add = [&](uint32_t a, uint32_t e) {           // ascending; touching neighbours are one
      if (nn && a <= f1) { f1 = max(f1, e); return; }
      if (nn) { if (nn >= cap) { ovf = true; return; } nxt[nn - 1] = make_uint2(f0, f1); }
      f0 = a; f1 = e; nn++;
    };
    if (n == 1) {
      // one source interval: symbol order is already ascending row order
      uint32_t r[16], d[16];
      rows_by_code<FMT>(F, lo, lo + rows, r, d);
      if (COUNT_TOUCH) touches += 2;
#pragma unroll
      for (int s = 0; s < 16; s++)
        if (((mask >> s) & 1) && d[s]) add(S.C[s] + r[s], S.C[s] + r[s] + d[s]);
    } else {
      // Children of symbol s lie in [C[s], C[s+1]) in source order: they are written to nxt
      // source by source, then placed into cur by symbol (a stable counting sort).  (Extending
      // the sources again to place the children: 0.64 ms against 0.49 for 500,000 patterns of
      // 32 codes on an IUPAC assembly.)
      constexpr int S0 = FMT == OCC_NARROW ? 1 : 0, S1 = FMT == OCC_NARROW ? 5 : 16;
      uint32_t cnt[16], total = 0;
#pragma unroll
      for (int s = S0; s < S1; s++) cnt[s] = 0;
      for (uint32_t i = 0; i < n; i++) {
        const uint2 iv = cur[i];
        uint32_t r[16], d[16];
        rows_by_code<FMT>(F, iv.x, iv.y, r, d);
        if (COUNT_TOUCH) touches += 2;
#pragma unroll
        for (int s = S0; s < S1; s++) {
          if (!((mask >> s) & 1) || !d[s]) continue;
          cnt[s]++;
          if (total < cap) nxt[total] = make_uint2(S.C[s] + r[s], S.C[s] + r[s] + d[s]);
          total++;
        }
        if (total > cap) return ~0u;
      }
      uint32_t below = 0;
#pragma unroll
      for (int s = S0; s < S1; s++) { const uint32_t t = cnt[s]; cnt[s] = below; below += t; }
      for (uint32_t e = 0; e < total; e++) {
        const uint2 v = nxt[e];
        uint32_t at = 0;
#pragma unroll
        for (int s = S0; s < S1; s++) {
          const bool is = v.x >= S.C[s] && (s == S1 - 1 || v.x < S.C[s + 1]);
          at = is ? cnt[s] : at;
          cnt[s] += is ? 1u : 0u;
        }
        cur[at] = v;
      }
      // coalesce touching neighbours (merge_intervals_inplace, query.rs:390-407)
      for (uint32_t e = 0; e < total; e++) { const uint2 v = cur[e]; add(v.x, v.y); }
    }
    if (ovf) return ~0u;
    if (nn == 0) return 0;
    if (nn == 1) { lo = f0; rows = f1 - f0; }
    else {
      if (nn > cap) return ~0u;
      nxt[nn - 1] = make_uint2(f0, f1);
      const SR t = cur; cur = nxt; nxt = t;
    }
    n = nn;
  }
  return n;
}

// Persistent backward search of queries 0..n-1.  Queries whose sets outgrow set_cap are listed
// for k_bsearch_warp.
template <bool COUNT_TOUCH, int STRIDE, uint32_t FMT>
__global__ void __launch_bounds__(256) k_bsearch(DevFm F, const uint16_t* __restrict__ compat_masks,
                                                const uint8_t* __restrict__ q, const uint64_t* __restrict__ qoff,
                                                uint32_t n, uint32_t hit_cap, uint2* work, uint32_t set_cap,
                                                unsigned int* queue, Pool pool, BsOut out, DevAux A) {
  __shared__ SmemFm S;
  __shared__ uint8_t s_sym[256];
  smem_fm_init(S, F, compat_masks);
  if (FMT == OCC_NARROW) sym_table_init(s_sym, compat_masks, F.sym_mask);
  __syncthreads();
  SetRef<uint2, STRIDE> A0 = thread_set<uint2, STRIDE>(work, set_cap, 2, 0);
  SetRef<uint2, STRIDE> B0 = thread_set<uint2, STRIDE>(work, set_cap, 2, 1);
  uint64_t touches = 0;
  uint32_t i;
  while (next_read(queue, n, nullptr, i)) {
    SetRef<uint2, STRIDE> cur = A0, nxt = B0;
    const uint64_t o = qoff[i];
    uint32_t lo, rows;
    uint32_t niv = backward_search_one<COUNT_TOUCH, FMT>(F, S, A, s_sym, out.nhits == nullptr, q + o,
                                                         (uint32_t)(qoff[i + 1] - o), cur, nxt, set_cap, lo, rows, touches);
    uint32_t st = ST_OK;
    if (niv == ~0u) { st = ST_SET_OVF; niv = 0; }
    uint32_t cnt = 0; uint64_t hits = 0;
    if (niv == 1) {
      cnt = rows; hits = (hit_cap && rows > hit_cap) ? hit_cap : rows;
    } else {
      for (uint32_t k = 0; k < niv; k++) {
        const uint2 v = cur[k];
        const uint32_t sz = v.y - v.x;
        cnt += sz; hits += (hit_cap && sz > hit_cap) ? hit_cap : sz;
      }
    }
    uint64_t off = 0;
    if (out.nhits && niv) {
      off = thread_reserve(pool, niv);
      if (off == ~0ull) st |= ST_POOL_OVF;
      else {
        uint2* dst = (uint2*)pool.base + off;
        if (niv == 1) dst[0] = make_uint2(lo, lo + rows);
        else for (uint32_t k = 0; k < niv; k++) dst[k] = cur[k];
      }
    }
    out.counts[i] = cnt;
    if (out.nhits) { out.nhits[i] = hits; out.niv[i] = niv; out.ivoff[i] = off; }
    out.status[i] = st;
    if (st & ST_SET_OVF) out.ovf_list[atomicAdd(out.n_ovf, 1u)] = i;
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

// =====================================================================================
// Bidirectional extension (BidirInterval::extend_right / extend_left,
// src/fm_index/bidir.rs:80-143) over a whole interval set (extend_multi_right/left,
// src/fm_index/smem.rs:332-357).  The set is emitted interval-major (the reference emits
// base-major); set order never changes which strings are found, and MEM hits are
// emitted in ascending fwd_lo order at the end.
// =====================================================================================

// A thread's interval set is kept as two lists in one slice of `cap` entries: intervals
// of one row from the front ([0, n1)) and larger ones from the back ([cap-nb, cap)).  A
// one-row interval extends only by the symbol of its row — one LF step on one record —
// so every lane runs a cheap uniform loop over its singles, then the full 16-symbol rank
// loop over the rest, instead of branching per interval (which diverges within a warp).
template <class SR>
struct TwoList {
  SR s; uint32_t n1, nb;
  __device__ __forceinline__ uint32_t size() const { return n1 + nb; }
};

// DIR 0 = right (ranks on the reverse index), 1 = left (ranks on the forward index).
template <int DIR, bool COUNT_TOUCH, uint32_t FMT, class SR>
__device__ __forceinline__ void extend_set(const DevFm& X, const SmemFm& S, uint32_t mask, const TwoList<SR>& in,
                                           TwoList<SR>& out, uint32_t cap, uint32_t& cov, bool& ovf,
                                           uint64_t& touches) {
  out.n1 = 0; out.nb = 0; cov = 0;
  const uint32_t top = mask ? 31u - __clz(mask) : 0u;     // highest code that can extend
  for (uint32_t i = 0; i < in.n1; i++) {
    BIv iv = in.s.single(i);
    uint32_t a = DIR == 0 ? iv.rlo : iv.flo, base = DIR == 0 ? iv.flo : iv.rlo;
    uint32_t s0, rk;
    row_code_rank<FMT>(X, a, s0, rk);
    if (COUNT_TOUCH) touches += 1;
    if ((mask >> s0) & 1) {
      if (out.n1 + out.nb >= cap) { ovf = true; return; }
      if (DIR == 0) out.s.set_single(out.n1++, base, S.C[s0] + rk);
      else out.s.set_single(out.n1++, S.C[s0] + rk, base);
      cov += 1;
    }
  }
  for (uint32_t k = 0; k < in.nb; k++) {
    BIv iv = in.s[cap - 1 - k];
    uint32_t a = DIR == 0 ? iv.rlo : iv.flo, b = DIR == 0 ? iv.rhi : iv.fhi;
    uint32_t base = DIR == 0 ? iv.flo : iv.rlo;
    if (COUNT_TOUCH) touches += (a != 0) + (b != 0);
    uint32_t run = 0;
    // count_smaller_than (src/fm_index/bidir.rs:125-143): the new interval of symbol s on
    // the other strand starts after every code below s, $ included
    split_by_symbol<FMT>(X, a, b, top, [&](int s, uint32_t d, uint32_t r, uint32_t sbi) {
      if (!ovf && ((mask >> s) & 1) && d) {
        if (out.n1 + out.nb >= cap) { ovf = true; return; }
        const uint32_t lo = S.C[s] + (FMT == OCC_WIDE ? r : sb_count(X, sbi, s) + r);
        if (d == 1) {
          if (DIR == 0) out.s.set_single(out.n1++, base + run, lo);
          else out.s.set_single(out.n1++, lo, base + run);
        } else {
          BIv e;
          if (DIR == 0) { e.flo = base + run; e.fhi = base + run + d; e.rlo = lo; e.rhi = lo + d; }
          else { e.flo = lo; e.fhi = lo + d; e.rlo = base + run; e.rhi = base + run + d; }
          out.s[cap - 1 - out.nb++] = e;
        }
        cov += d;
      }
      run += d;
    });
    if (ovf) return;
  }
}

// Does any interval of the set extend by a compatible symbol?
template <int DIR, bool COUNT_TOUCH, uint32_t FMT, class SR>
__device__ __forceinline__ bool any_extend(const DevFm& X, const SmemFm& S, uint32_t mask, const TwoList<SR>& in,
                                           uint32_t cap, uint64_t& touches) {
  bool any = false;
  const uint32_t top = mask ? 31u - __clz(mask) : 0u;
  for (uint32_t i = 0; i < in.n1; i++) {
    BIv iv = in.s.single(i);
    uint32_t s0, rk;
    row_code_rank<FMT>(X, DIR == 0 ? iv.rlo : iv.flo, s0, rk);
    if (COUNT_TOUCH) touches += 1;
    any |= (mask >> s0) & 1;
  }
  if (any) return true;
  for (uint32_t k = 0; k < in.nb; k++) {
    BIv iv = in.s[cap - 1 - k];
    uint32_t a = DIR == 0 ? iv.rlo : iv.flo, b = DIR == 0 ? iv.rhi : iv.fhi;
    if (COUNT_TOUCH) touches += (a != 0) + (b != 0);
    split_by_symbol<FMT>(X, a, b, top, [&](int s, uint32_t d, uint32_t, uint32_t) { any |= ((mask >> s) & 1) && d; });
    if (any) return true;
  }
  return false;
}

struct Cand { uint32_t qs, qe, count, nivs; uint64_t ivoff; uint32_t pivot, _pad; };

struct MemsOut {
  uint64_t* hit_start;      // per slot (read or segment): offset of its hits in the hit pool
  uint32_t* hit_count;      // per slot: number of hits
  uint64_t* pos_count;      // per slot: positions of its hits
  uint32_t* status;
  uint32_t* ovf_list;
  uint32_t* n_ovf;
  unsigned long long* touches;
};

struct MemsParams {
  uint32_t min_len, mode, max_hits, resolve;   // resolve = ref bounds given
};

// Shell sort of a set by fwd_lo (hits of one MEM in ascending fwd_lo order).
__device__ __forceinline__ void sort_by_flo(BIv* a, uint32_t n) {
  for (uint32_t gap = n / 2; gap > 0; gap /= 2)
    for (uint32_t i = gap; i < n; i++) {
      BIv t = a[i]; uint32_t j = i;
      while (j >= gap && a[j - gap].flo > t.flo) { a[j] = a[j - gap]; j -= gap; }
      a[j] = t;
    }
}

// The full interval (the empty pattern) as a one-element two-list set.
template <class SR>
__device__ __forceinline__ void start_full(TwoList<SR>& t, const BIv& full, uint32_t set_cap) {
  if (full.fhi - full.flo == 1) { t.s.set_single(0, full.flo, full.rlo); t.n1 = 1; t.nb = 0; }
  else { t.s[set_cap - 1] = full; t.n1 = 0; t.nb = 1; }
}

__device__ __forceinline__ uint32_t qmask(const SmemFm& S, uint8_t c) { return c < 16 ? S.compat_mask[c] : 0u; }

// One pivot of the SMEM sweep (collect_smem_candidates loop body,
// src/fm_index/smem.rs:154-222): forward extension from `pivot`, every right-maximal prefix
// extended left maximally (extend_left_maximally, smem.rs:227-243), candidates passed to
// emit(qs, qe, count, set, pivot).  Returns the next pivot, max(reach, pivot + 1), or ~0u
// on overflow (flags in st).  The sweep is a chain pivot -> next(pivot) that depends only
// on the read, which is what lets a long read be cut into independently swept segments.
template <bool COUNT_TOUCH, uint32_t FMT, class SR, class Emit>
__device__ __forceinline__ uint32_t smem_pivot(const DevFm& Fw, const DevFm& Rv, const SmemFm& Sf, const SmemFm& Sr,
                                               const uint8_t* q, uint32_t n, uint32_t pivot, const MemsParams& P,
                                               const SR& curr, const SR& nxt, const SR& wa, const SR& wb,
                                               uint32_t set_cap, uint32_t& st, uint64_t& touches, Emit& emit) {
  using TL = TwoList<SR>;
  const BIv full = {0, Fw.text_len, 0, Fw.text_len};
  bool ovf = false;
  TL c{curr, 0, 0}, x{nxt, 0, 0};
  start_full(x, full, set_cap);
  uint32_t cov;
  extend_set<0, COUNT_TOUCH, FMT>(Rv, Sr, qmask(Sr, q[pivot]), x, c, set_cap, cov, ovf, touches);
  if (ovf) { st |= ST_SET_OVF; return ~0u; }
  if (c.size() == 0) return pivot + 1;
  uint32_t j = pivot + 1, reach = pivot + 1;
  for (;;) {
    uint32_t end, ncov = 0;
    bool next_empty, record;
    x.n1 = x.nb = 0;
    if (j == n) { end = n; next_empty = true; record = true; }
    else {
      extend_set<0, COUNT_TOUCH, FMT>(Rv, Sr, qmask(Sr, q[j]), c, x, set_cap, ncov, ovf, touches);
      if (ovf) { st |= ST_SET_OVF; return ~0u; }
      end = j; next_empty = x.size() == 0; record = ncov != cov;
    }
    if (record) {
      // right-maximal prefix [pivot, end): extend_left_maximally (smem.rs:227-243)
      reach = end;
      TL b = c;
      uint32_t start = pivot, bcov = cov;
      TL bufs[2] = {TL{wa, 0, 0}, TL{wb, 0, 0}};
      int t = 0;
      while (start > 0) {
        uint32_t lcov;
        extend_set<1, COUNT_TOUCH, FMT>(Fw, Sf, qmask(Sf, q[start - 1]), b, bufs[t], set_cap, lcov, ovf, touches);
        if (ovf) { st |= ST_SET_OVF; return ~0u; }
        if (bufs[t].size() == 0) break;
        b = bufs[t]; bcov = lcov; t ^= 1; start--;
      }
      if (end - start >= P.min_len) {
        // right-maximality (smem.rs:202-207); with no left extension it is next_empty
        bool rmax = end == n ||
                    (start == pivot ? next_empty : !any_extend<0, COUNT_TOUCH, FMT>(Rv, Sr, qmask(Sr, q[end]), b, set_cap, touches));
        if (rmax && !emit(start, end, bcov, b, pivot)) return ~0u;
      }
    }
    if (j == n || x.size() == 0) break;
    TL tt = c; c = x; x = tt; cov = ncov; j++;
  }
  return max(reach, pivot + 1);
}

// Appends candidates (with their interval sets copied to the interval pool) to a list.
template <class SR>
struct CandSink {
  Cand* cands; uint32_t nc, cap; Pool* ivpool; uint32_t* st; uint32_t set_cap;
  __device__ __forceinline__ bool operator()(uint32_t qs, uint32_t qe, uint32_t count, const TwoList<SR>& ivs,
                                             uint32_t pivot) {
    if (nc >= cap) { *st |= ST_CAND_OVF; return false; }
    uint32_t niv = ivs.size();
    uint64_t off = thread_reserve(*ivpool, niv);
    if (off == ~0ull) { *st |= ST_POOL_OVF; return false; }
    BIv* dst = (BIv*)ivpool->base + off;
    for (uint32_t k = 0; k < ivs.n1; k++) dst[k] = ivs.s.single(k);
    for (uint32_t k = 0; k < ivs.nb; k++) dst[ivs.n1 + k] = ivs.s[set_cap - 1 - k];
    cands[nc++] = Cand{qs, qe, count, niv, off, pivot, 0u};
    return true;
  }
};

// Candidate search for one read into `sink` (find_mems or find_smems candidates).  Returns
// the number of candidates, or ~0u on overflow of a set, the candidate list or the
// interval pool (flags in st).
template <bool COUNT_TOUCH, uint32_t FMT, class SR, class Sink>
__device__ uint32_t mems_sweep(const DevFm& Fw, const DevFm& Rv, const SmemFm& Sf, const SmemFm& Sr,
                               const uint8_t* q, uint32_t n, const MemsParams& P, const SR& curr, const SR& nxt,
                               const SR& wa, const SR& wb, uint32_t set_cap, Sink& sink, uint32_t& st,
                               uint64_t& touches) {
  using TL = TwoList<SR>;
  if (n == 0 || P.min_len == 0) return 0;
  const BIv full = {0, Fw.text_len, 0, Fw.text_len};
  bool ovf = false;
  if (P.mode == 1) {
    // find_mems: raw_mem_from(i) for every start (src/fm_index/smem.rs:250-295)
    for (uint32_t i = 0; i < n; i++) {
      TL c{curr, 0, 0}, x{nxt, 0, 0};
      start_full(c, full, set_cap);
      uint32_t cov = 0, j = i;
      bool matched = false;
      while (j < n) {
        uint32_t ncov;
        extend_set<0, COUNT_TOUCH, FMT>(Rv, Sr, qmask(Sr, q[j]), c, x, set_cap, ncov, ovf, touches);
        if (ovf) { st |= ST_SET_OVF; return ~0u; }
        if (x.size() == 0) break;
        TL t = c; c = x; x = t; cov = ncov; j++; matched = true;
      }
      if (!matched || j - i < P.min_len) continue;
      bool lmax = i == 0 || !any_extend<1, COUNT_TOUCH, FMT>(Fw, Sf, qmask(Sf, q[i - 1]), c, set_cap, touches);
      if (!lmax) continue;
      if (!sink(i, j, cov, c, i)) return ~0u;
    }
    return sink.nc;
  }
  // find_smems: collect_smem_candidates (src/fm_index/smem.rs:154-222)
  uint32_t pivot = 0;
  while (pivot < n) {
    pivot = smem_pivot<COUNT_TOUCH, FMT>(Fw, Rv, Sf, Sr, q, n, pivot, P, curr, nxt, wa, wb, set_cap, st, touches, sink);
    if (pivot == ~0u) return ~0u;
  }
  return sink.nc;
}

// Sort candidates by (qs, qe) (stable), drop duplicates, keep the containment-maximal ones
// (find_smems, src/fm_index/smem.rs:84-103).  Returns the survivors compacted in place.
__device__ __forceinline__ uint32_t finalize_smems(Cand* c, uint32_t n) {
  for (uint32_t i = 1; i < n; i++) {           // insertion sort
    Cand t = c[i]; uint32_t j = i;
    while (j > 0 && (c[j - 1].qs > t.qs || (c[j - 1].qs == t.qs && c[j - 1].qe > t.qe))) { c[j] = c[j - 1]; j--; }
    c[j] = t;
  }
  uint32_t w = 0;
  for (uint32_t i = 0; i < n; i++)
    if (w == 0 || c[w - 1].qs != c[i].qs || c[w - 1].qe != c[i].qe) c[w++] = c[i];
  n = w; w = 0;
  // Sorted by (qs, qe) and distinct, c[i] lies inside another candidate exactly when the
  // next one shares its start (and so ends later) or an earlier one (qs <= c[i].qs) ends
  // at or after c[i].qe: a running maximum of qe replaces the all-pairs test.
  uint32_t max_qe = 0;
  bool any = false;
  for (uint32_t i = 0; i < n; i++) {
    bool contained = (i + 1 < n && c[i + 1].qs == c[i].qs) || (any && max_qe >= c[i].qe);
    uint32_t qe = c[i].qe;
    if (!any || qe > max_qe) max_qe = qe;
    any = true;
    if (!contained) c[w++] = c[i];
  }
  return w;
}

// Writes the hits of one read (one per SA interval of each surviving MEM) into the hit
// pool; returns false on pool exhaustion.
__device__ __forceinline__ bool write_hits(Cand* c, uint32_t n, const MemsParams& P, Pool& ivpool,
                                           Pool& hitpool, uint64_t& start, uint32_t& count, uint64_t& positions) {
  uint32_t total = 0;
  positions = 0;
  for (uint32_t k = 0; k < n; k++) total += c[k].nivs;
  count = total;
  if (total == 0) { start = 0; return true; }
  uint64_t off = thread_reserve(hitpool, total);
  if (off == ~0ull) return false;
  start = off;
  uint32_t* h = (uint32_t*)hitpool.base + off * 8;
  for (uint32_t k = 0; k < n; k++) {
    BIv* ivs = (BIv*)ivpool.base + c[k].ivoff;
    sort_by_flo(ivs, c[k].nivs);
    for (uint32_t t = 0; t < c[k].nivs; t++) {
      uint32_t sz = ivs[t].fhi - ivs[t].flo;
      uint32_t eff = P.resolve ? min(sz, P.max_hits) : 0u;
      positions += eff;
      uint4 a = make_uint4(c[k].qs, c[k].qe, sz, sz > P.max_hits ? 1u : 0u);
      uint4 b = make_uint4(ivs[t].flo, eff, 0u, 0u);
      reinterpret_cast<uint4*>(h)[0] = a; reinterpret_cast<uint4*>(h)[1] = b;
      h += 8;
    }
  }
  return true;
}

struct MemsWork {
  BIv* sets; uint32_t set_cap;        // two sets per thread (per lane group)
  Cand* cands; uint32_t cand_cap;     // lane-group kernels: candidate list per group
  uint4* hits; uint32_t hit_cap;      // per-thread kernel: hit list per thread (two uint4 a hit)
  unsigned int* queue;
  const uint32_t* ids; uint32_t n;    // lane-group kernels: reads to process, in queue order
  uint32_t* still_ovf;
  uint32_t rerun;                     // 1: a rerun of overflowed reads (counted in still_ovf)
  uint32_t* work_log;                 // COUNT_TOUCH only: 4 u32 per read, [0] += Occ touches, [3] |= 1 on overflow
                                      // (the lane-group kernels also set bit 1)
  const uint32_t* n_dev;              // when set, the number of reads is read here (graph-captured chains)
  uint32_t chunk;                     // queue entries taken per atomic (0 or 1: one)
  const uint64_t* slot_base;          // first result slot of each read (nullptr: slot = read)
  __device__ __forceinline__ uint32_t count() const { return n_dev ? *n_dev : n; }
  __device__ __forceinline__ uint32_t step() const { return chunk > 1 ? chunk : 1u; }
};

// Splits the fast pass's overflow list: the first `first_warp` entries (reads a schedule
// routed) and reads whose interval sets overflowed go to the warp-per-read list; reads that
// outgrew only the candidate list go to the per-thread rerun with a larger global list.
__global__ void k_split_ovf(const uint32_t* __restrict__ list, uint32_t n, uint32_t first_warp,
                            const uint32_t* __restrict__ status, uint32_t* __restrict__ mid,
                            uint32_t* __restrict__ n_mid, uint32_t* __restrict__ wrp, uint32_t* __restrict__ n_wrp,
                            const uint32_t* __restrict__ n_dev = nullptr) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (n_dev ? *n_dev : n)) return;
  uint32_t i = list[k];
  if (k < first_warp || (status[i] & ST_SET_OVF)) wrp[atomicAdd(n_wrp, 1u)] = i;
  else mid[atomicAdd(n_mid, 1u)] = i;
}

// =====================================================================================
// The plain launch: one thread per read over a grid the size of the batch, interval sets
// and candidate list in the thread's local memory, and a count pass before the write pass
// whose totals the host reads back to size the outputs — the structure of the reference's
// GPU search (one invocation per query, count-then-write, host prefix sum;
// shaders/mem_find.wgsl:179-372, src/gpu/mem_find.rs:213-244) restated with the CPU
// semantics.  It is the baseline the persistent path is measured against.  Reads whose
// sets or candidates outgrow the local capacity go to the warp-per-read kernel, so the
// results are those of every other path.
// =====================================================================================
constexpr uint32_t PLAIN_SET_CAP = 64;
constexpr int PLAIN_KC = 32;

// Count-pass sink: candidates with their MemHit count (nivs) and position count (in
// ivoff), no interval copies.
template <class SR>
struct CountSink {
  Cand* cands; uint32_t nc, cap; uint32_t* st; uint32_t set_cap; uint32_t max_hits, resolve;
  unsigned long long ivs_all;       // intervals of every candidate (the write pass's pool need)
  __device__ __forceinline__ bool operator()(uint32_t qs, uint32_t qe, uint32_t count, const TwoList<SR>& ivs,
                                             uint32_t pivot) {
    if (nc >= cap) { *st |= ST_CAND_OVF; return false; }
    uint64_t npos = 0;
    if (resolve) {
      npos = max_hits ? ivs.n1 : 0u;
      for (uint32_t k = 0; k < ivs.nb; k++) {
        BIv iv = ivs.s[set_cap - 1 - k];
        npos += min(iv.fhi - iv.flo, max_hits);
      }
    }
    ivs_all += ivs.size();
    cands[nc++] = Cand{qs, qe, count, ivs.size(), npos, pivot, 0u};
    return true;
  }
};

template <bool COUNT_TOUCH, int PASS, uint32_t FMT>
__global__ void __launch_bounds__(128) k_mems_plain(DevFm Fw, DevFm Rv, const uint16_t* __restrict__ compat_fw,
                                                   const uint16_t* __restrict__ compat_rv, const uint8_t* __restrict__ q,
                                                   const uint64_t* __restrict__ qoff, MemsParams P, uint32_t n,
                                                   Pool ivpool, Pool hitpool, MemsOut out, uint32_t* pos_count,
                                                   unsigned long long* ivs_need) {
  __shared__ SmemFm Sf, Sr;
  smem_fm_init(Sf, Fw, compat_fw);
  smem_fm_init(Sr, Rv, compat_rv);
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  using SR = SetRef<BIv, 1>;
  uint32_t lset[4][3 * PLAIN_SET_CAP];
  SR s0{lset[0], PLAIN_SET_CAP}, s1{lset[1], PLAIN_SET_CAP}, s2{lset[2], PLAIN_SET_CAP}, s3{lset[3], PLAIN_SET_CAP};
  Cand cands[PLAIN_KC];
  uint64_t touches = 0;
  const uint64_t o = qoff[i];
  const uint32_t len = (uint32_t)(qoff[i + 1] - o);
  if (PASS == 0) {
    uint32_t st = ST_OK;
    CountSink<SR> sink{cands, 0, (uint32_t)PLAIN_KC, &st, PLAIN_SET_CAP, P.max_hits, P.resolve, 0ull};
    uint32_t nc = mems_sweep<COUNT_TOUCH, FMT>(Fw, Rv, Sf, Sr, q + o, len, P, s0, s1, s2, s3, PLAIN_SET_CAP, sink, st,
                                               touches);
    uint32_t hits = 0, pos = 0;
    if (nc != ~0u) {
      if (P.mode == 0) nc = finalize_smems(cands, nc);
      for (uint32_t k = 0; k < nc; k++) { hits += cands[k].nivs; pos += (uint32_t)cands[k].ivoff; }
      atomicAdd(ivs_need, sink.ivs_all);
    }
    if (st) { hits = 0; pos = 0; }
    out.hit_count[i] = hits; pos_count[i] = pos; out.status[i] = st;
  } else {
    // reads the count pass found too large for local memory keep their flags; a pool
    // overflow of an earlier attempt is cleared (the host regrew the pools)
    uint32_t st = out.status[i] & (ST_SET_OVF | ST_CAND_OVF);
    uint64_t hs = 0, hp = 0; uint32_t hc = 0;
    if (st == ST_OK) {
      CandSink<SR> sink{cands, 0, (uint32_t)PLAIN_KC, &ivpool, &st, PLAIN_SET_CAP};
      uint32_t nc = mems_sweep<COUNT_TOUCH, FMT>(Fw, Rv, Sf, Sr, q + o, len, P, s0, s1, s2, s3, PLAIN_SET_CAP, sink,
                                                 st, touches);
      if (nc != ~0u) {
        if (P.mode == 0) nc = finalize_smems(cands, nc);
        if (!write_hits(cands, nc, P, ivpool, hitpool, hs, hc, hp)) st |= ST_POOL_OVF;
      }
      if (st) { hs = 0; hc = 0; hp = 0; }
    }
    out.status[i] = st;
    out.hit_start[i] = hs; out.hit_count[i] = hc; out.pos_count[i] = hp;
    if (st & (ST_SET_OVF | ST_CAND_OVF)) out.ovf_list[atomicAdd(out.n_ovf, 1u)] = i;
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

// =====================================================================================
// Long reads are cut into segments of seg_len positions (smem.cuh): the lists of their
// segments and of the reads in one piece.
// =====================================================================================
constexpr uint32_t SEG_MAX = 4096;   // longest segment

// The segment length of a batch: the tuned one, or for an ACGT text (threads > 0) a smaller
// one, down to 64, while the batch's codes do not give every resident thread SEGS_PER_THREAD
// segments of it: a small batch is bound by its longest chain of steps, which is a segment's
// length plus a match, and a larger one by the last segments while most lanes are idle.
// (Search of 60,000 mixed reads up to 10 kbp, 49 M codes for 151,552 threads: 3.2 ms at 512,
// 2.2 at 256, 2.0 at 128, 2.3 at 64, where the windows that segments share cost more.)
constexpr uint64_t SEGS_PER_THREAD = 4;
__device__ __forceinline__ uint32_t batch_seg_len(uint64_t bases, uint32_t seg_len, uint64_t threads) {
  if (!threads) return seg_len;
  uint32_t s = 64;
  while (s < seg_len && bases / s > SEGS_PER_THREAD * threads) s *= 2;
  return min(s, seg_len);
}

// Reads ids[k] (k itself without ids): flags[k] = 1 when the read is longer than two
// segments, nslot[read] = its segments (1 for a read in one piece), and the totals.
__global__ void k_long_reads(const uint32_t* __restrict__ ids, uint32_t n, const uint64_t* __restrict__ qoff,
                             uint32_t nq, uint32_t tuned_len, uint64_t threads, uint32_t* __restrict__ flags,
                             uint32_t* __restrict__ nslot, uint32_t* __restrict__ n_long,
                             unsigned long long* __restrict__ n_units, uint32_t* __restrict__ used_len,
                             unsigned long long* __restrict__ bases) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t seg_len = batch_seg_len(qoff[nq] - qoff[0], tuned_len, threads);
  if (k == 0) { *used_len = seg_len; *bases = qoff[nq] - qoff[0]; }
  const uint32_t i = ids ? ids[k] : k;
  const uint64_t len = qoff[i + 1] - qoff[i];
  const bool is_long = len > 2 * (uint64_t)seg_len;
  const uint32_t segs = is_long ? (uint32_t)((len + seg_len - 1) / seg_len) : 1u;
  flags[k] = is_long ? 1u : 0u;
  nslot[i] = segs;
  if (is_long) { atomicAdd(n_long, 1u); atomicAdd(n_units, (unsigned long long)segs); }
}

// out[list[k]] = v.
__global__ void k_fill_listed(const uint32_t* __restrict__ list, uint32_t n, uint32_t* __restrict__ out, uint32_t v) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[list[k]] = v;
}

// hit_base[i] = first hit of read i = first hit of its first slot (i <= n).
__global__ void k_slot_to_read(const uint64_t* __restrict__ slot_hits, const uint64_t* __restrict__ slot_base, uint32_t n,
                               uint64_t* __restrict__ hit_base) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= n) hit_base[i] = slot_hits[slot_base[i]];
}

// Stable split of ids by flag (lpos = exclusive scan of flags).
__global__ void k_split_ids(const uint32_t* __restrict__ ids, uint32_t n, const uint32_t* __restrict__ flags,
                            const uint64_t* __restrict__ lpos, uint32_t* __restrict__ short_ids,
                            uint32_t* __restrict__ long_ids, uint32_t* __restrict__ seg_count,
                            const uint64_t* __restrict__ qoff, uint32_t seg_len) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  uint32_t i = ids ? ids[k] : k;
  uint32_t l = (uint32_t)lpos[k];
  if (flags[k]) {
    long_ids[l] = i;
    uint32_t len = (uint32_t)(qoff[i + 1] - qoff[i]);
    seg_count[l] = (len + seg_len - 1) / seg_len;
  } else {
    short_ids[k - l] = i;
  }
}

__global__ void k_unit_fill(const uint32_t* __restrict__ long_ids, uint32_t n_long,
                            const uint64_t* __restrict__ unit_base, uint32_t* __restrict__ unit_read,
                            uint32_t* __restrict__ unit_k, const uint64_t* __restrict__ n_long_dev = nullptr) {
  uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (n_long_dev ? (uint32_t)*n_long_dev : n_long)) return;
  uint64_t b = unit_base[r], e = unit_base[r + 1];
  for (uint64_t u = b; u < e; u++) { unit_read[u] = long_ids[r]; unit_k[u] = (uint32_t)(u - b); }
}

}  // namespace hfm

// =====================================================================================
// Warp-cooperative long-tail pass: one warp per read, the 32 lanes share the interval set
// of every step (reads whose sets outgrow the per-thread fast path: ambiguity codes near
// the start of a read, unseeded patterns inside N runs).  Same results as the per-thread
// code; sets live in a per-warp global region.
// =====================================================================================
namespace hfm {

__device__ __forceinline__ uint32_t lane_lt_mask() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
  return v;
}
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t& total) {
  const int lane = threadIdx.x & 31;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) { uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d); if (lane >= d) x += y; }
  total = __shfl_sync(0xFFFFFFFFu, x, 31);
  return x - v;
}

// Lane groups of G = 4, 8, 16 or 32 lanes (one read per group in the sub-warp and
// warp-per-read SMEM kernels): the group's member mask, sum and exclusive scan.
template <int G>
__device__ __forceinline__ uint32_t grp_mask() {
  if (G == 32) return 0xFFFFFFFFu;
  return ((1u << G) - 1u) << ((threadIdx.x & 31) & ~(uint32_t)(G - 1));
}
template <int G>
__device__ __forceinline__ uint32_t grp_sum(uint32_t v) {
  const uint32_t m = grp_mask<G>();
#pragma unroll
  for (int d = G / 2; d > 0; d >>= 1) v += __shfl_xor_sync(m, v, d, G);
  return v;
}
template <int G>
__device__ __forceinline__ uint32_t grp_excl_scan(uint32_t v, uint32_t& total) {
  const uint32_t m = grp_mask<G>();
  const int gl = threadIdx.x & (G - 1);
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < G; d <<= 1) { uint32_t y = __shfl_up_sync(m, x, d, G); if (gl >= d) x += y; }
  total = __shfl_sync(m, x, G - 1, G);
  return x - v;
}

// Backward search of one pattern by a warp.  The sources are extended once, 32 at a time and
// only by the symbols of the code; the children are placed by symbol (a stable counting sort);
// then touching neighbours are coalesced: an interval is the first of its run when it does not
// touch the one before it, so a run's place is the number of firsts up to it and every lane
// writes the ends that it knows.  Bound by the chain of dependent loads of a pattern, some 90
// groups of 32 intervals on an IUPAC assembly.  5,000 patterns with an N among the seeded codes,
// of 500,000: 2.4 ms when lane 0 coalesced alone, 1.1 when the sources were extended a second
// time to place the children, 0.8 now.
template <bool COUNT_TOUCH, uint32_t FMT>
__device__ uint32_t warp_backward_search(const DevFm& F, const SmemFm& S, const DevAux& A, const uint8_t* p, uint32_t m,
                                         uint2*& cur, uint2*& nxt, uint32_t cap, uint64_t& touches) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = lane_lt_mask();
  uint32_t lo, rows, start;
  uint64_t seeds = 0;
  seed_pattern<COUNT_TOUCH>(F, A, S.dig, p, m, lo, rows, start, seeds);
  if (lane == 0) touches += seeds;
  if (!rows) return 0;
  if (lane == 0) cur[0] = make_uint2(lo, lo + rows);
  uint32_t n = 1;
  __syncwarp();
  for (uint32_t k = start; k-- > 0;) {
    const uint8_t c = p[k];
    const uint32_t mask = (c < 16 ? S.compat_mask[c] : 0) & F.sym_mask;
    if (!mask) return 0;
    // extend: 32 sources at a time, symbol by symbol; lane s < 16 counts the children of s
    uint32_t total = 0, mine = 0;
    for (uint32_t b = 0; b < n; b += 32) {
      const uint32_t i = b + lane;
      const uint2 iv = i < n ? cur[i] : make_uint2(0, 1);
      if (COUNT_TOUCH && i < n) touches += 2;
      each_code<FMT>(F, iv.x, iv.y, mask, [&](int s, uint32_t r, uint32_t d) {
        const bool e = i < n && d;
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, e), at = total + __popc(bal & lt), k = __popc(bal);
        if (e && at < cap) nxt[at] = make_uint2(S.C[s] + r, S.C[s] + r + d);
        mine += lane == s ? k : 0u;
        total += k;
      });
      if (total > cap) return ~0u;
    }
    if (total == 0) return 0;
    __syncwarp();
    // place: a child's symbol is that of the C range that holds it; its place, the symbol's
    // first, the earlier ones of the symbol and those of lower lanes
    uint32_t all;
    uint32_t place = grp_excl_scan<32>(mine, all);                 // lane s: the next place of symbol s
    for (uint32_t b = 0; b < total; b += 32) {
      const uint32_t i = b + lane;
      const uint2 v = i < total ? nxt[i] : make_uint2(0, 0);
      uint32_t s = 0;
#pragma unroll
      for (int t = 1; t < 16; t++) s += v.x >= S.C[t] ? 1u : 0u;
      uint32_t same = __ballot_sync(0xFFFFFFFFu, i < total), own = same;   // of this child's symbol; of symbol `lane`
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const uint32_t bit = __ballot_sync(0xFFFFFFFFu, s >> t & 1);
        same &= s >> t & 1 ? bit : ~bit;
        own &= lane >> t & 1 ? bit : ~bit;
      }
      const uint32_t at = __shfl_sync(0xFFFFFFFFu, place, s) + __popc(same & lt);
      if (i < total) cur[at] = v;
      place += __popc(own);
    }
    __syncwarp();
    // coalesce touching neighbours in place (merge_intervals_inplace, query.rs:390-407)
    uint32_t nn = 0, before = 0;                        // runs so far; end of the interval before this chunk
    for (uint32_t b = 0; b < total; b += 32) {
      const uint32_t i = b + lane;
      const uint2 v = i < total ? cur[i] : make_uint2(0, 0);
      uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, v.y, 1);
      if (lane == 0) prev = before;
      const bool first = i < total && (i == 0 || v.x > prev);
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, first);
      const uint32_t run = nn + __popc(bal & (lt | 1u << lane));          // runs up to and with this interval
      if (first) {
        cur[run - 1].x = v.x;
        if (i) cur[run - 2].y = prev;
      }
      nn += __popc(bal);
      before = __shfl_sync(0xFFFFFFFFu, v.y, 31);
      if (i == total - 1) cur[run - 1].y = v.y;
    }
    __syncwarp();
    n = nn;
  }
  return n;
}

template <bool COUNT_TOUCH, uint32_t FMT>
__global__ void __launch_bounds__(128) k_bsearch_warp(DevFm F, const uint16_t* __restrict__ compat_masks,
                                                     const uint8_t* __restrict__ q, const uint64_t* __restrict__ qoff,
                                                     const uint32_t* __restrict__ ids, uint32_t n, uint32_t hit_cap,
                                                     uint2* work, uint32_t set_cap, unsigned int* queue, Pool pool,
                                                     BsOut out, uint32_t* still_ovf, DevAux X,
                                                     const uint32_t* __restrict__ n_dev = nullptr) {
  __shared__ SmemFm S;
  smem_fm_init(S, F, compat_masks);
  __syncthreads();
  if (n_dev) n = *n_dev;                   // graph-captured chains: the count is on the device
  const int lane = threadIdx.x & 31;
  uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint2* A = work + warp * 2 * set_cap;
  uint2* B = A + set_cap;
  uint64_t touches = 0;
  for (;;) {
    uint32_t k = 0;
    if (lane == 0) k = atomicAdd(queue, 1u);
    k = __shfl_sync(0xFFFFFFFFu, k, 0);
    if (k >= n) break;
    uint32_t i = ids[k];
    uint2* cur = A; uint2* nxt = B;
    uint64_t o = qoff[i];
    uint32_t niv = warp_backward_search<COUNT_TOUCH, FMT>(F, S, X, q + o, (uint32_t)(qoff[i + 1] - o), cur, nxt, set_cap, touches);
    if (niv == ~0u) {
      if (lane == 0) { atomicAdd(still_ovf, 1u); out.status[i] = ST_SET_OVF; }
      continue;
    }
    uint32_t cnt = 0; uint64_t hits = 0;
    for (uint32_t b = lane; b < niv; b += 32) {
      uint2 v = cur[b]; uint32_t sz = v.y - v.x;
      cnt += sz; hits += (hit_cap && sz > hit_cap) ? hit_cap : sz;
    }
    cnt = warp_sum(cnt);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) hits += __shfl_xor_sync(0xFFFFFFFFu, hits, d);
    uint64_t off = 0; uint32_t st = ST_OK;
    if (out.nhits && niv) {
      if (lane == 0) off = thread_reserve(pool, niv);
      off = __shfl_sync(0xFFFFFFFFu, off, 0);
      if (off == ~0ull) st = ST_POOL_OVF;
      else { uint2* dst = (uint2*)pool.base + off; for (uint32_t b = lane; b < niv; b += 32) dst[b] = cur[b]; }
    }
    if (lane == 0) {
      out.counts[i] = cnt;
      if (out.nhits) { out.nhits[i] = hits; out.niv[i] = niv; out.ivoff[i] = off; }
      out.status[i] = st;
    }
    __syncwarp();
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

// One extension of the whole set by a group of G lanes (outputs in lane-chunk order).
template <int DIR, bool COUNT_TOUCH, int G = 32>
__device__ uint32_t warp_extend_set(const DevFm& X, const SmemFm& S, uint32_t mask, const BIv* in, uint32_t nin,
                                    BIv* out, uint32_t cap, uint32_t& cov, bool& ovf, uint64_t& touches) {
  const int lane = threadIdx.x & (G - 1);
  uint32_t nout = 0, covl = 0;
  for (uint32_t b = 0; b < nin; b += G) {
    uint32_t i = b + lane;
    BIv iv = i < nin ? in[i] : BIv{0, 0, 0, 0};
    uint32_t a = DIR == 0 ? iv.rlo : iv.flo, e = DIR == 0 ? iv.rhi : iv.fhi;
    uint32_t base = DIR == 0 ? iv.flo : iv.rlo;
    uint32_t rl[16], rh[16];
    sym_ranks(X, S, a, rl);
    sym_ranks(X, S, e, rh);
    if (COUNT_TOUCH && i < nin) touches += (a != 0) + (e != 0);
    uint32_t k = 0;
#pragma unroll
    for (int s = 0; s < 16; s++) k += (i < nin && ((mask >> s) & 1) && rh[s] > rl[s]) ? 1u : 0u;
    uint32_t total;
    uint32_t pos = nout + grp_excl_scan<G>(k, total);
    if (nout + total > cap) { ovf = true; return nout; }
    uint32_t run = 0;
#pragma unroll
    for (int s = 0; s < 16; s++) {
      uint32_t d = rh[s] - rl[s];
      if (i < nin && ((mask >> s) & 1) && d) {
        BIv o;
        if (DIR == 0) { o.flo = base + run; o.fhi = base + run + d; o.rlo = S.C[s] + rl[s]; o.rhi = S.C[s] + rh[s]; }
        else { o.flo = S.C[s] + rl[s]; o.fhi = S.C[s] + rh[s]; o.rlo = base + run; o.rhi = base + run + d; }
        out[pos++] = o;
        covl += d;
      }
      run += d;
    }
    nout += total;
  }
  cov = grp_sum<G>(covl);
  __syncwarp(grp_mask<G>());
  return nout;
}

// Codes of several symbols that a window may hold and still be searched from its end, and the
// run of ACGT that a search is started from without looking for a longer one.
constexpr uint32_t SEED_AMBIGUOUS = 3, SEED_RUN = 12;

// Where the search of the window q[i, e) starts: its codes before the returned place are taken
// to the left first, those from it on to the right after them.  A code that matches nothing
// ends the window at once.
__device__ __forceinline__ uint32_t seed_end(const uint16_t* compat, const uint8_t* q, uint32_t i, uint32_t e) {
  uint32_t run = 0, best = 0, at = e, others = 0;
  for (uint32_t k = e; k > i && best < SEED_RUN; k--) {
    const uint32_t c = q[k - 1];
    if (c > 15 || !compat[c]) return k;
    if (c <= 4) {
      if (++run > best) { best = run; at = k - 1 + run; }
    } else {
      run = 0;
      others++;
    }
  }
  return others > SEED_AMBIGUOUS ? at : e;
}

// The search of one read (window, forward, next: smem.cuh) by a group of G lanes; control
// flow is group-uniform.
template <bool COUNT_TOUCH, int G = 32>
__device__ uint32_t warp_mems_one(const DevFm& Fw, const DevFm& Rv, const SmemFm& Sf, const SmemFm& Sr,
                                  const uint8_t* q, uint32_t n, const MemsParams& P, BIv* cur, BIv* alt,
                                  uint32_t set_cap, Cand* cands, uint32_t cand_cap, Pool& ivpool,
                                  uint32_t& st, uint64_t& touches) {
  const int lane = threadIdx.x & (G - 1);
  const uint32_t gm = grp_mask<G>();
  uint32_t nc = 0;
  if (n == 0 || P.min_len == 0) return 0;
  uint32_t ncur = 0, cov;
  bool ovf = false;
  auto reset = [&]() {
    __syncwarp(gm);
    if (lane == 0) cur[0] = BIv{0, Fw.text_len, 0, Fw.text_len};
    __syncwarp(gm);
    ncur = 1;
  };
  // one step; false, with the set as it was, when nothing extends (or the set outgrew its area)
  auto left = [&](uint32_t pos) -> bool {
    uint32_t m = warp_extend_set<1, COUNT_TOUCH, G>(Fw, Sf, qmask(Sf, q[pos]), cur, ncur, alt, set_cap, cov, ovf, touches);
    if (ovf || m == 0) return false;
    BIv* t = cur; cur = alt; alt = t; ncur = m;
    return true;
  };
  auto right = [&](uint32_t pos) -> bool {
    uint32_t m = warp_extend_set<0, COUNT_TOUCH, G>(Rv, Sr, qmask(Sr, q[pos]), cur, ncur, alt, set_cap, cov, ovf, touches);
    if (ovf || m == 0) return false;
    BIv* t = cur; cur = alt; alt = t; ncur = m;
    return true;
  };
  uint32_t i = 0;
  while (n - i >= P.min_len) {
    reset();
    // from the window's end, and from its seed_end where that gives a large set (looking for it
    // in every window costs a load's wait: 4% with a warp a read).  Smaller groups leave reads
    // with such sets to the warp.
    uint32_t k = i + P.min_len, from = k;
    if constexpr (G < 32) {
      while (k > i && left(k - 1)) k--;
    } else {
      bool looked = false;
      while (k > i && left(k - 1)) {
        k--;
        if (ncur > (Fw.fmt == OCC_NARROW ? 64u : 256u) && !looked && k > i) {
          looked = true;
          const uint32_t at = seed_end(Sf.compat_mask, q, i, from);
          if (at < from) { from = k = at; reset(); }
        }
      }
    }
    if (ovf) { st |= ST_SET_OVF; return ~0u; }
    if (k > i) { i = k; continue; }
    uint32_t e = G < 32 ? i + P.min_len : from;
    while (e < n && right(e)) e++;
    if (ovf) { st |= ST_SET_OVF; return ~0u; }
    if (G == 32 && e < i + P.min_len) { i++; continue; }          // the window at i does not match
    if (nc >= cand_cap) { st |= ST_CAND_OVF; return ~0u; }
    uint64_t off = 0;
    if (lane == 0) off = thread_reserve(ivpool, ncur);
    off = __shfl_sync(gm, off, 0, G);
    if (off == ~0ull) { st |= ST_POOL_OVF; return ~0u; }
    BIv* dst = (BIv*)ivpool.base + off;
    for (uint32_t c = lane; c < ncur; c += G) dst[c] = cur[c];
    if (lane == 0) cands[nc] = Cand{i, e, 0u, ncur, off, i, 0u};
    nc++;
    if (e == n) break;
    reset();
    k = e + 1;
    while (k > i + 1 && left(k - 1)) k--;
    if (ovf) { st |= ST_SET_OVF; return ~0u; }
    i = k;
  }
  __syncwarp(gm);
  return nc;
}

// Persistent SMEM / MEM search with one read per group of G lanes (G = 32: the warp tier
// of reads whose sets outgrew the per-thread kernels; G = 4, 8, 16: the sub-warp
// candidates of the autotuner).  Group g of the grid owns two sets and a candidate list at
// g * 2 * set_cap / g * cand_cap.
template <bool COUNT_TOUCH, int G = 32>
__global__ void __launch_bounds__(128) k_mems_warp(DevFm Fw, DevFm Rv, const uint16_t* __restrict__ compat_fw,
                                                  const uint16_t* __restrict__ compat_rv, const uint8_t* __restrict__ q,
                                                  const uint64_t* __restrict__ qoff, MemsParams P, Pool ivpool,
                                                  Pool hitpool, MemsOut out, MemsWork W) {
  __shared__ SmemFm Sf, Sr;
  smem_fm_init(Sf, Fw, compat_fw);
  smem_fm_init(Sr, Rv, compat_rv);
  __syncthreads();
  const int lane = threadIdx.x & (G - 1);
  const uint32_t gm = grp_mask<G>();
  uint64_t grp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  BIv* base = W.sets + grp * 2 * W.set_cap;
  Cand* cands = W.cands + grp * W.cand_cap;
  uint64_t touches = 0;
  for (;;) {
    uint32_t k = 0;
    if (lane == 0) k = atomicAdd(W.queue, 1u);
    k = __shfl_sync(gm, k, 0, G);
    if (k >= W.count()) break;
    uint32_t i = W.ids[k];
    uint32_t st = ST_OK;
    uint64_t o = qoff[i];
    uint64_t t0 = touches;
    uint32_t nc = warp_mems_one<COUNT_TOUCH, G>(Fw, Rv, Sf, Sr, q + o, (uint32_t)(qoff[i + 1] - o), P, base,
                                                base + W.set_cap, W.set_cap, cands, W.cand_cap, ivpool, st, touches);
    __syncwarp(gm);
    if (COUNT_TOUCH && W.work_log) {
      uint32_t d = grp_sum<G>((uint32_t)(touches - t0));
      if (lane == 0) { W.work_log[4 * (size_t)i] += d; W.work_log[4 * (size_t)i + 3] |= 3u; }
    }
    if (lane == 0) {
      uint64_t hs = 0, hp = 0; uint32_t hc = 0;
      if (nc != ~0u) {
        if (!write_hits(cands, nc, P, ivpool, hitpool, hs, hc, hp)) st |= ST_POOL_OVF;
      }
      if (st) { hs = 0; hc = 0; hp = 0; }
      const uint64_t slot = W.slot_base ? W.slot_base[i] : (uint64_t)i;
      out.hit_start[slot] = hs; out.hit_count[slot] = hc; out.pos_count[slot] = hp; out.status[i] = st;
      if (W.slot_base)
        for (uint64_t x = slot + 1; x < W.slot_base[i + 1]; x++) { out.hit_count[x] = 0; out.pos_count[x] = 0; }
      if (st & (ST_SET_OVF | ST_CAND_OVF)) {
        if (W.rerun) atomicAdd(W.still_ovf, 1u);
        else out.ovf_list[atomicAdd(out.n_ovf, 1u)] = i;      // on to the warp tier
      }
    }
    __syncwarp(gm);
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

}  // namespace hfm
