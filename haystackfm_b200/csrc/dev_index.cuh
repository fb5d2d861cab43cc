// dev_index.cuh — device-resident FM-index layout and the rank / LF / extension
// primitives every kernel uses.
//
// Device layout (built once by hfm_index_load from the reference's bincode records):
//   occ   : one record per 64 BWT rows, two formats:
//             wide   (96 B, any text): 16 x u32 counts of every code before the record's row
//                    32, then the four planes of its rows' 4-bit codes, u32 each, of rows
//                    0..31 and of rows 32..63 (three 32-byte sectors).  A count at any row
//                    is the one at row 32 plus the rows between (or minus them, for rows
//                    0..31), so half the planes are loaded, masked and counted: the 16 counts
//                    of a border are 16 popcounts of 32 bits instead of 32 of them, and
//                    popcounts (16 lanes a cycle) bound the search on IUPAC texts;
//             narrow (32 B, texts of codes 0..4 only — ExactDna and ACGT-only IUPAC texts):
//                    4 x u16 counts of codes 1..4 from the start of the record's superblock
//                    (1,024 records = 65,536 rows) to the record's row 32, then for rows
//                    0..31 and for rows 32..63 three u32 planes: the two bits of code - 1,
//                    and the sentinels (one sector); the count of code 0 is the rows before
//                    the border minus the other four.
//   sb    : (narrow) 16 x u32 per superblock: count of every code before the superblock
//           (a few MB at 3.1 Gbp; it stays in L2).
//   ssa   : one 16-byte record per 64 rows: u64 "row is sampled" bits + u32 count of
//           sampled rows before the word (SampledSuffixArray, src/suffix_array/mod.rs:54-63).
//   sa_vals, seq_boundaries, lookup intervals: as in the reference.
// Narrow: rank(c, i) = count[(i-1)/64][c] + sb[(i-1)/65536][c] + popc(rows of code c <=
// (i-1)%64); both are identical to OccTable::rank (src/occ/mod.rs:330-363), whose records instead
// hold compacted lanes with a u32 superblock count and a u16 delta per lane
// (src/occ/mod.rs:144).  Wide records keep whole counts: on IUPAC texts an extension emits
// many intervals, and each would otherwise need one more dependent load for its superblock
// count (measured: 173 ms against 199 ms for the SMEM search of 1M reads).
#pragma once
#include <cstdint>

namespace hfm {

enum : uint32_t { OCC_WIDE = 0, OCC_NARROW = 1 };
constexpr uint32_t SB_BLOCK_SHIFT = 10;           // records per superblock: 1024 (65,536 rows)
constexpr uint32_t OCC_WIDE_U4 = 6;               // uint4 per wide record
constexpr uint32_t OCC_NARROW_U4 = 2;             // uint4 per narrow record

struct DevFm {
  const uint4* occ;          // OCC_WIDE_U4 or OCC_NARROW_U4 uint4 per record
  const uint32_t* sb;        // 16 x u32 per superblock (narrow records)
  const uint4* ssa;          // 1 x uint4 per block
  const uint32_t* sa_vals;
  const uint2* lut;          // nullptr when the index has no lookup table
  const uint32_t* seq_bounds;
  uint32_t text_len, num_seqs, sample_rate, lut_depth;
  uint32_t tag, lut_radix, num_blocks, fmt;
  uint32_t C[16];
  uint8_t s2l[16], l2s[16], lut_digit[16];
  uint16_t sym_mask;         // symbols present in the text
  uint16_t _pad2;
};

struct BIv { uint32_t flo, fhi, rlo, rhi; };

// Per-kernel shared copies of the small tables (divergent indexing from registers or
// the parameter bank would serialise).
struct SmemFm {
  uint32_t C[16];
  uint8_t s2l[16], l2s[16], dig[16];
  uint16_t compat_mask[16];   // compatible-symbol set of each query code as a bit mask
};

__device__ __forceinline__ void smem_fm_init(SmemFm& s, const DevFm& F, const uint16_t* compat_masks) {
  int t = threadIdx.x;
  if (t < 16) {
    s.C[t] = F.C[t]; s.s2l[t] = F.s2l[t]; s.l2s[t] = F.l2s[t]; s.dig[t] = F.lut_digit[t];
    s.compat_mask[t] = compat_masks[t];
  }
}

__device__ __forceinline__ uint64_t u2to64(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

__device__ __forceinline__ uint32_t sel4(uint4 x, uint32_t i) {
  return (i & 2) ? ((i & 1) ? x.w : x.z) : ((i & 1) ? x.y : x.x);
}

// One record with the rows of a border selected.  A border i (0 <= i <= text_len) is the
// position between BWT rows i-1 and i: the record of row i-1, rows 0..(i-1)%64 selected
// (border 0: record 0 with no row selected; its counts and superblock entry are 0).
template <uint32_t FMT> struct Border;

// A border x rows (0..64) into a record: the rows between it and row 32, and whether they
// are added to the counts there (1) or taken off (~0).
__device__ __forceinline__ uint32_t half_rows(uint32_t x) {
  const uint32_t k = x & 31;
  return x >= 64 ? ~0u : x >= 32 ? (1u << k) - 1u : ~0u << k;
}
__device__ __forceinline__ uint32_t half_sign(uint32_t x) { return x >= 32 ? 1u : ~0u; }

template <>
struct Border<OCC_WIDE> {
  uint4 a, b, c, d;        // counts before row 32
  uint4 w;                 // the four planes of the half that holds the border
  uint32_t m, sg;          // rows between row 32 and the border; 1 after row 32, ~0 before it

  // the rows of `w` counted for a border x rows (0..64) into the record
  __device__ __forceinline__ void select(uint32_t x) { m = half_rows(x); sg = half_sign(x); }
  // rows of code s among the selected ones (s a compile-time constant after unrolling)
  __device__ __forceinline__ uint32_t eq(int s) const {
    return m & ((s & 1) ? w.x : ~w.x) & ((s & 2) ? w.y : ~w.y) & ((s & 4) ? w.z : ~w.z) & ((s & 8) ? w.w : ~w.w);
  }
  __device__ __forceinline__ uint32_t delta(int s) const {
    const uint4 v = s < 4 ? a : s < 8 ? b : s < 12 ? c : d;
    return sel4(v, (uint32_t)s & 3);
  }
  // rank of code s at the border
  __device__ __forceinline__ uint32_t local(int s) const { return delta(s) + (uint32_t)__popc(eq(s)) * sg; }
};

template <>
struct Border<OCC_NARROW> {
  uint32_t c12, c34;       // counts before row 32, from the superblock start
  uint32_t b0, b1, z;      // the planes of the half that holds the border
  uint32_t m, sg;          // rows between row 32 and the border; 1 after row 32, ~0 before it
  uint32_t sbi, i;         // superblock, the border itself

  __device__ __forceinline__ void take(const uint4& u, const uint4& v, uint32_t x) {
    c12 = u.x; c34 = u.y;
    const bool up = x >= 32;
    b0 = up ? v.y : u.z; b1 = up ? v.z : u.w; z = up ? v.w : v.x;
    m = half_rows(x); sg = half_sign(x);
  }
  __device__ __forceinline__ uint32_t eq(int s) const {      // s in 1..4
    return m & ~z & (((s - 1) & 1) ? b0 : ~b0) & (((s - 1) & 2) ? b1 : ~b1);
  }
  __device__ __forceinline__ uint32_t delta(int s) const {
    const uint32_t w = s <= 2 ? c12 : c34;
    return ((s - 1) & 1) ? (w >> 16) : (w & 0xFFFFu);
  }
  // rank of code s within the superblock
  __device__ __forceinline__ uint32_t local(int s) const { return delta(s) + (uint32_t)__popc(eq(s)) * sg; }
};

template <uint32_t FMT, class FM>
__device__ __forceinline__ Border<FMT> load_border(const FM& F, uint32_t i) {
  Border<FMT> r;
  const uint32_t pos = i ? i - 1 : 0u, blk = pos >> 6;
  if constexpr (FMT == OCC_WIDE) {
    const uint4* p = F.occ + (size_t)blk * OCC_WIDE_U4;
    const uint32_t x = i ? (pos & 63) + 1u : 0u;
    r.a = __ldg(p); r.b = __ldg(p + 1); r.c = __ldg(p + 2); r.d = __ldg(p + 3);
    r.w = __ldg(p + (x >= 32 ? 5 : 4));
    r.select(x);
  } else {
    r.sbi = blk >> SB_BLOCK_SHIFT;
    r.i = i;
    const uint4* p = F.occ + (size_t)blk * OCC_NARROW_U4;
    r.take(__ldg(p), __ldg(p + 1), i ? (pos & 63) + 1u : 0u);
  }
  return r;
}

// The selected rows of a wide border split by code: m[s] for s = 0..15.
__device__ __forceinline__ void wide_masks(const uint4& w, uint32_t sel, uint32_t m[16]) {
  uint32_t q[4];
#pragma unroll
  for (int k = 0; k < 4; k++) q[k] = sel & ((k & 1) ? w.x : ~w.x) & ((k & 2) ? w.y : ~w.y);
#pragma unroll
  for (int s = 0; s < 16; s++) m[s] = q[s & 3] & ((s & 4) ? w.z : ~w.z) & ((s & 8) ? w.w : ~w.w);
}

// Ranks of all 16 codes at a wide border.
__device__ __forceinline__ void wide_ranks(const Border<OCC_WIDE>& B, uint32_t r[16]) {
  uint32_t m[16];
  wide_masks(B.w, B.m, m);
#pragma unroll
  for (int s = 0; s < 16; s++) r[s] = B.delta(s) + (uint32_t)__popc(m[s]) * B.sg;
}

template <class FM>
__device__ __forceinline__ uint32_t sb_count(const FM& F, uint32_t sbi, uint32_t s) {
  return __ldg(F.sb + (size_t)sbi * 16 + s);
}

// Absolute rank of code s at a border of an ACGT text (occ(s, i)).
template <class FM>
__device__ __forceinline__ uint32_t border_rank(const FM& F, const Border<OCC_NARROW>& B, int s) {
  if (s == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int c = 1; c <= 4; c++) t += sb_count(F, B.sbi, c) + B.local(c);
    return B.i - t;
  }
  return sb_count(F, B.sbi, s) + B.local(s);
}

// The interval [lo, hi) of the BWT split by symbol: calls f(s, d, r, sbi) for every code s
// in ascending order (0..4 narrow, 0..15 wide), d = occ(s, hi) - occ(s, lo), and the lo
// border's count r: occ(s, lo) = r (wide) or sb_count(F, sbi, s) + r (narrow; one
// L2-resident load, made only for the codes the caller keeps).  `last` = the highest code
// the caller needs.
template <uint32_t FMT, class FM, class Fn>
__device__ __forceinline__ void split_by_symbol(const FM& F, uint32_t lo, uint32_t hi, uint32_t last, Fn&& f) {
  if constexpr (FMT == OCC_NARROW) {
    const Border<FMT> L = load_border<FMT>(F, lo), H = load_border<FMT>(F, hi);
    const bool same_sb = L.sbi == H.sbi;
    uint32_t d[5], r[5];
    uint32_t sum = 0, rsum = 0;
#pragma unroll
    for (int s = 1; s <= 4; s++) {
      const uint32_t a = L.local(s);
      uint32_t v = H.local(s) - a;
      if (!same_sb) v += sb_count(F, H.sbi, s) - sb_count(F, L.sbi, s);
      d[s] = v; sum += v; r[s] = a; rsum += a;
    }
    d[0] = (hi - lo) - sum;
    r[0] = (lo - (L.sbi << (SB_BLOCK_SHIFT + 6))) - rsum;   // rows of the superblock before lo, minus codes 1..4
#pragma unroll
    for (int s = 0; s <= 4; s++) f(s, d[s], r[s], L.sbi);
  } else {
    const Border<FMT> L = load_border<FMT>(F, lo), H = load_border<FMT>(F, hi);
    uint32_t rl[16], rh[16];
    wide_ranks(L, rl);
    wide_ranks(H, rh);
#pragma unroll
    for (int t = 0; t < 16; t++) {
      if ((uint32_t)t > last) break;
      f(t, rh[t] - rl[t], rl[t], 0u);
    }
  }
}

// The code of BWT row `row` and its rank at that row (LF step of a one-row interval,
// lane_and_mask_bitplane + rank_at_lane, src/occ/mod.rs:434-480).
template <uint32_t FMT, class FM>
__device__ __forceinline__ void row_code_rank(const FM& F, uint32_t row, uint32_t& code, uint32_t& rank) {
  const uint32_t off = row & 63;
  if constexpr (FMT == OCC_WIDE) {
    // the half of `row` and its one count: 20 of the record's 96 bytes
    const uint4* p = F.occ + (size_t)(row >> 6) * OCC_WIDE_U4;
    Border<FMT> B;
    B.w = __ldg(p + (off >= 32 ? 5 : 4));
    B.select(off);
    const uint32_t k = off & 31;
    const uint32_t c = ((B.w.x >> k) & 1) | ((B.w.y >> k) & 1) << 1 | ((B.w.z >> k) & 1) << 2 | ((B.w.w >> k) & 1) << 3;
    const uint32_t m = B.m & ((c & 1) ? B.w.x : ~B.w.x) & ((c & 2) ? B.w.y : ~B.w.y) & ((c & 4) ? B.w.z : ~B.w.z) &
                       ((c & 8) ? B.w.w : ~B.w.w);
    code = c;
    rank = __ldg(reinterpret_cast<const uint32_t*>(p) + c) + (uint32_t)__popc(m) * B.sg;
  } else {
    const uint4* p = F.occ + (size_t)(row >> 6) * OCC_NARROW_U4;
    Border<FMT> B;
    B.take(__ldg(p), __ldg(p + 1), off);               // rows before `row` only
    B.sbi = row >> (6 + SB_BLOCK_SHIFT);
    B.i = row;
    const uint32_t k = off & 31;
    const uint32_t c = ((B.z >> k) & 1) ? 0u : 1u + (((B.b0 >> k) & 1) | ((B.b1 >> k) & 1) << 1);
    code = c;
    if (c == 0) {
      rank = border_rank(F, B, 0);
    } else {
      const uint32_t m = B.m & ~B.z & (((c - 1) & 1) ? B.b0 : ~B.b0) & (((c - 1) & 2) ? B.b1 : ~B.b1);
      const uint32_t w = c <= 2 ? B.c12 : B.c34;
      rank = sb_count(F, B.sbi, c) + (((c - 1) & 1) ? (w >> 16) : (w & 0xFFFFu)) + (uint32_t)__popc(m) * B.sg;
    }
  }
}

// Rank of every symbol code at border i (counts of code s in bwt[0..i)), absent codes 0.
// Used by the backward search and the warp-per-read kernels.
template <uint32_t FMT>
__device__ __forceinline__ void sym_ranks_t(const DevFm& F, uint32_t i, uint32_t r[16]) {
  const Border<FMT> B = load_border<FMT>(F, i);
  if constexpr (FMT == OCC_NARROW) {
    uint32_t t = 0;
#pragma unroll
    for (int s = 1; s <= 4; s++) { r[s] = sb_count(F, B.sbi, s) + B.local(s); t += r[s]; }
    r[0] = i - t;
#pragma unroll
    for (int s = 5; s < 16; s++) r[s] = 0;
  } else {
    wide_ranks(B, r);
  }
}

__device__ __forceinline__ void sym_ranks(const DevFm& F, const SmemFm& S, uint32_t i, uint32_t r[16]) {
  (void)S;
  if (F.fmt == OCC_NARROW) sym_ranks_t<OCC_NARROW>(F, i, r);
  else sym_ranks_t<OCC_WIDE>(F, i, r);
}

// One LF step with the sampled-SA test (FmIndex::resolve_sa loop body,
// src/fm_index/query.rs:282-291; lf_step src/occ/mod.rs:456-480).  Returns true with
// *val = SA value when row `pos` is sampled; otherwise advances pos = LF(pos).
template <uint32_t FMT>
__device__ __forceinline__ bool lf_or_sample_t(const DevFm& F, const SmemFm& S, uint32_t& pos, uint32_t& val) {
  const uint32_t blk = pos >> 6, off = pos & 63;
  uint4 w = __ldg(F.ssa + blk);
  uint32_t code, rank;
  row_code_rank<FMT>(F, pos, code, rank);            // issued before the sampled test: overlaps its latency
  uint64_t word = u2to64(w.x, w.y);
  if ((word >> off) & 1ull) {
    val = __ldg(F.sa_vals + w.z + (uint32_t)__popcll(word & ((1ull << off) - 1ull)));
    return true;
  }
  pos = S.C[code] + rank;
  return false;
}

__device__ __forceinline__ bool lf_or_sample(const DevFm& F, const SmemFm& S, uint32_t& pos, uint32_t& val) {
  if (F.fmt == OCC_NARROW) return lf_or_sample_t<OCC_NARROW>(F, S, pos, val);
  return lf_or_sample_t<OCC_WIDE>(F, S, pos, val);
}

// partition_point(bounds, b <= p): first index with bounds[idx] > p.
__device__ __forceinline__ uint32_t upper_bound_u32(const uint32_t* b, uint32_t n, uint32_t p) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) { uint32_t mid = (lo + hi) >> 1; if (b[mid] <= p) lo = mid + 1; else hi = mid; }
  return lo;
}

// Records from their form in the device-layout blob (counts before row 0, planes of the
// codes' bits as u64) to their form on the device.
__global__ void k_device_records(uint4* __restrict__ occ, uint32_t nblk, uint32_t fmt) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nblk) return;
  if (fmt == OCC_WIDE) {
    uint4* p = occ + (size_t)b * OCC_WIDE_U4;
    Border<OCC_WIDE> B;
    B.a = p[0]; B.b = p[1]; B.c = p[2]; B.d = p[3];
    const uint4 e = p[4], f = p[5];
    B.w = make_uint4(e.x, e.z, f.x, f.z);
    B.m = ~0u; B.sg = 1u;
    uint32_t r[16];
    wide_ranks(B, r);
#pragma unroll
    for (int k = 0; k < 4; k++) p[k] = make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
    p[4] = B.w;
    p[5] = make_uint4(e.y, e.w, f.y, f.w);
  } else {
    uint4* p = occ + (size_t)b * OCC_NARROW_U4;
    const uint4 u = p[0], v = p[1];       // counts; planes 0, 1, 2 as u64
    auto half = [](uint32_t p0, uint32_t p1, uint32_t p2, uint32_t& b0, uint32_t& b1, uint32_t& z) {
      z = ~(p0 | p1 | p2);                // code 1..4 = 001 010 011 100 -> code - 1 = 00 01 10 11
      b0 = (p1 & ~p0) | p2;
      b1 = (p1 & p0) | p2;
    };
    uint4 x = u, y = v;
    half(u.z, v.x, v.z, x.z, x.w, y.x);
    half(u.w, v.y, v.w, y.y, y.z, y.w);
    const uint32_t n1 = __popc(~x.z & ~x.w & ~y.x), n2 = __popc(x.z & ~x.w), n3 = __popc(~x.z & x.w), n4 = __popc(x.z & x.w);
    x.x = u.x + (n1 | n2 << 16);
    x.y = u.y + (n3 | n4 << 16);
    p[0] = x; p[1] = y;
  }
}

}  // namespace hfm
