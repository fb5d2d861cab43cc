// resolve.cuh — SA-position resolve fused with the reference boundary map, plus the scan /
// gather kernels that lay results out per read.
//
// A position is the row's entry of the whole suffix array when the handle has it: the index
// carries every sample_rate-th position (src/suffix_array/mod.rs:54-63), which saves memory
// that a B200 has, and k_sa_rows walks the others out once when it is loaded (4 bytes a row).
// Rows of one interval are neighbours, so the reads coalesce, where a walk of 16 dependent
// steps on average touched two sectors a step.  Without the array (no memory for it, or a
// sample rate above SA_ROWS_RATE) the rows are walked as before.  Measured on a B200, 256 Mbp
// ACGT, k_resolve: 3.4 M rows of 1M reads 1.20 -> 0.08 ms, 4,500 rows 47 -> 10 us.
//
// One thread per output position.  Positions are grouped in segments (one per SA
// interval, rows lo .. lo+n); a block finds its segments once and every thread locates
// its own segment in shared memory.  Replaces locate_resolve.wgsl:98-176,
// mem_resolve.wgsl:101-136 and ref_map.wgsl:32-59 of the reference, with the CPU
// resolve_sa / map_position semantics (src/fm_index/query.rs:282-357).
#pragma once
#include "dev_index.cuh"

namespace hfm {

struct ResolveArgs {
  const uint32_t* seg_row;      // row of the segment's first position
  uint32_t row_stride;          // in u32 units
  const uint64_t* seg_off;      // nseg + 1 ascending position offsets
  uint32_t nseg;
  uint64_t total;
  const uint32_t* bounds;       // map position -> (index, offset): partition_point(bounds <= p)
  uint32_t nb;
  uint32_t guard;               // max LF steps before the walk is declared broken
  uint32_t* out;                // 2 * total u32
  uint32_t* walk_err;
  unsigned long long* steps;    // LF steps (nullptr: not counted)
  const uint32_t* block_first;  // segment containing the first position of each block
  const uint64_t* total_dev;    // when set (graph-captured chains), the position count is read here
  const uint32_t* sa;           // position of every row (SA_UNKNOWN: walk), or nullptr
};

constexpr uint32_t SA_UNKNOWN = 0xFFFFFFFFu;
constexpr uint32_t SA_ROWS_RATE = 1024;     // longest walks that k_sa_rows is run for

// The suffix array from its samples: every sampled row knows its position, the rows reached
// from it by LF steps are those of the positions before it, down to the next sampled one.
// The rows of the sentinels (the first num_seqs rows) cover the ends of the sequences; their
// positions come from a walk first.  sa is filled with SA_UNKNOWN by the caller.  A chain counts
// only when the sampled row at its end has the position that it leads to: every entry is what a
// walk from that row gives, and rows whose samples disagree (or that no chain reaches) stay
// unknown and are walked, with the walk's answer or error.  A layout blob is not checked beyond
// its sizes: marks past the text and places outside the n_vals sampled values count for nothing.
template <uint32_t FMT>
__global__ void __launch_bounds__(128) k_sa_rows(DevFm F, uint64_t n_vals, uint32_t* __restrict__ sa) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto step = [&](uint32_t& row) -> bool {
    uint32_t c, rk;
    row_code_rank<FMT>(F, row, c, rk);
    if (!c) return false;                     // a sequence starts here
    row = F.C[c] + rk;
    return row < F.text_len;
  };
  auto sampled = [&](uint32_t row, uint32_t& val) -> bool {
    const uint4 w = __ldg(F.ssa + (row >> 6));
    const uint64_t word = u2to64(w.x, w.y);
    if (!((word >> (row & 63)) & 1)) return false;
    const uint64_t at = (uint64_t)w.z + (uint32_t)__popcll(word & ((1ull << (row & 63)) - 1ull));
    if (at >= n_vals) return false;
    val = __ldg(F.sa_vals + at);
    return true;
  };
  auto fill = [&](uint32_t first, uint32_t v) {
    sa[first] = v;
    uint32_t row = first, k = 0, x;
    bool met = false;
    for (; k < F.sample_rate && v > 0 && step(row); k++) {
      v--;
      if (sampled(row, x)) { met = x == v; break; }
      sa[row] = v;
    }
    if (met || !k) return;
    for (row = first; k && step(row); k--) sa[row] = SA_UNKNOWN;
  };
  if (t < F.num_blocks) {
    const uint4 w = __ldg(F.ssa + t);
    uint64_t at = w.z;
    for (uint64_t m = u2to64(w.x, w.y); m; m &= m - 1, at++) {
      const uint64_t row = t * 64 + (uint32_t)__ffsll((long long)m) - 1u;
      if (row < F.text_len && at < n_vals) fill((uint32_t)row, __ldg(F.sa_vals + at));
    }
  } else if (t - F.num_blocks < F.num_seqs) {
    const uint32_t first = (uint32_t)(t - F.num_blocks);
    uint32_t row = first, steps = 0, v = 0;
    bool found = sampled(row, v);
    while (!found && steps < F.sample_rate && step(row)) { steps++; found = sampled(row, v); }
    if (found && steps) fill(first, v + steps);
  }
}

// block_first[b] = segment holding position b * blk (positions are CSR over segments).
// Blocks at or past max_blocks (the map's size) are skipped: a chain with fixed capacities
// runs this before it knows whether the positions fit.
__global__ void k_block_first(const uint64_t* __restrict__ seg_off, uint32_t nseg, uint32_t blk,
                              uint32_t* __restrict__ block_first, uint64_t max_blocks = ~0ull) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  uint64_t a = seg_off[s], e = seg_off[s + 1];
  if (a == e) return;
  const uint64_t last = min((e - 1) / blk, max_blocks - 1);
  for (uint64_t b = (a + blk - 1) / blk; b <= last; b++) block_first[b] = s;
}

// Segments [first, first + cnt) cover positions [b * blk, (b + 1) * blk) of block b.
__device__ __forceinline__ void block_segments(const uint32_t* block_first, uint64_t nblocks, uint32_t nseg,
                                               uint32_t& first, uint32_t& cnt) {
  uint64_t b = blockIdx.x;
  first = block_first[b];
  uint32_t last = b + 1 < nblocks ? block_first[b + 1] : nseg - 1;
  cnt = last - first + 1;
}

constexpr int RES_T = 256;
constexpr int RES_BOUNDS_SMEM = 2048;

template <bool COUNT>
__global__ void __launch_bounds__(RES_T) k_resolve(DevFm F, ResolveArgs A) {
  __shared__ SmemFm S;
  __shared__ uint64_t s_off[RES_T + 1];
  __shared__ uint32_t s_row[RES_T];
  __shared__ uint32_t s_b[RES_BOUNDS_SMEM];
  __shared__ uint32_t s_first, s_cnt;
  if (threadIdx.x < 16) { S.C[threadIdx.x] = F.C[threadIdx.x]; }
  const uint64_t total = A.total_dev ? *A.total_dev : A.total;
  uint64_t p0 = (uint64_t)blockIdx.x * RES_T;
  if (p0 >= total) return;                 // a grid sized for a capacity: blocks past the positions
  uint64_t p1 = min(p0 + RES_T, total);
  if (threadIdx.x == 0) {
    uint32_t f, c;
    block_segments(A.block_first, (total + RES_T - 1) / RES_T, A.nseg, f, c);
    s_first = f; s_cnt = c;
  }
  bool smem_b = A.nb <= RES_BOUNDS_SMEM;
  if (smem_b) for (uint32_t k = threadIdx.x; k < A.nb; k += RES_T) s_b[k] = A.bounds[k];
  __syncthreads();
  uint32_t first = s_first, cnt = s_cnt;
  bool local = cnt <= RES_T;
  if (local) {
    for (uint32_t k = threadIdx.x; k <= cnt; k += RES_T) s_off[k] = A.seg_off[first + k];
    for (uint32_t k = threadIdx.x; k < cnt; k += RES_T) s_row[k] = A.seg_row[(size_t)(first + k) * A.row_stride];
  }
  __syncthreads();
  uint64_t p = p0 + threadIdx.x;
  if (p >= p1) return;
  uint32_t seg, row;
  if (local) {
    uint32_t lo = 0, hi = cnt - 1;
    while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (s_off[mid] <= p) lo = mid; else hi = mid - 1; }
    seg = lo; row = s_row[lo] + (uint32_t)(p - s_off[lo]);
  } else {
    uint32_t lo = first, hi = first + cnt - 1;
    while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (A.seg_off[mid] <= p) lo = mid; else hi = mid - 1; }
    seg = lo; row = A.seg_row[(size_t)lo * A.row_stride] + (uint32_t)(p - A.seg_off[lo]);
  }
  (void)seg;
  uint32_t pos = row, steps = 0, val = A.sa ? __ldg(A.sa + row) : SA_UNKNOWN, text;
  bool ok = true;
  const bool walk = val == SA_UNKNOWN;
  // LF walk (resolve_sa, src/fm_index/query.rs:282-291)
  while (walk) {
    if (lf_or_sample(F, S, pos, val)) break;
    if (++steps > A.guard) { ok = false; break; }
  }
  uint32_t r0, r1;
  if (ok) {
    text = val + steps;
    uint32_t idx = smem_b ? upper_bound_u32(s_b, A.nb, text) : upper_bound_u32(A.bounds, A.nb, text);
    uint32_t start = idx == 0 ? 0 : (smem_b ? s_b[idx - 1] : A.bounds[idx - 1]);
    r0 = idx; r1 = text - start;
  } else {
    atomicAdd(A.walk_err, 1u);
    r0 = 0xFFFFFFFFu; r1 = 0xFFFFFFFFu;
  }
  reinterpret_cast<uint2*>(A.out)[p] = make_uint2(r0, r1);
  if (COUNT && walk) atomicAdd(A.steps, (unsigned long long)(steps + 1));
}

// ---- resolve deduplication ----------------------------------------------------------
// Segments with the same (first row, length) resolve to the same positions: across a
// batch, hits on repeated strings (N runs, repeat copies) share their SA interval.  The
// segments are hashed, each distinct one is resolved once, and every hit copies its
// positions from it.  Output is identical to resolving every row.

constexpr unsigned long long HASH_EMPTY = ~0ull;

__device__ __forceinline__ uint64_t mix64(uint64_t k) {      // splitmix64 finaliser
  k ^= k >> 30; k *= 0xbf58476d1ce4e5b9ull; k ^= k >> 27; k *= 0x94d049bb133111ebull; k ^= k >> 31;
  return k;
}

__global__ void k_dedup_insert(const uint32_t* __restrict__ seg_row, uint32_t stride, const uint64_t* __restrict__ seg_off,
                               uint32_t nseg, unsigned long long* __restrict__ keys, uint64_t mask,
                               uint32_t* __restrict__ seg_slot) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  uint64_t n = seg_off[s + 1] - seg_off[s];
  if (n == 0) { seg_slot[s] = 0xFFFFFFFFu; return; }
  unsigned long long key = ((unsigned long long)seg_row[(size_t)s * stride] << 32) | (uint32_t)n;
  uint64_t h = mix64(key) & mask;
  // the table has at least twice as many slots as segments: an empty slot is always found
  for (uint64_t probe = 0; probe <= mask; probe++) {
    unsigned long long prev = atomicCAS(keys + h, HASH_EMPTY, key);
    if (prev == HASH_EMPTY || prev == key) { seg_slot[s] = (uint32_t)h; return; }
    h = (h + 1) & mask;
  }
  seg_slot[s] = 0xFFFFFFFFu;    // unreachable with a half-empty table
}

__global__ void k_dedup_flags(const unsigned long long* __restrict__ keys, uint64_t size, uint32_t* __restrict__ flags) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < size) flags[i] = keys[i] != HASH_EMPTY;
}

__global__ void k_dedup_compact(const unsigned long long* __restrict__ keys, uint64_t size,
                                const uint64_t* __restrict__ uid, uint32_t* __restrict__ urow,
                                uint32_t* __restrict__ ulen) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= size) return;
  unsigned long long k = keys[i];
  if (k == HASH_EMPTY) return;
  uint64_t u = uid[i];
  urow[u] = (uint32_t)(k >> 32); ulen[u] = (uint32_t)k;
}

// out[p] = resolved position of its segment's distinct copy.  A block copies EXP_BLK
// consecutive positions; its segments are staged in shared memory once.  Where they are EXP_LONG
// positions long on average a warp copies a segment at a time (no search for a position's
// segment), else a thread EXP_PER positions, strided for coalescing.  (592 M positions in
// segments of 86: 1.86 ms by position in blocks of 2,048, 1.71 by segment, 1.09 in
// blocks of 8,192, whose staging is three dependent loads; writing them takes 0.64.)
constexpr uint32_t EXP_LONG = 24;
constexpr int EXP_T = 256, EXP_PER = 32, EXP_BLK = EXP_T * EXP_PER, EXP_SEGS = 2048;   // segments staged
__global__ void __launch_bounds__(EXP_T) k_dedup_expand(const uint64_t* __restrict__ seg_off, uint32_t nseg, uint64_t total,
                                                        const uint32_t* __restrict__ seg_slot,
                                                        const uint64_t* __restrict__ uid,
                                                        const uint64_t* __restrict__ uoff,
                                                        const uint2* __restrict__ uout, uint2* __restrict__ out,
                                                        const uint32_t* __restrict__ block_first,
                                                        const uint64_t* __restrict__ total_dev = nullptr) {
  __shared__ uint64_t s_off[EXP_SEGS + 1];
  __shared__ uint64_t s_src[EXP_SEGS];
  __shared__ uint32_t s_first, s_cnt;
  if (total_dev) total = *total_dev;
  uint64_t p0 = (uint64_t)blockIdx.x * EXP_BLK;
  if (p0 >= total) return;                 // a grid sized for a capacity: blocks past the positions
  uint64_t p1 = min(p0 + EXP_BLK, total);
  if (threadIdx.x == 0) {
    uint32_t f, c;
    block_segments(block_first, (total + EXP_BLK - 1) / EXP_BLK, nseg, f, c);
    s_first = f; s_cnt = c;
  }
  __syncthreads();
  uint32_t first = s_first, cnt = s_cnt;
  bool local = cnt <= EXP_SEGS;
  if (local) {
    for (uint32_t k = threadIdx.x; k <= cnt; k += EXP_T) s_off[k] = seg_off[first + k];
    for (uint32_t k = threadIdx.x; k < cnt; k += EXP_T) {
      uint32_t slot = seg_slot[first + k];
      s_src[k] = slot == 0xFFFFFFFFu ? 0 : uoff[uid[slot]];
    }
  }
  __syncthreads();
  if (local && (uint64_t)cnt * EXP_LONG <= p1 - p0) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t k = threadIdx.x >> 5; k < cnt; k += EXP_T / 32) {
      const uint64_t a = max(s_off[k], p0), e = min(s_off[k + 1], p1);
      const uint2* src = uout + (s_src[k] - s_off[k]);       // of position 0, were it in this segment
      for (uint64_t p = a + lane; p < e; p += 32) out[p] = src[p];
    }
    return;
  }
  uint32_t lo = 0;                       // positions ascend per thread: resume the search
  for (int k = 0; k < EXP_PER; k++) {
    uint64_t p = p0 + threadIdx.x + (uint64_t)k * EXP_T;
    if (p >= p1) return;
    uint64_t src;
    if (local) {
      // still in the previous position's segment (the usual case for segments of more than
      // EXP_T positions), else a binary search over the rest
      if (lo + 1 < cnt && s_off[lo + 1] <= p) {
        uint32_t hi = cnt - 1;
        lo++;
        while (lo < hi) { uint32_t mid = (lo + hi + 1) >> 1; if (s_off[mid] <= p) lo = mid; else hi = mid - 1; }
      }
      src = s_src[lo] + (p - s_off[lo]);
    } else {
      uint32_t l = first, hi = first + cnt - 1;
      while (l < hi) { uint32_t mid = (l + hi + 1) >> 1; if (seg_off[mid] <= p) l = mid; else hi = mid - 1; }
      src = uoff[uid[seg_slot[l]]] + (p - seg_off[l]);
    }
    out[p] = uout[src];
  }
}

// ---- exclusive scan (u32 or u64 input) -> u64 output with out[n] = total ----------
constexpr int SCAN_T = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_T * SCAN_ITEMS;

template <class T>
__global__ void __launch_bounds__(SCAN_T) k_scan_tiles(const T* __restrict__ in, uint32_t in_stride, uint64_t n,
                                                      uint64_t* __restrict__ out, uint64_t* __restrict__ tile_sums) {
  __shared__ uint64_t s[SCAN_T];
  uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
  uint64_t v[SCAN_ITEMS], sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    uint64_t i = base + k;
    v[k] = i < n ? (uint64_t)in[i * in_stride] : 0;
    sum += v[k];
  }
  s[threadIdx.x] = sum;
  __syncthreads();
  for (int d = 1; d < SCAN_T; d <<= 1) {
    uint64_t t = threadIdx.x >= d ? s[threadIdx.x - d] : 0;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  uint64_t run = s[threadIdx.x] - sum;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    uint64_t i = base + k;
    if (i < n) out[i] = run;
    run += v[k];
  }
  if (threadIdx.x == SCAN_T - 1) tile_sums[blockIdx.x] = s[SCAN_T - 1];
}

// Scans tile sums in place (single block, sequential chunks).
__global__ void __launch_bounds__(1024) k_scan_sums(uint64_t* sums, uint32_t ntiles) {
  __shared__ uint64_t s[1024];
  __shared__ uint64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < ntiles; base += 1024) {
    uint32_t i = base + threadIdx.x;
    uint64_t v = i < ntiles ? sums[i] : 0;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
      uint64_t t = threadIdx.x >= d ? s[threadIdx.x - d] : 0;
      __syncthreads();
      s[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < ntiles) sums[i] = carry + s[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += s[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[ntiles] = carry;
}

__global__ void k_scan_add(uint64_t* out, uint64_t n, const uint64_t* __restrict__ sums, uint32_t ntiles) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += sums[i / SCAN_TILE];
  if (i == 0) out[n] = sums[ntiles];
}

// ---- exclusive scans of two arrays at once (u32 and u64), out[n] = totals ------------
// The tiles' own sums first; then every block adds the sums of the tiles before its own, which
// it sums itself (a launch and a round through one block less than a scan of the sums: the
// scan of a batch of up to SCAN_TILE is one launch).
struct ScanPair { unsigned long long a, b; };

__device__ __forceinline__ ScanPair block_scan_pair(ScanPair v, ScanPair* s_warp, ScanPair& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ScanPair x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long ya = __shfl_up_sync(0xFFFFFFFFu, x.a, d), yb = __shfl_up_sync(0xFFFFFFFFu, x.b, d);
    if (lane >= d) { x.a += ya; x.b += yb; }
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  ScanPair before{0, 0};
  total = ScanPair{0, 0};
#pragma unroll
  for (int w = 0; w < SCAN_T / 32; w++) {
    const ScanPair t = s_warp[w];
    if (w < warp) { before.a += t.a; before.b += t.b; }
    total.a += t.a; total.b += t.b;
  }
  __syncthreads();
  return ScanPair{x.a - v.a + before.a, x.b - v.b + before.b};
}

__global__ void __launch_bounds__(SCAN_T) k_scan_pair_tiles(const uint32_t* __restrict__ in_a, const uint64_t* __restrict__ in_b,
                                                           uint64_t n, uint64_t* __restrict__ out_a, uint64_t* __restrict__ out_b,
                                                           ScanPair* __restrict__ sums, ScanPair* __restrict__ totals) {
  __shared__ ScanPair s_warp[SCAN_T / 32];
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
  unsigned long long va[SCAN_ITEMS], vb[SCAN_ITEMS];
  ScanPair sum{0, 0}, total;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const uint64_t i = base + k;
    va[k] = i < n ? in_a[i] : 0; vb[k] = i < n ? in_b[i] : 0;
    sum.a += va[k]; sum.b += vb[k];
  }
  ScanPair run = block_scan_pair(sum, s_warp, total);
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const uint64_t i = base + k;
    if (i < n) { out_a[i] = run.a; out_b[i] = run.b; }
    run.a += va[k]; run.b += vb[k];
  }
  if (threadIdx.x == 0) {
    sums[blockIdx.x] = total;
    if (gridDim.x == 1) { out_a[n] = total.a; out_b[n] = total.b; *totals = total; }
  }
}

__global__ void __launch_bounds__(SCAN_T) k_scan_pair_add(uint64_t n, uint64_t* __restrict__ out_a, uint64_t* __restrict__ out_b,
                                                         const ScanPair* __restrict__ sums, ScanPair* __restrict__ totals) {
  __shared__ ScanPair s_warp[SCAN_T / 32];
  ScanPair mine{0, 0}, before;
  for (uint32_t t = threadIdx.x; t < blockIdx.x; t += SCAN_T) { mine.a += sums[t].a; mine.b += sums[t].b; }
  block_scan_pair(mine, s_warp, before);
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
  for (uint64_t i = base + threadIdx.x; i < min(n, base + SCAN_TILE); i += SCAN_T) { out_a[i] += before.a; out_b[i] += before.b; }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    const ScanPair last = sums[blockIdx.x], total{before.a + last.a, before.b + last.b};
    out_a[n] = total.a; out_b[n] = total.b;
    *totals = total;
  }
}

// ---- gathers ------------------------------------------------------------------
// Locate: query intervals (pool) -> resolve segments in query order.  With blk, also the end of
// the last segment and the first segment of each block of blk positions (k_block_first): a small
// batch is a chain of launches, and this saves two of them.  (Host call of one 24-mer on a B200:
// 124 us, 114 with this and the result's copies queued before the call's last wait; of 10,000
// 32-mers: 202 -> 188.)
__global__ void k_gather_locate(const uint2* __restrict__ ivpool, const uint64_t* __restrict__ ivoff,
                                const uint32_t* __restrict__ niv, const uint64_t* __restrict__ seg_base,
                                const uint64_t* __restrict__ pos_base, uint32_t nq, uint32_t cap,
                                uint32_t* __restrict__ seg_row, uint64_t* __restrict__ seg_off,
                                uint32_t blk = 0, uint32_t* __restrict__ block_first = nullptr) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  uint64_t sb = seg_base[i], run = pos_base[i];
  const uint2* iv = ivpool + ivoff[i];
  const uint32_t n = niv[i];
  for (uint32_t k = 0; k < n; k++) {
    uint2 v = iv[k];
    uint32_t sz = v.y - v.x;
    seg_row[sb + k] = v.x; seg_off[sb + k] = run;
    const uint64_t end = run + ((cap && sz > cap) ? cap : sz);
    if (blk)
      for (uint64_t b = (run + blk - 1) / blk; b * blk < end; b++) block_first[b] = (uint32_t)(sb + k);
    run = end;
  }
  if (blk && i == nq - 1) seg_off[sb + n] = run;
}

// Mems: hits of every slot (pool) -> CSR hit array, with the offsets of their positions, also
// as the resolve's segment offsets.  A group of GATHER_LANES lanes takes a slot: its hits are
// neighbours in the pool and in the array, so the group's loads and stores coalesce (6.9 M hits
// of 200,000 reads: 367 us with a thread a slot, 93 with a group).
constexpr int GATHER_LANES = 8;
__global__ void __launch_bounds__(256) k_gather_hits(const uint4* __restrict__ hitpool, const uint64_t* __restrict__ hit_start,
                              const uint32_t* __restrict__ hit_count, const uint64_t* __restrict__ hit_base,
                              const uint64_t* __restrict__ pos_base, uint64_t n_slots, uint4* __restrict__ hits,
                              uint64_t* __restrict__ seg_off, uint64_t hit_cap = ~0ull) {
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / GATHER_LANES;
  const uint32_t lane = threadIdx.x & (GATHER_LANES - 1);
  const uint32_t mask = ((1u << GATHER_LANES) - 1u) << (threadIdx.x & 31 & ~(GATHER_LANES - 1));
  if (i >= n_slots) return;                            // a whole group at a time
  const uint32_t n = hit_count[i];
  if (!n) return;
  const uint4* src = hitpool + hit_start[i] * 2;
  const uint64_t base = hit_base[i];
  uint64_t run = pos_base[i];
  for (uint32_t k0 = 0; k0 < n; k0 += GATHER_LANES) {
    const uint32_t k = k0 + lane;
    const bool on = k < n && base + k < hit_cap;
    uint4 a = make_uint4(0, 0, 0, 0), b = a;
    if (on) { a = src[2 * k]; b = src[2 * k + 1]; }
    uint64_t x = b.y;                                  // positions of this hit, then of those up to it
#pragma unroll
    for (int d = 1; d < GATHER_LANES; d <<= 1) {
      const uint64_t y = __shfl_up_sync(mask, x, d, GATHER_LANES);
      if ((int)lane >= d) x += y;
    }
    const uint64_t at = run + x - b.y;
    run += __shfl_sync(mask, x, GATHER_LANES - 1, GATHER_LANES);
    if (on) {
      b.z = (uint32_t)at; b.w = (uint32_t)(at >> 32);
      hits[2 * (base + k)] = a;
      hits[2 * (base + k) + 1] = b;
      seg_off[base + k] = at;
    }
  }
}

// Per-read work record, words 1 and 2: MemHits and positions reported for read i.
__global__ void k_work_log(const uint64_t* __restrict__ hit_base, const uint64_t* __restrict__ npos_scan, uint32_t nq,
                           uint32_t* __restrict__ log) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  uint64_t h0 = hit_base[i], h1 = hit_base[i + 1];
  log[4 * (size_t)i + 1] = (uint32_t)(h1 - h0);
  uint64_t np = npos_scan[h1] - npos_scan[h0];
  log[4 * (size_t)i + 2] = np > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)np;
}

// Graph-captured locate chain: queries whose intervals did not fit the pool report none
// (they are flagged; the batch is rerun), so the CSR never reaches past the pool.
__global__ void k_zero_failed(const uint32_t* __restrict__ status, uint32_t n, uint32_t* __restrict__ niv,
                              uint64_t* __restrict__ nhits) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n && status[k] != 0) { niv[k] = 0; nhits[k] = 0; }
}

// seg_off[k] = total for k in [nseg, cap]: segments past the count are empty.
__global__ void k_seal_segments(uint64_t* __restrict__ seg_off, const uint64_t* __restrict__ nseg_p,
                                const uint64_t* __restrict__ total_p, uint64_t cap) {
  const uint64_t nseg = *nseg_p, total = *total_p;
  for (uint64_t k = nseg + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k <= cap; k += (uint64_t)gridDim.x * blockDim.x)
    seg_off[k] = total;
}

__global__ void k_iota(uint32_t* __restrict__ ids, uint32_t n) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) ids[k] = k;
}

// seen[] zeroed by the caller; *bad set when ids is not a permutation of 0..n-1.
__global__ void k_check_perm(const uint32_t* __restrict__ ids, uint32_t n, uint32_t* __restrict__ seen,
                             uint32_t* __restrict__ bad) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  uint32_t i = ids[k];
  if (i >= n || atomicExch(seen + i, 1u) != 0) atomicExch(bad, 1u);
}

}  // namespace hfm
