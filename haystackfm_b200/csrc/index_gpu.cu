// index_gpu.cu — FM-index construction on the GPU, emitting the same bincode bytes as the
// CPU builder (index_build.cpp).
//
// Replaces FmIndex::build / BidirFmIndex::build (src/fm_index/mod.rs:209-284,
// src/fm_index/bidir_index.rs:91-116), whose wgpu pipelines sort suffixes by prefix
// doubling (src/suffix_array/gpu.rs:86) and build a 16-lane Occ table
// (src/occ/gpu.rs:34).  This builder keeps the CPU builder's contract instead — compacted
// lanes, either alphabet, the depth-k lookup table (src/fm_index/mod.rs:117-195) — so its
// bytes equal FmIndex::build_cpu_with's for the same input, at genome scale.
//
// Suffix sorting is prefix doubling (Manber & Myers) over CUB radix sort, refining only the
// suffixes whose group is still tied (as Larsson & Sadakane do): round 0 sorts every suffix
// by its first 21 (ACGT texts) or 12 (IUPAC texts) codes packed into 64 bits; each later
// round h sorts the tied suffixes by (rank[i], rank[i + h]) and splits their groups.
// Ranks are 1 + the first SA slot of the suffix's group; 0 stands for "past the end", so a
// proper prefix sorts first, as build_suffix_array_naive (src/suffix_array/cpu.rs:20-25).
// Device memory: about 38 bytes per text position during the sort, one allocation for all of
// a build.
//
// Everything that takes time in proportion to the text runs here: sequences are joined,
// counted and reversed on the device, the sizes of all sections follow from the code counts
// and the sequence starts alone, and the sections are copied from the device to their places
// in the returned block.  With host loops for these, a vector per section, three copies of
// the bytes, some 45 allocations and a thread per 64 rows, a 5 Mbp bidirectional IUPAC build
// took 77 ms on a B200 (a call and a copy of its 25 MB); it takes 12.5.

#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "hfm_internal.h"

namespace hfm {

#define GCK(call)                                                                                 \
  do {                                                                                            \
    cudaError_t _e = (call);                                                                      \
    if (_e != cudaSuccess)                                                                        \
      return set_error(_e == cudaErrorMemoryAllocation ? HFM_E_OOM : HFM_E_CUDA,                  \
                       std::string(#call) + ": " + cudaGetErrorString(_e));                       \
  } while (0)
#define GRET(x) do { int _r = (x); if (_r != HFM_OK) return _r; } while (0)

// One device allocation, handed out in pieces.  take() before a base is there only adds up
// (the pass that finds the size); back_to() gives the pieces after a mark back.
struct Arena {
  uint8_t* base = nullptr;
  uint64_t used = 0, most = 0;
  template <class T> T* take(uint64_t count) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (count * sizeof(T) + 255) & ~255ull;
    most = std::max(most, used);
    return p;
  }
  void back_to(uint64_t mark) { used = mark; }
};

static unsigned grid_for(uint64_t n, unsigned t = 256) {
  uint64_t g = (n + t - 1) / t;
  return (unsigned)std::min<uint64_t>(g, 1u << 30);
}

// ---- the text ------------------------------------------------------------------------

// Joins the sequences (codes, back to back) with a sentinel after each (bounds: exclusive
// ends) and counts the codes; a thread takes 16 positions.  `text` has room for whole chunks.
__global__ void __launch_bounds__(256) k_join(const uint8_t* __restrict__ codes, const uint32_t* __restrict__ bounds,
                                              uint32_t nseq, uint64_t n, uint8_t* __restrict__ text,
                                              uint32_t* __restrict__ freq) {
  __shared__ uint32_t s_freq[16];
  if (threadIdx.x < 16) s_freq[threadIdx.x] = 0;
  __syncthreads();
  uint32_t cnt[16];
#pragma unroll
  for (int c = 0; c < 16; c++) cnt[c] = 0;
  const uint64_t chunks = (n + 15) / 16;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < chunks; w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = nseq - 1;                         // sequence of the first position
    while (lo < hi) {
      const uint32_t mid = (lo + hi) / 2;
      if (bounds[mid] > w * 16) hi = mid; else lo = mid + 1;
    }
    uint64_t end = bounds[lo];
    uint32_t out[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const uint64_t p = w * 16 + k;
      if (p < n) {
        uint32_t c = 0;
        if (p + 1 == end) { lo++; if (lo < nseq) end = bounds[lo]; }
        else c = codes[p - lo];
        out[k >> 2] |= c << (8 * (k & 3));
#pragma unroll
        for (int x = 0; x < 16; x++) cnt[x] += c == (uint32_t)x ? 1u : 0u;
      }
    }
    reinterpret_cast<uint4*>(text)[w] = make_uint4(out[0], out[1], out[2], out[3]);
  }
#pragma unroll
  for (int c = 0; c < 16; c++) {
    const uint32_t v = __reduce_add_sync(0xFFFFFFFFu, cnt[c]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_freq[c], v);
  }
  __syncthreads();
  if (threadIdx.x < 16 && s_freq[threadIdx.x]) atomicAdd(freq + threadIdx.x, s_freq[threadIdx.x]);
}

// Reverses p[0..n) in place.
__global__ void k_reverse(uint8_t* __restrict__ p, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n / 2; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint8_t a = p[i];
    p[i] = p[n - 1 - i];
    p[n - 1 - i] = a;
  }
}

// ---- suffix sorting ------------------------------------------------------------------

// key[i] = the first k codes of suffix i, each as code + 1 in `bits` bits (0 past the end).
__global__ void k_sa_keys0(const uint8_t* __restrict__ t, uint64_t n, int bits, int k, uint64_t* __restrict__ key,
                           uint32_t* __restrict__ val) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t v = 0;
    for (int j = 0; j < k; j++) v = (v << bits) | (i + j < n ? (uint64_t)t[i + j] + 1 : 0ull);
    key[i] = v;
    val[i] = (uint32_t)i;
  }
}

// g_in[j] = slot of sorted key j (slots: `slot` or j itself) when it starts a new group, else 0.
__global__ void k_head_slots(const uint64_t* __restrict__ key, const uint32_t* __restrict__ slot, uint64_t m,
                             uint32_t* __restrict__ g_in) {
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < m; j += (uint64_t)gridDim.x * blockDim.x)
    g_in[j] = j == 0 || key[j] != key[j - 1] ? (slot ? slot[j] : (uint32_t)j) : 0u;
}

// sa[slot] = suffix; rank[suffix] = 1 + first slot of its group; tied[j] = its group has more
// than one member.
__global__ void k_set_ranks(const uint64_t* __restrict__ key, const uint32_t* __restrict__ slot,
                            const uint32_t* __restrict__ suf, const uint32_t* __restrict__ g, uint64_t m,
                            uint32_t* __restrict__ sa, uint32_t* __restrict__ rank, uint8_t* __restrict__ tied) {
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < m; j += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = suf[j];
    const uint64_t k = key[j];
    sa[slot ? slot[j] : j] = i;
    rank[i] = g[j] + 1;
    tied[j] = (j > 0 && key[j - 1] == k) || (j + 1 < m && key[j + 1] == k) ? 1 : 0;
  }
}

// Round h: the tied suffixes (slots U) keyed by (rank[i], rank[i + h]), `bits` bits each.
__global__ void k_sa_keys(const uint32_t* __restrict__ U, uint64_t m, const uint32_t* __restrict__ sa,
                          const uint32_t* __restrict__ rank, uint64_t n, uint64_t h, int bits, uint64_t* __restrict__ key,
                          uint32_t* __restrict__ val) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < m; t += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t i = sa[U[t]];
    uint64_t r2 = (uint64_t)i + h < n ? rank[i + h] : 0u;
    key[t] = ((uint64_t)rank[i] << bits) | r2;
    val[t] = i;
  }
}

struct SaBufs {
  uint64_t *k0, *k1;
  uint32_t *v0, *v1, *U, *rank;
  uint8_t *tied, *tmp;
  uint64_t* nsel;
  size_t tmp_bytes;
};

static int take_sa_bufs(Arena& A, uint64_t n, SaBufs& B) {
  B.k0 = A.take<uint64_t>(n); B.k1 = A.take<uint64_t>(n);
  B.v0 = A.take<uint32_t>(n); B.v1 = A.take<uint32_t>(n);
  B.U = A.take<uint32_t>(n); B.rank = A.take<uint32_t>(n);
  B.tied = A.take<uint8_t>(n); B.nsel = A.take<uint64_t>(1);
  // what CUB asks for grows with the number of items
  size_t need[3] = {0, 0, 0};
  cub::DoubleBuffer<uint64_t> dk(nullptr, nullptr);
  cub::DoubleBuffer<uint32_t> dv(nullptr, nullptr);
  GCK(cub::DeviceRadixSort::SortPairs(nullptr, need[0], dk, dv, n, 0, 64));
  GCK(cub::DeviceScan::InclusiveScan(nullptr, need[1], (uint32_t*)nullptr, (uint32_t*)nullptr, cub::Max(), n));
  GCK(cub::DeviceSelect::Flagged(nullptr, need[2], (uint32_t*)nullptr, (uint8_t*)nullptr, (uint32_t*)nullptr,
                                 (uint64_t*)nullptr, (int64_t)n));
  B.tmp_bytes = std::max({need[0], need[1], need[2]}) + 4096;
  B.tmp = A.take<uint8_t>(B.tmp_bytes);
  return HFM_OK;
}

// Suffix array of d_text[0..n) into d_sa (device, n u32).
static int gpu_suffix_array(const uint8_t* d_text, uint64_t n, uint32_t* d_sa, uint8_t max_code, SaBufs B, cudaStream_t s) {
  const int bits = max_code + 1 <= 7 ? 3 : 5;
  const int k = 64 / bits;
  int rank_bits = 1;                                        // ranks and 0: 0..n
  while ((n >> rank_bits) != 0) rank_bits++;
  uint64_t m = n;                                           // suffixes sorted in this round: slots U, or all
  for (uint64_t h = 0; m > 0; h = h ? 2 * h : (uint64_t)k) {
    if (h >= 2 * n + k) return set_error(HFM_E_CUDA, "suffix sort did not converge");
    const uint32_t* slots = h ? B.U : nullptr;
    if (h) k_sa_keys<<<grid_for(m), 256, 0, s>>>(slots, m, d_sa, B.rank, n, h, rank_bits, B.k0, B.v0);
    else k_sa_keys0<<<grid_for(n), 256, 0, s>>>(d_text, n, bits, k, B.k0, B.v0);
    GCK(cudaGetLastError());
    cub::DoubleBuffer<uint64_t> dk(B.k0, B.k1);
    cub::DoubleBuffer<uint32_t> dv(B.v0, B.v1);
    size_t bytes = B.tmp_bytes;
    GCK(cub::DeviceRadixSort::SortPairs(B.tmp, bytes, dk, dv, m, 0, h ? 2 * rank_bits : bits * k, s));
    const uint64_t* kk = dk.Current();
    uint32_t* vv = dv.Current();
    uint32_t* gi = reinterpret_cast<uint32_t*>(dk.Alternate());          // 2m u32 of free room
    uint32_t* gg = gi + m;
    k_head_slots<<<grid_for(m), 256, 0, s>>>(kk, slots, m, gi);
    GCK(cudaGetLastError());
    bytes = B.tmp_bytes;
    GCK(cub::DeviceScan::InclusiveScan(B.tmp, bytes, gi, gg, cub::Max(), m, s));
    k_set_ranks<<<grid_for(m), 256, 0, s>>>(kk, slots, vv, gg, m, d_sa, B.rank, B.tied);
    GCK(cudaGetLastError());
    // the next round's tied slots (ascending, so they keep the group order) go to the value
    // buffer the sort left free, which then becomes U (the old U takes its place)
    uint32_t*& vfree = vv == B.v0 ? B.v1 : B.v0;
    bytes = B.tmp_bytes;
    if (h) {
      GCK(cub::DeviceSelect::Flagged(B.tmp, bytes, slots, B.tied, vfree, B.nsel, (int64_t)m, s));
    } else {
      thrust::counting_iterator<uint32_t> it(0);
      GCK(cub::DeviceSelect::Flagged(B.tmp, bytes, it, B.tied, vfree, B.nsel, (int64_t)m, s));
    }
    GCK(cudaMemcpyAsync(&m, B.nsel, 8, cudaMemcpyDeviceToHost, s));
    GCK(cudaStreamSynchronize(s));
    std::swap(B.U, vfree);
  }
  return HFM_OK;
}

// ---- BWT, Occ records, sampled SA, lookup table ---------------------------------------

// Codes to lanes (compacted in code order), the record's shape, and the rows of smaller lanes.
struct LaneMap { uint8_t s2l[16], l2s[16]; uint32_t base[17]; uint32_t L, width, enc, stride; };

constexpr int ROW_WARPS = 4;                // superblocks (512 rows, 8 records) of a block, a warp each
constexpr uint32_t OCC_REC_MAX = 16 * 6 + 16 * 8, SSA_REC = 14;

// Bits of the text positions whose rows are sampled whatever the rate: the sequence starts
// (src/fm_index/mod.rs:154-162).
__global__ void k_forced(const uint32_t* __restrict__ bounds, uint32_t nseq, uint32_t* __restrict__ bits) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nseq; k += gridDim.x * blockDim.x) {
    const uint32_t p = k ? bounds[k - 1] : 0u;
    atomicOr(bits + (p >> 5), 1u << (p & 31));
  }
}

// The rows of a superblock: their BWT codes (src/bwt/cpu.rs:14-35) as bit planes of the lane,
// which rows are sampled (a multiple of the rate, or forced; src/suffix_array/mod.rs:71-118),
// and how many rows each lane has, the sampled ones counted as lane L: cnt[lane * nsb + sb].
//
// A warp takes 32 rows at a time, so that loads are consecutive and a ballot is a plane; all
// 16 suffix-array entries of a lane are in flight before the first code is looked up.
__global__ void __launch_bounds__(ROW_WARPS * 32) k_rows(const uint8_t* __restrict__ t, const uint32_t* __restrict__ sa,
                                                         uint64_t n, uint64_t nsb, LaneMap M, uint32_t rate,
                                                         const uint32_t* __restrict__ forced, uint32_t* __restrict__ planes,
                                                         uint32_t* __restrict__ words, uint32_t* __restrict__ cnt) {
  __shared__ uint8_t s_lane[16];
  if (threadIdx.x < 16) s_lane[threadIdx.x] = M.s2l[threadIdx.x];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t sb = blockIdx.x * (uint64_t)ROW_WARPS + (threadIdx.x >> 5);
  if (sb >= nsb) return;
  uint32_t v[16];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint64_t r = sb * 512 + k * 32 + lane;
    v[k] = r < n ? sa[r] : 0u;
  }
  uint8_t c[16];
#pragma unroll
  for (int k = 0; k < 16; k++) c[k] = t[v[k] == 0 ? n - 1 : v[k] - 1];
  uint32_t count = 0;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint64_t first = sb * 512 + k * 32;
    if (first >= ((n + 63) & ~63ull)) break;
    const bool in = first + lane < n;
    const uint32_t l = s_lane[c[k] & 15];
    const bool take = in && ((rate ? v[k] % rate == 0 : v[k] == 0) || ((forced[v[k] >> 5] >> (v[k] & 31)) & 1));
    const uint32_t all = __ballot_sync(0xFFFFFFFFu, in), sel = __ballot_sync(0xFFFFFFFFu, take);
    uint32_t mine = 0, same = all;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, in && ((l >> p) & 1));
      if (lane == p) mine = b;
      same &= (lane >> p) & 1 ? b : ~b;
    }
    if (lane == M.L) same = sel;            // L <= 16
    count += __popc(same);
    // a record's planes: the 4 of its first 32 rows, then of the others
    if (lane < 4) planes[first / 8 + lane] = mine;
    if (lane == 4) words[first / 32] = sel;
  }
  if (lane <= M.L) cnt[lane * nsb + sb] = count;
}

// dst[0..2) = v, as 16-bit halves (the records are 2-byte aligned).
__device__ __forceinline__ void put32(uint16_t* dst, uint32_t v) { dst[0] = (uint16_t)v; dst[1] = (uint16_t)(v >> 16); }

// The records [sb u32 x L][delta u16 x L][words u64 x width] (src/occ/mod.rs:114-183) of a
// superblock with its checkpoint (src/occ/cpu.rs:23-119), its sampled-SA records [word u64]
// [sb u32][delta u16], and the sampled values.  cum = exclusive scan of k_rows' counts over
// all lanes, one after the other.  Records are put together in shared memory and written by
// 16 bytes.
__global__ void __launch_bounds__(ROW_WARPS * 32) k_records(const uint32_t* __restrict__ sa, uint64_t n, uint64_t nsb,
                                                            LaneMap M, const uint32_t* __restrict__ planes,
                                                            const uint32_t* __restrict__ words, const uint32_t* __restrict__ cum,
                                                            uint8_t* __restrict__ rec, uint32_t* __restrict__ sbout,
                                                            uint8_t* __restrict__ ssa, uint32_t* __restrict__ vals) {
  __shared__ __align__(16) uint8_t s_occ[ROW_WARPS][8 * OCC_REC_MAX];
  __shared__ __align__(16) uint8_t s_ssa[ROW_WARPS][8 * SSA_REC];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t sb = blockIdx.x * (uint64_t)ROW_WARPS + warp;
  if (sb >= nsb) return;
  const uint32_t nrec = (uint32_t)min((uint64_t)8, (n + 63) / 64 - sb * 8);
  const uint32_t base = lane <= M.L ? cum[lane * nsb + sb] - M.base[lane] : 0u;
  if (lane < M.L) sbout[sb * M.L + lane] = base;
  uint32_t run = 0;                         // rows of this lane (sampled rows) before the record
  for (uint32_t b = 0; b < nrec; b++) {
    const uint64_t blk = sb * 8 + b;
    const uint4 p0 = reinterpret_cast<const uint4*>(planes)[blk * 2], p1 = reinterpret_cast<const uint4*>(planes)[blk * 2 + 1];
    const uint2 sel = reinterpret_cast<const uint2*>(words)[blk];
    const uint64_t left = n - blk * 64;
    const uint64_t all = left >= 64 ? ~0ull : (1ull << left) - 1;
    const uint64_t p[4] = {(uint64_t)p1.x << 32 | p0.x, (uint64_t)p1.y << 32 | p0.y, (uint64_t)p1.z << 32 | p0.z,
                           (uint64_t)p1.w << 32 | p0.w};
    uint64_t same = all, plane = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      same &= (lane >> k) & 1 ? p[k] : ~p[k];
      if (lane == k) plane = p[k];
    }
    const uint64_t word = (uint64_t)sel.y << 32 | sel.x;
    if (lane == M.L) same = word;
    uint16_t* r = reinterpret_cast<uint16_t*>(s_occ[warp] + b * M.stride);
    if (lane < M.L) {
      put32(r + lane * 2, base);
      r[M.L * 2 + lane] = (uint16_t)run;
    } else if (lane == M.L) {
      uint16_t* w = reinterpret_cast<uint16_t*>(s_ssa[warp] + b * SSA_REC);
      put32(w, sel.x); put32(w + 2, sel.y); put32(w + 4, base);
      w[6] = (uint16_t)run;
    }
    if (lane < M.width) {
      const uint64_t x = M.enc == 0 ? plane : same;
      put32(r + M.L * 3 + lane * 4, (uint32_t)x); put32(r + M.L * 3 + lane * 4 + 2, (uint32_t)(x >> 32));
    }
    uint32_t at = __shfl_sync(0xFFFFFFFFu, base + run, M.L);      // samples before this record
    const uint32_t below = (1u << lane) - 1u;
    if ((sel.x >> lane) & 1) vals[at + __popc(sel.x & below)] = sa[blk * 64 + lane];
    at += __popc(sel.x);
    if ((sel.y >> lane) & 1) vals[at + __popc(sel.y & below)] = sa[blk * 64 + 32 + lane];
    run += (uint32_t)__popcll(same);
  }
  __syncwarp();
  auto flush = [&](const uint8_t* from, uint8_t* to, uint32_t bytes) {       // even, `to` by 16
    for (uint32_t k = lane; k < bytes / 16; k += 32) reinterpret_cast<uint4*>(to)[k] = reinterpret_cast<const uint4*>(from)[k];
    for (uint32_t k = bytes / 16 * 8 + lane; k < bytes / 2; k += 32)
      reinterpret_cast<uint16_t*>(to)[k] = reinterpret_cast<const uint16_t*>(from)[k];
  };
  flush(s_occ[warp], rec + sb * 8 * M.stride, nrec * M.stride);
  flush(s_ssa[warp], ssa + sb * 8 * SSA_REC, nrec * SSA_REC);
}

// OccTable::rank over the records just built (src/occ/mod.rs:330-363); `c` occurs in the text.
__device__ uint32_t ref_rank(const uint8_t* rec, const LaneMap& M, uint32_t lane, uint32_t i) {
  if (i == 0) return 0;
  const uint32_t pos = i - 1, off = pos & 63;
  const uint16_t* r = reinterpret_cast<const uint16_t*>(rec + (uint64_t)(pos >> 6) * M.stride);
  const uint32_t sbv = r[lane * 2] | (uint32_t)r[lane * 2 + 1] << 16, dv = r[M.L * 2 + lane];
  auto word = [&](uint32_t w) {
    const uint16_t* p = r + M.L * 3 + w * 4;
    return (uint64_t)p[0] | (uint64_t)p[1] << 16 | (uint64_t)p[2] << 32 | (uint64_t)p[3] << 48;
  };
  uint64_t m = ~0ull;
  if (M.enc == 1) m = word(lane);
  else for (uint32_t p = 0; p < M.width; p++) { const uint64_t v = word(p); m &= (lane >> p) & 1 ? v : ~v; }
  return sbv + dv + (uint32_t)__popcll(m & (~0ull >> (63 - off)));
}

// One level of the lookup table (LookupTable::build, src/fm_index/lookup.rs:37-91): entry idx
// extends entry idx / 4 of the level before (nullptr: the whole text) by code idx % 4 + 1.  An
// empty parent and a symbol that is absent from the text leave (0, 0).
__global__ void k_lookup_level(const uint8_t* __restrict__ rec, LaneMap M, const uint2* __restrict__ in, uint32_t n,
                               uint64_t size, uint2* __restrict__ out) {
  for (uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; idx < size; idx += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 p = in ? in[idx >> 2] : make_uint2(0, n);
    const uint32_t lane = M.s2l[(idx & 3) + 1];
    uint2 res = make_uint2(0, 0);
    if (p.x < p.y && lane != 0xFF) {
      const uint32_t base = M.base[lane];   // C of the code: the rows of smaller lanes
      res = make_uint2(base + ref_rank(rec, M, lane, p.x), base + ref_rank(rec, M, lane, p.y));
    }
    out[idx] = res;
  }
}

// The device side of one direction: its sections, for the copies to the host.
struct FmWork {
  uint32_t *planes, *words, *cnt, *cum, *forced, *sbout, *vals;
  uint8_t *rec, *ssa, *tmp;
  uint2 *lut, *lut2;
  size_t tmp_bytes;
};

static int take_fm_work(Arena& A, const FmMeta& f, FmWork& W) {
  const uint64_t n = f.text_len, nblk = (n + 63) / 64, nsb = (n + 511) / 512, lanes = f.num_lanes + 1;
  W.planes = A.take<uint32_t>(nblk * 8); W.words = A.take<uint32_t>(nblk * 2);
  W.cnt = A.take<uint32_t>(lanes * nsb); W.cum = A.take<uint32_t>(lanes * nsb);
  W.forced = A.take<uint32_t>((n + 31) / 32);
  W.rec = A.take<uint8_t>(f.n_block); W.sbout = A.take<uint32_t>(f.n_sb);
  W.ssa = A.take<uint8_t>(f.n_ssa); W.vals = A.take<uint32_t>(f.n_vals);
  W.lut = A.take<uint2>(f.n_lut); W.lut2 = A.take<uint2>(f.n_lut / 4);
  W.tmp_bytes = 0;
  GCK(cub::DeviceScan::ExclusiveSum(nullptr, W.tmp_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, lanes * nsb));
  W.tmp = A.take<uint8_t>(W.tmp_bytes);
  return HFM_OK;
}

// Everything of an FmIndex that the counts of its codes and its sequence starts determine.
static void describe(const uint32_t freq[16], const hfm_build_opts& o, uint32_t lookup_depth, FmMeta& f, LaneMap& M) {
  const uint64_t n = f.text_len;
  f.tag = (uint8_t)o.alphabet_tag; f.encoding = o.occ_encoding; f.rate = o.sa_sample_rate;
  f.num_sequences = (uint32_t)f.bounds.size(); f.lookup_depth = lookup_depth;
  // C array (src/c_array.rs:14-31) and lanes: the symbols present, in code order
  // (src/occ/cpu.rs:23-60)
  std::memset(f.s2l, 0xFF, 16); std::memset(f.l2s, 0, 16);
  uint32_t acc = 0;
  uint8_t L = 0, P = 0;
  for (int c = 0; c < 16; c++) {
    f.C[c] = acc;
    if (freq[c]) { f.s2l[c] = L; f.l2s[L] = (uint8_t)c; M.base[L] = acc; L++; }
    acc += freq[c];
  }
  M.base[L] = acc;                          // the sampled rows are counted after the last lane
  if (L > 1) { uint32_t v = L - 1; while (v) { P++; v >>= 1; } }
  f.num_lanes = L; f.num_planes = P;
  std::memcpy(M.s2l, f.s2l, 16); std::memcpy(M.l2s, f.l2s, 16);
  M.L = L; M.width = f.encoding == 0 ? P : L; M.enc = f.encoding; M.stride = L * 6u + M.width * 8u;
  f.block_stride = M.stride;
  f.n_sb = (n + 511) / 512 * L; f.n_block = (n + 63) / 64 * M.stride; f.n_ssa = (n + 63) / 64 * SSA_REC;
  f.n_vals = f.rate ? (n + f.rate - 1) / f.rate : 1;
  for (size_t k = 0; k + 1 < f.bounds.size(); k++) f.n_vals += !f.rate || f.bounds[k] % f.rate != 0;
  f.n_lut = lookup_depth ? 1ull << (2 * lookup_depth) : 0;
}

// Writes one FmIndex at `at`: small fields by the host, sections by copies from the device.
struct DeviceWriter {
  uint8_t* at;
  const void* sections[5];
  cudaStream_t stream;
  cudaError_t err = cudaSuccess;
  void put(const void* p, size_t k) { if (k) std::memcpy(at, p, k); at += k; }
  void section(FmSection id, uint64_t bytes) {
    if (bytes && err == cudaSuccess) err = cudaMemcpyAsync(at, sections[id], bytes, cudaMemcpyDeviceToHost, stream);
    at += bytes;
  }
};

struct SizeWriter {
  uint64_t bytes = 0;
  void put(const void*, size_t k) { bytes += k; }
  void section(FmSection, uint64_t k) { bytes += k; }
};

// One FmIndex of d_text[0..n) to `out`.  Workspaces come from A and go back to it.
static int build_fm_gpu(const uint8_t* d_text, const FmMeta& f, const LaneMap& M, const uint32_t* d_bounds, Arena& A,
                        uint8_t* out, cudaStream_t s) {
  const uint64_t n = f.text_len, nsb = (n + 511) / 512, mark = A.used;
  uint32_t* sa = A.take<uint32_t>(n);
  const uint64_t mark_sa = A.used;
  SaBufs B;
  GRET(take_sa_bufs(A, n, B));
  GRET(gpu_suffix_array(d_text, n, sa, f.l2s[f.num_lanes - 1], B, s));
  A.back_to(mark_sa);
  FmWork W;
  GRET(take_fm_work(A, f, W));
  GCK(cudaMemsetAsync(W.forced, 0, (n + 31) / 32 * 4, s));
  k_forced<<<grid_for(f.num_sequences), 256, 0, s>>>(d_bounds, f.num_sequences, W.forced);
  const unsigned grid = (unsigned)((nsb + ROW_WARPS - 1) / ROW_WARPS);
  k_rows<<<grid, ROW_WARPS * 32, 0, s>>>(d_text, sa, n, nsb, M, f.rate, W.forced, W.planes, W.words, W.cnt);
  GCK(cudaGetLastError());
  GCK(cub::DeviceScan::ExclusiveSum(W.tmp, W.tmp_bytes, W.cnt, W.cum, (f.num_lanes + 1) * nsb, s));
  k_records<<<grid, ROW_WARPS * 32, 0, s>>>(sa, n, nsb, M, W.planes, W.words, W.cum, W.rec, W.sbout, W.ssa, W.vals);
  GCK(cudaGetLastError());
  // levels alternate between the two tables so that the last one ends in lut
  const uint2* in = nullptr;
  for (uint32_t level = 1; level <= f.lookup_depth; level++) {
    const uint64_t size = 1ull << (2 * level);
    uint2* to = ((f.lookup_depth - level) & 1) ? W.lut2 : W.lut;
    k_lookup_level<<<grid_for(size), 256, 0, s>>>(W.rec, M, in, (uint32_t)n, size, to);
    in = to;
  }
  GCK(cudaGetLastError());
  DeviceWriter w{out, {W.sbout, W.rec, W.ssa, W.vals, W.lut}, s};
  write_fm(f, w);
  GCK(w.err);
  A.back_to(mark);                          // in stream order: what comes next is queued behind the copies
  return HFM_OK;
}

}  // namespace hfm

using namespace hfm;

// Blocks up to this size are pinned (copies at the link's rate, reused by the next call);
// above it pinned memory that the cache goes on holding would cost more than it gives.
static constexpr uint64_t BUILD_PINNED_MAX = 256ull << 20;

extern "C" int hfm_build_index_gpu(const uint8_t* codes, const uint64_t* seq_off, uint32_t nseq,
                                   const char* const* headers, const hfm_build_opts* opts, int kind, int device,
                                   uint8_t** bytes_out, size_t* len_out) {
  if (!codes && nseq) return set_error(HFM_E_ARG, "codes is NULL");
  if (nseq == 0) return set_error(HFM_E_ARG, "empty sequence list");
  if (!opts || !bytes_out || !len_out || !seq_off) return set_error(HFM_E_ARG, "NULL argument");
  if (kind != HFM_KIND_FM && kind != HFM_KIND_BIDIR) return set_error(HFM_E_ARG, "kind must be 0 or 1");
  if (opts->alphabet_tag > 1 || opts->occ_encoding > 1) return set_error(HFM_E_ARG, "bad alphabet tag or encoding");
  if (opts->lookup_depth > 13) return set_error(HFM_E_ARG, "lookup_depth above 13 (4^13 entries)");
  FmMeta fwd, rev;
  GRET(sequence_bounds(codes, seq_off, nseq, headers, fwd.bounds, fwd.headers));
  int ndev = 0;
  GCK(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) return set_error(HFM_E_ARG, "device ordinal out of range");
  GCK(cudaSetDevice(device));
  int sms = 0;
  GCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const uint64_t n = fwd.bounds.back(), raw = n - nseq;
  const bool both = kind == HFM_KIND_BIDIR;
  fwd.text_len = rev.text_len = (uint32_t)n;
  try {
    // reverse_as_sequence (src/fm_index/bidir_index.rs:523-532): one sequence of the same codes
    rev.bounds.assign(1, (uint32_t)n); rev.headers.assign(1, "seq_0");
  } catch (const std::bad_alloc&) {
    return set_error(HFM_E_OOM, "host allocation failed");
  }
  struct Resources {
    cudaStream_t s = nullptr;
    void* dev = nullptr;
    uint8_t* out = nullptr;
    ~Resources() {
      if (s) { cudaStreamSynchronize(s); cudaStreamDestroy(s); }
      if (dev) cudaFree(dev);
      if (out) host_result_free(out);
    }
  } R;
  GCK(cudaStreamCreateWithFlags(&R.s, cudaStreamNonBlocking));
  // the sizes of the pieces, for the largest lane count and both sample counts, then the pieces
  Arena A;
  uint8_t *text = nullptr, *staged = nullptr;
  uint32_t *d_bounds = nullptr, *d_freq = nullptr;
  LaneMap M{};
  uint32_t freq[16];
  for (int pass = 0; pass < 2; pass++) {
    A.used = 0;
    text = A.take<uint8_t>(n + 16);
    d_bounds = A.take<uint32_t>(nseq); d_freq = A.take<uint32_t>(16);
    if (pass) break;
    const uint64_t mark = A.used;
    A.take<uint8_t>(raw);
    A.back_to(mark);
    A.take<uint32_t>(n);
    const uint64_t mark_sa = A.used;
    SaBufs B;
    GRET(take_sa_bufs(A, n, B));
    A.back_to(mark_sa);
    for (uint32_t& x : freq) x = 1;
    describe(freq, *opts, opts->lookup_depth, fwd, M);
    FmWork W;
    GRET(take_fm_work(A, fwd, W));
    if (cudaMalloc(&R.dev, A.most) != cudaSuccess) {
      cudaGetLastError();
      return set_error(HFM_E_OOM, "cudaMalloc failed during GPU index construction: " + std::to_string(A.most) + " bytes");
    }
    A.base = static_cast<uint8_t*>(R.dev);
  }
  const uint64_t mark = A.used;
  staged = A.take<uint8_t>(raw);
  A.back_to(mark);
  if (raw) GCK(cudaMemcpyAsync(staged, codes + seq_off[0], raw, cudaMemcpyHostToDevice, R.s));
  GCK(cudaMemcpyAsync(d_bounds, fwd.bounds.data(), (size_t)nseq * 4, cudaMemcpyHostToDevice, R.s));
  GCK(cudaMemsetAsync(d_freq, 0, 64, R.s));
  k_join<<<std::min<unsigned>(grid_for((n + 15) / 16), (unsigned)sms * 4), 256, 0, R.s>>>(staged, d_bounds, nseq, n, text, d_freq);
  GCK(cudaGetLastError());
  GCK(cudaMemcpyAsync(freq, d_freq, 64, cudaMemcpyDeviceToHost, R.s));
  GCK(cudaStreamSynchronize(R.s));
  describe(freq, *opts, opts->lookup_depth, fwd, M);
  SizeWriter fwd_size, rev_size;
  write_fm(fwd, fwd_size);
  LaneMap Mr = M;
  if (both) {
    describe(freq, *opts, 0, rev, Mr);
    write_fm(rev, rev_size);
  }
  // FmIndex bytes, or BidirFmIndex bytes [u32 fwd_len][fwd][rev] (src/fm_index/bidir_index.rs:183-192)
  const uint64_t total = both ? 4 + fwd_size.bytes + rev_size.bytes : fwd_size.bytes;
  R.out = static_cast<uint8_t*>(total <= BUILD_PINNED_MAX ? host_result_alloc(total) : std::malloc(total));
  if (!R.out) return set_error(HFM_E_OOM, "host allocation failed during index construction");
  uint8_t* at = R.out;
  if (both) {
    const uint32_t fl = (uint32_t)fwd_size.bytes;
    std::memcpy(at, &fl, 4);
    at += 4;
  }
  GRET(build_fm_gpu(text, fwd, M, d_bounds, A, at, R.s));
  if (both) {
    // reversed without its final sentinel, which stays where it is
    if (n > 2) k_reverse<<<grid_for((n - 1) / 2), 256, 0, R.s>>>(text, n - 1);
    GCK(cudaGetLastError());
    GRET(build_fm_gpu(text, rev, Mr, d_bounds, A, at + fwd_size.bytes, R.s));
  }
  GCK(cudaStreamSynchronize(R.s));
  *bytes_out = R.out; *len_out = total;
  R.out = nullptr;
  return HFM_OK;
}
