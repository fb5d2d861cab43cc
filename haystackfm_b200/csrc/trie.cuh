// trie.cuh — the first forward sweep of up to 32 reads of an IUPAC text by one block.
//
// On a text with N runs and ambiguity codes a read matches tens of text strings at once,
// nearly all of them windows that touch an N run: they depend on the read's first or last
// few bases only, so the reads of a batch extend the same intervals over and over (98% of
// the extensions of 60,000 reads of 150 bp on a 100 Mbp assembly repeat one made for another
// read).  Here the union of the interval sets of a group's reads is kept as one list of
// nodes, each with the mask of the reads that hold it.  From one position to the next every
// node is split by symbol once, whatever the number of reads; the child of symbol s keeps
// the reads whose code there matches s.  A child has one parent and one symbol, so the list
// never holds an interval twice and no lookup is needed.  The threads of the block take a
// node each, one-row nodes (one LF step on one record) and larger ones (16 counts at both
// borders) in lists of their own, so that a warp runs one kind at a time.  The order of a
// list is the order in which its warps reserved their places: nothing depends on it.
//
// A block, not a warp, per group: reads with an N among their first bases grow a group's
// list to thousands of nodes, and with one warp to work them off such groups ran on alone
// for more than half of the kernel (60,000 reads: SMs active 37% of the time).
//
// A read that reaches its end with a non-empty set has one result, the whole read.  One
// whose set empties at position j has the result [0, j) (if it is long enough) and goes on
// in k_smem, which starts behind it (SmemJobs::resume).  The set is that of the window and
// forward phases there (smem.cuh): the SA intervals of the text strings that match.
//
// With a work log every read is charged with the nodes that hold it, as if its set were extended
// for it alone: what it costs does not depend on the reads around it, unless a list outgrows its
// area (the log says so).
//
// Measured on a B200, 150 bp reads on the 100 Mbp IUPAC text, kernel times of a thread per
// read, of this sweep with a warp per group, with a block, and as it is (one warp prepares a
// position, symbols without children skipped, both kinds of nodes at a time, five blocks an SM
// where four had 124 registers): 200,000 reads by prefix 39.5 / 12.6 / 12.7 / 10.4 ms, 4,099
// reads 16.2 / 1.30 / 0.88 / 0.82 ms, 64 reads (one a block: its nodes share the threads) 10.7
// / 0.67 / 0.65 / 0.46 ms.  Bound by issue: some 400 instructions for 32 larger nodes (the 16
// masks and popcounts of two borders, then their children); 30 reads carry about 130 of those
// and as many one-row nodes a position, where one read alone carries some 35.
#pragma once
#include "smem.cuh"

namespace hfm {

constexpr uint32_t TRIE_WARPS = 4;          // warps per block
constexpr uint32_t TRIE_S1 = 640;           // one-row nodes of a list kept in shared memory
constexpr uint32_t TRIE_SB = 384;           // larger nodes kept in shared memory
constexpr uint32_t TRIE_CAP = 16384;        // nodes of one list in all
constexpr uint32_t TRIE_EMIT = 256;         // intervals of one read's set (more: k_smem takes the read)
constexpr size_t TRIE_NODE_BYTES = 4ull * TRIE_CAP * 16;   // global node area per block (two sizes, two buffers)

struct TrieShared {
  uint4 one[2][TRIE_S1];
  uint4 big[2][TRIE_SB];
  uint2 set[TRIE_WARPS][TRIE_EMIT];
  uint32_t reads[2][16];                    // reads whose code at this (the next) position matches symbol s
  // of the next list: nodes, reads that hold one.  Position j counts in [j % 3] and clears
  // the one after it, which every thread has read two barriers ago.
  uint32_t n1[3], nb[3], still[3];
  uint32_t C[16];
  uint32_t group;
  uint16_t compat[16];
};

struct TrieWork {
  uint4* nodes;                             // TRIE_NODE_BYTES per block
  unsigned int* queue;
  uint32_t group;                           // reads per block, 1..32
  uint32_t* left; uint32_t* n_left;         // reads that k_smem goes on with
  uint32_t* resume;                         // for each of them: where, or RESUME_START
  uint32_t* work_log;                       // COUNT_TOUCH only, 4 u32 per read (MemsWork), or nullptr
};

// A node list: the first SC nodes in shared memory, the others in the warp's global area.
struct NodeList {
  uint4* s; uint4* g; uint32_t sc;
  __device__ __forceinline__ uint4 get(uint32_t k) const { return k < sc ? s[k] : g[k]; }
  __device__ __forceinline__ void put(uint32_t k, const uint4& v) const { if (k < sc) s[k] = v; else g[k] = v; }
};

template <bool COUNT_TOUCH>
__global__ void __launch_bounds__(TRIE_WARPS * 32, 5) k_trie(DevFm Fw, DevFm Rv, const uint16_t* __restrict__ compat,
                                                             const uint8_t* __restrict__ q,
                                                             const uint64_t* __restrict__ qoff, MemsParams P,
                                                             Pool hitpool, MemsOut out, TrieWork W, SmemJobs J) {
  extern __shared__ __align__(16) unsigned char trie_smem[];
  TrieShared& S = *reinterpret_cast<TrieShared*>(trie_smem);
  if (threadIdx.x < 16) { S.C[threadIdx.x] = Rv.C[threadIdx.x]; S.compat[threadIdx.x] = compat[threadIdx.x] & Fw.sym_mask; }
  const uint32_t lane = threadIdx.x & 31, lt = lane_lt_mask(), warp = threadIdx.x >> 5;
  uint2* set = S.set[warp];
  uint4* g = W.nodes + (size_t)blockIdx.x * 4 * TRIE_CAP;
  const uint32_t n_reads = J.whole(), n_groups = (n_reads + W.group - 1) / W.group;
  const FmView X{Rv.occ, Rv.sb};
  uint64_t touches = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      S.group = atomicAdd(W.queue, 1u);
      S.n1[0] = S.nb[0] = S.still[0] = 0;
    }
    __syncthreads();
    const uint32_t grp = S.group;
    if (grp >= n_groups) break;
    // lane r of every warp holds read r of the group
    const uint32_t k = grp * W.group + lane;
    const bool mine = lane < W.group && k < n_reads;
    const uint32_t read = mine ? (J.ids ? J.ids[k] : k) : 0u;
    const uint64_t o = mine ? qoff[read] : 0;
    const uint32_t n = mine ? (uint32_t)(qoff[read + 1] - o) : 0u;
    const uint8_t* p = q + o;
    const uint64_t slot = mine ? (J.slot_base ? J.slot_base[read] : (uint64_t)read) : 0;
    if (mine && warp == 0) { out.hit_start[slot] = 0; out.hit_count[slot] = 0; out.pos_count[slot] = 0; }
    uint32_t alive = __ballot_sync(0xFFFFFFFFu, mine && n >= P.min_len);      // min_len >= 1 here
    uint32_t work = 0;                      // COUNT_TOUCH: this warp's touches for read `lane`
    auto charge = [&](uint32_t holds, uint32_t touch) {
      if (!W.work_log) return;
      for (uint32_t m = __reduce_or_sync(0xFFFFFFFFu, holds); m; m &= m - 1) {
        const uint32_t r = __ffs(m) - 1, b = __ballot_sync(0xFFFFFFFFu, (holds >> r) & 1);
        if (lane == r) work += touch * (uint32_t)__popc(b);
      }
    };

    // Hands the reads in `who` to k_smem: after [0, j), or from the start.
    auto leave = [&](uint32_t who, uint32_t j) {
      if (!who) return;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(W.n_left, (uint32_t)__popc(who));
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      if ((who >> lane) & 1) {
        W.left[at + __popc(who & lt)] = read;
        W.resume[at + __popc(who & lt)] = j;
        if (COUNT_TOUCH && W.work_log && j == RESUME_START) atomicOr(W.work_log + 4 * (size_t)read + 3, 1u);
      }
    };
    // The result [0, j) of the reads in `who`, a warp per read: one hit per node that holds
    // the read, ascending by forward start.  A set too large for it is left to k_smem; the
    // reads that end before their last base go on there.
    auto emit = [&](uint32_t who, uint32_t j, bool ends, const NodeList& one, uint32_t n1, const NodeList& big, uint32_t nb) {
      uint32_t later = 0, again = 0;
      for (; who; who &= who - 1) {
        const uint32_t r = __ffs(who) - 1;
        if (r % TRIE_WARPS != warp) continue;
        if (!ends) later |= 1u << r;
        if (j < P.min_len) continue;
        uint32_t cnt = 0;
        for (int kind = 0; kind < 2; kind++) {
          const NodeList& l = kind ? big : one;
          const uint32_t m = kind ? nb : n1;
          for (uint32_t b = 0; b < m; b += 32) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (b + lane < m) v = l.get(b + lane);
            const bool has = (v.w >> r) & 1;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, has), at = cnt + __popc(bal & lt);
            if (has && at < TRIE_EMIT) set[at] = make_uint2(v.x, v.z);
            cnt += __popc(bal);
          }
        }
        if (cnt > TRIE_EMIT) { again |= 1u << r; continue; }
        __syncwarp();
        uint64_t off = 0;
        if (lane == r) off = thread_reserve(hitpool, cnt);
        off = __shfl_sync(0xFFFFFFFFu, off, r);
        uint64_t hp = 0;
        if (off != ~0ull) {
          uint4* dst = (uint4*)hitpool.base + off * 2;
          for (uint32_t e = lane; e < cnt; e += 32) {
            const uint2 v = set[e];
            uint32_t rank = 0;
            for (uint32_t t = 0; t < cnt; t++) rank += set[t].x < v.x ? 1u : 0u;
            dst[2 * rank] = make_uint4(0u, j, v.y, v.y > P.max_hits ? 1u : 0u);
            const uint32_t positions = P.resolve ? min(v.y, P.max_hits) : 0u;
            dst[2 * rank + 1] = make_uint4(v.x, positions, 0u, 0u);
            hp += positions;
          }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) hp += __shfl_xor_sync(0xFFFFFFFFu, hp, d);
        if (lane == r) {
          if (off == ~0ull) atomicOr(out.status + read, (uint32_t)ST_POOL_OVF);
          else { out.hit_start[slot] = off; out.hit_count[slot] = cnt; out.pos_count[slot] = hp; }
        }
        __syncwarp();
      }
      leave(later & ~again, j);
      leave(again, RESUME_START);
    };

    uint32_t t = 0, n1 = 0, nb = 0;
    if (threadIdx.x == 0) {
      const uint4 full = make_uint4(0u, 0u, Fw.text_len, alive);
      if (Fw.text_len == 1) S.one[0][0] = full; else S.big[0][0] = full;
    }
    if (Fw.text_len == 1) n1 = 1; else nb = 1;
    // the reads whose code c matches each symbol; a read that has ended or whose set is empty
    // may keep its bits: no node has it any more, and one that ends here is taken out
    auto match_reads = [&](uint32_t code, uint32_t* to) {
      const uint32_t match = code < 16 ? S.compat[code] : 0u;
#pragma unroll
      for (int s = 0; s < 16; s++) {
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, (match >> s) & 1);
        if (lane == s) to[s] = b;
      }
    };
    if (warp == 0) match_reads(((alive >> lane) & 1) ? p[0] : 16u, S.reads[0]);
    __syncthreads();
    for (uint32_t j = 0, c = 0;; j++) {
      const NodeList one{S.one[t], g + (size_t)t * TRIE_CAP, TRIE_S1}, big{S.big[t], g + (size_t)(2 + t) * TRIE_CAP, TRIE_SB};
      const NodeList one2{S.one[t ^ 1], g + (size_t)(t ^ 1) * TRIE_CAP, TRIE_S1},
          big2{S.big[t ^ 1], g + (size_t)(2 + (t ^ 1)) * TRIE_CAP, TRIE_SB};
      const uint32_t fin = alive & __ballot_sync(0xFFFFFFFFu, n == j);
      if (fin) {
        emit(fin, j, true, one, n1, big, nb);
        alive &= ~fin;
      }
      if (!alive) break;
      const uint32_t cn = c == 2 ? 0 : c + 1;
      if (threadIdx.x == 0) { S.n1[cn] = 0; S.nb[cn] = 0; S.still[cn] = 0; }
      const uint32_t* reads = S.reads[j & 1];
      // one warp, another each time, prepares the next position
      if ((j & (TRIE_WARPS - 1)) == warp) match_reads(((alive >> lane) & 1) && j + 1 < n ? p[j + 1] : 16u, S.reads[(j + 1) & 1]);
      uint32_t still = 0;
      // larger nodes: their one-row children go to the one-row list
      for (uint32_t b = warp * 32; b < nb; b += TRIE_WARPS * 32) {
        uint32_t r[16], d[16], kids = 0, syms = 0;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (b + lane < nb) {
          v = big.get(b + lane);
          wide_split(X.occ, v.y, v.z, r, d);
          if (COUNT_TOUCH) touches += 2;
#pragma unroll
          for (int s = 1; s < 16; s++)
            if (d[s] && (v.w & reads[s])) { kids += d[s] == 1 ? 1u : 0x10000u; syms |= 1u << s; }
        }
        if (COUNT_TOUCH) charge(v.w & alive, 2);
        uint32_t total;
        const uint32_t at = warp_excl_scan(kids, total);
        uint32_t a1 = 0, ab = 0;
        if (lane == 0) {
          if (total & 0xFFFFu) a1 = atomicAdd(&S.n1[c], total & 0xFFFFu);
          if (total >> 16) ab = atomicAdd(&S.nb[c], total >> 16);
        }
        a1 = __shfl_sync(0xFFFFFFFFu, a1, 0);
        ab = __shfl_sync(0xFFFFFFFFu, ab, 0);
        if (a1 + (total & 0xFFFFu) > TRIE_CAP || ab + (total >> 16) > TRIE_CAP) break;   // the counts tell everyone
        a1 += at & 0xFFFFu; ab += at >> 16;
        const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, syms);       // half of the symbols, on average
        uint32_t run = d[0];
#pragma unroll
        for (int s = 1; s < 16; s++) {
          if ((any >> s) & 1) {
            if ((syms >> s) & 1) {
              const uint32_t who = v.w & reads[s];
              const uint4 kid = make_uint4(v.x + run, S.C[s] + r[s], d[s], who);
              if (d[s] == 1) one2.put(a1++, kid); else big2.put(ab++, kid);
              still |= who;
            }
          }
          run += d[s];
        }
      }
      // one-row nodes: one LF step each; from the last warp on, so that short lists of both
      // kinds are worked off at the same time
      for (uint32_t b = (TRIE_WARPS - 1 - warp) * 32; b < n1; b += TRIE_WARPS * 32) {
        uint4 kid = make_uint4(0, 0, 0, 0), v = kid;
        if (b + lane < n1) {
          v = one.get(b + lane);
          uint32_t s, rk;
          row_code_rank<OCC_WIDE>(X, v.y, s, rk);
          if (COUNT_TOUCH) touches += 1;
          const uint32_t who = v.w & reads[s];
          kid = make_uint4(v.x, S.C[s] + rk, 1u, who);
          still |= who;
        }
        if (COUNT_TOUCH) charge(v.w & alive, 1);
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, kid.w != 0);
        if (!bal) continue;
        uint32_t a1 = 0;
        if (lane == 0) a1 = atomicAdd(&S.n1[c], (uint32_t)__popc(bal));
        a1 = __shfl_sync(0xFFFFFFFFu, a1, 0);
        if (a1 + __popc(bal) > TRIE_CAP) break;
        if (kid.w) one2.put(a1 + __popc(bal & lt), kid);
      }
      still = __reduce_or_sync(0xFFFFFFFFu, still);
      if (lane == 0 && still) atomicOr(&S.still[c], still);
      __syncthreads();
      const uint32_t m1 = S.n1[c], mb = S.nb[c];
      if (m1 > TRIE_CAP || mb > TRIE_CAP) {
        if (warp == 0) leave(alive, RESUME_START);
        break;
      }
      still = S.still[c];
      const uint32_t dead = alive & ~still;
      if (dead) {
        emit(dead, j, false, one, n1, big, nb);
        alive = still;
        __syncthreads();                    // the next position writes where these lists are
      }
      n1 = m1; nb = mb; t ^= 1; c = cn;
    }
    if (COUNT_TOUCH && W.work_log && mine && work) atomicAdd(W.work_log + 4 * (size_t)read, work);
    __syncthreads();
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

}  // namespace hfm
