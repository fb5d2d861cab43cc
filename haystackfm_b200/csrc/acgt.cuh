// acgt.cuh — SMEM / MEM search of ACGT texts: a packing pass, then one thread per read or
// read segment.
//
// The search of smem.cuh (window, forward, next) for reads whose codes match at most one
// symbol of the text: a set is then one interval, held in registers.  A job that meets a code
// with several symbols (IUPAC queries) is left to k_smem.
//
// Anchors.  A window of min_len codes holds exactly one of the strings of seen_k codes that
// start at multiples of min_len - seen_k + 1.  k_acgt_pack looks every such anchor of the
// batch up in the bits of the strings that occur in the text (A.seen), converged and with all
// loads independent; where an anchor does not occur, neither does any window around it.  So
// stretches that match nowhere (a read of the other strand is one) are passed without a load:
// the search goes from one anchor that occurs to the next.  The same pass turns the codes into
// bit planes (a ballot per 32 codes), which the table, the steps and the comparison take.
//
// One load a turn.  A read's search is a chain of dependent loads: records (a step), table
// entries, positions, text.  All lanes of a warp go through the same turn, whatever their
// phase: each forms its address, one load serves them all, then each phase uses what came.
// What needs no long load (a result, the end of a read, the next one, the next window) is
// done between turns once SIDE_LANES lanes wait for it, or when no lane has a load to make:
// for one or two lanes at a time it would fill most turns.
//
// One-row matches.  A one-row interval extends as long as the text at its position goes on
// like the read, and its forward row stays the same.  With the whole suffix array and the
// text on the device the rest of the match is one look at each instead of one dependent
// record per code: up to 32 codes are compared at a time.
//
// Few lanes for small batches.  A turn costs the code of every phase that some lane is in, so
// a batch that does not fill the resident threads runs `lanes` jobs a warp on all warps.
//
// Bound by the instructions of a turn (some 540 with 32 lanes in all phases) and, for large
// batches, by the longest reads at the end.  Measured on a B200, 256 Mbp ACGT repeats, search
// kernels of k_smem (steps for everything) and of this file: 1M reads of 150 bp 5.9 -> 4.0 ms
// (0.55 of it the packing pass), 60,000 mixed reads up to 10 kbp 3.5 -> 1.9, 250 of them 0.38
// -> 0.21, find_mems of 20,000 ragged reads 0.70 -> 0.51.  Without the text, 1M reads take 4.4
// ms; without anchors and probes 4.3; side work as it comes up (6 lanes) 4.4.
#pragma once
#include "smem.cuh"

namespace hfm {

constexpr int SIDE_LANES = 16;              // lanes (of 32) that wait for side work before it is done
// Steps past the window after which a one-row match is compared with the text, and the codes
// that must be left for that: the two dependent loads are worth a few steps.
constexpr uint32_t TEXT_AFTER = 2, TEXT_LEFT = 12;

// A batch as k_acgt_pack lays it out.  Word w of read r is at words[(o_r - o_0) / 32 + r + w]
// (o: code offsets; no two reads share one): bit planes of 32 codes, the bits of symbol - 1,
// codes that match no symbol (and the places past the read's end), codes that match several.
// Anchor j of read r is bit j % 32 of anchors[(o_r - o_0) / (32 * stride) + r + j / 32].
struct PackedReads {
  uint4* words;
  uint32_t* anchors;
  uint32_t seen_k, stride;                  // 0: no anchors (every window is searched)
};

// A warp per job (segment or whole read): its words, and the bits of the anchors that start
// in it (anchors is zeroed by the caller).
template <bool COUNT_TOUCH>
__global__ void __launch_bounds__(256) k_acgt_pack(const uint16_t* __restrict__ compat, uint32_t sym_mask,
                                                  const uint8_t* __restrict__ q, const uint64_t* __restrict__ qoff,
                                                  SmemJobs J, DevAux A, PackedReads R, unsigned long long* touches) {
  __shared__ uint8_t s_sym[256];
  sym_table_init(s_sym, compat, sym_mask);
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, n_units = J.units(), n_jobs = n_units + J.whole();
  const uint64_t first_off = qoff[0];
  uint32_t looked = 0;
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n_jobs; u += (gridDim.x * blockDim.x) >> 5) {
    const bool unit = u < n_units;
    const uint32_t read = unit ? J.unit_read[u] : J.ids ? J.ids[u - n_units] : u - n_units;
    const uint64_t o = qoff[read];
    const uint32_t n = (uint32_t)(qoff[read + 1] - o);
    const uint8_t* p = q + o;
    const uint32_t from = unit ? J.unit_k[u] * J.seg_len : 0u, to = unit ? min(n, from + J.seg_len) : n;
    uint4* words = R.words + ((o - first_off) / 32 + read);
    uint32_t* anchors = R.stride ? R.anchors + ((o - first_off) / (32ull * R.stride) + read) : nullptr;
    // 32 words at a time, lane w holding word w; an anchor needs the word after its own too
    for (uint32_t at = from; at < to; at += 31 * 32) {
      uint4 mine = make_uint4(0, 0, ~0u, 0);
      const uint32_t have = min(32u, (n - at + 31) / 32);
      for (uint32_t w = 0; w < have; w += 4) {              // four loads in flight
        uint32_t sym[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t t = at + (w + k) * 32 + lane;
          sym[k] = t < n ? s_sym[p[t]] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t c = sym[k] - 1u;
          const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, sym[k] && (c & 1)), b1 = __ballot_sync(0xFFFFFFFFu, sym[k] && (c & 2)),
                         none = __ballot_sync(0xFFFFFFFFu, sym[k] == 0), many = __ballot_sync(0xFFFFFFFFu, sym[k] == SYM_MANY);
          if (lane == w + k) mine = make_uint4(b0, b1, none, many);
        }
      }
      const uint32_t end = min(to, at + 31 * 32);           // the part of this turn
      if (lane < (end - at + 31) / 32) words[at / 32 + lane] = mine;
      if (!R.stride || n < R.seen_k) continue;
      const uint32_t j0 = (at + R.stride - 1) / R.stride, j1 = (min(end, n - R.seen_k + 1) + R.stride - 1) / R.stride;
      for (uint32_t jw = j0 / 32; jw * 32 < j1; jw++) {
        const uint32_t j = jw * 32 + lane, pos = j * R.stride - at;
        const bool on = j >= j0 && j < j1;
        const uint32_t w = on ? pos >> 5 : 0u, sh = pos & 31;
        const uint32_t b0 = __funnelshift_r(__shfl_sync(0xFFFFFFFFu, mine.x, w), __shfl_sync(0xFFFFFFFFu, mine.x, (w + 1) & 31), sh);
        const uint32_t b1 = __funnelshift_r(__shfl_sync(0xFFFFFFFFu, mine.y, w), __shfl_sync(0xFFFFFFFFu, mine.y, (w + 1) & 31), sh);
        const uint32_t no = __funnelshift_r(__shfl_sync(0xFFFFFFFFu, mine.z, w), __shfl_sync(0xFFFFFFFFu, mine.z, (w + 1) & 31), sh);
        const uint32_t mn = __funnelshift_r(__shfl_sync(0xFFFFFFFFu, mine.w, w), __shfl_sync(0xFFFFFFFFu, mine.w, (w + 1) & 31), sh);
        const uint32_t part = (1u << R.seen_k) - 1u;
        bool occurs = false;
        if (on && !(no & part)) {
          if (mn & part) occurs = true;                     // not known: searched
          else {
            const uint64_t key = plane_key(b0, b1, R.seen_k);
            occurs = (__ldg(A.seen + (key >> 5)) >> (key & 31)) & 1;
            if (COUNT_TOUCH) looked++;
          }
        }
        const uint32_t bits = __ballot_sync(0xFFFFFFFFu, occurs);
        if (lane == 0 && bits) atomicOr(anchors + jw, bits);
      }
    }
  }
  if (COUNT_TOUCH && looked) atomicAdd(touches, (unsigned long long)looked);
}

template <bool COUNT_TOUCH, int KC, int MINB>
__global__ void __launch_bounds__(128, MINB) k_acgt(DevFm Fw, DevFm Rv, const uint64_t* __restrict__ qoff, MemsParams P,
                                                   Pool hitpool, MemsOut out, MemsWork W, SmemJobs J, DevAux A,
                                                   PackedReads R, uint32_t lanes, uint32_t* __restrict__ left_jobs,
                                                   uint32_t* __restrict__ n_left) {
  __shared__ uint32_t s_C[2][8];            // of the reverse and of the forward index: the same in an index of one text
  if (threadIdx.x < 5) { s_C[0][threadIdx.x] = Rv.C[threadIdx.x]; s_C[1][threadIdx.x] = Fw.C[threadIdx.x]; }
  __syncthreads();
  uint4 local_h[KC > 0 ? 2 * KC : 1];
  uint4* hits = local_h;
  uint32_t hit_cap = KC;
  if (KC == 0) {
    // a list for each lane that takes jobs
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    hits = W.hits + (warp * lanes + min(threadIdx.x & 31, lanes - 1)) * W.hit_cap * 2;
    hit_cap = W.hit_cap;
  }
  // BACK .. LEFT_MAX take a step; SEEN, KMER, PLACE and TEXT make another load; the others wait
  // for side work
  enum : uint32_t { BACK, FORWARD, NEXT, LEFT_MAX, SEEN, KMER, PLACE, TEXT, RESULT, DONE, FETCH, WINDOW, NEXT_START, GONE };
  constexpr uint32_t ST_LEAVE = 0x80000000u;
  const uint32_t n_units = J.units(), n_jobs = n_units + J.whole(), chunk = W.step(), min_len = P.min_len;
  const uint32_t k_len = A.kmer && A.k <= min_len ? A.k : 0u;
  const uint64_t first_off = qoff[0];
  QueueCursor qc;
  uint64_t touches = 0, t0 = 0;
  uint32_t ph = (threadIdx.x & 31) < lanes ? FETCH : GONE, u = 0, read = 0, st = ST_OK;
  const int side_lanes = lanes < 32 ? max(1, (int)lanes * SIDE_LANES / 32) : SIDE_LANES;
  uint32_t n = 0, i = 0, stop = 0, pos = 0, end = 0, nh = 0;
  uint32_t flo = 0, rlo = 0, sz = 0;
  bool first = false;                       // the left-maximality of i is not known yet
  bool next = false;                        // SEEN and KMER: of a NEXT_START, not of a window
  const uint4* words = nullptr;
  const uint32_t* anchors = nullptr;
  for (;;) {
    const uint32_t gone = __ballot_sync(0xFFFFFFFFu, ph == GONE);
    if (gone == 0xFFFFFFFFu) break;
    const uint32_t wait = __ballot_sync(0xFFFFFFFFu, ph > TEXT && ph != GONE);
    if (__popc(wait) >= side_lanes || (wait | gone) == 0xFFFFFFFFu) {
      if (ph == RESULT) {
        // q[i, end) is a longest match from i: a result unless it extends left
        if (first) { ph = LEFT_MAX; pos = i - 1; }
        else if (nh >= hit_cap) { st |= ST_CAND_OVF; ph = DONE; }
        else {
          hits[2 * nh] = make_uint4(i, end, sz, sz > P.max_hits ? 1u : 0u);
          hits[2 * nh + 1] = make_uint4(flo, P.resolve ? min(sz, P.max_hits) : 0u, 0u, 0u);
          nh++;
          ph = end == n ? DONE : NEXT_START;
        }
      }
      if (ph == DONE) {
        const bool unit = u < n_units;
        const uint64_t slot = (J.slot_base ? J.slot_base[read] : (uint64_t)read) + (unit ? J.unit_k[u] : 0u);
        uint64_t hs = 0, hp = 0;
        if (st) nh = 0;
        if (nh) {
          hs = thread_reserve(hitpool, nh);
          if (hs == ~0ull) { st |= ST_POOL_OVF; hs = 0; nh = 0; }
          else {
            uint4* dst = (uint4*)hitpool.base + hs * 2;
#pragma unroll 1
            for (uint32_t k = 0; k < nh; k++) {
              const uint4 v = hits[2 * k + 1];
              dst[2 * k] = hits[2 * k]; dst[2 * k + 1] = v;
              hp += v.y;
            }
          }
        }
        out.hit_start[slot] = hs; out.hit_count[slot] = nh; out.pos_count[slot] = hp;
        if (st == ST_LEAVE) {
          left_jobs[atomicAdd(n_left, 1u)] = u;
        } else {
          if (COUNT_TOUCH && W.work_log) {
            atomicAdd(W.work_log + 4 * (size_t)read, (uint32_t)(touches - t0));
            if (st & ST_CAND_OVF) atomicOr(W.work_log + 4 * (size_t)read + 3, 1u);
          }
          if (st) {
            const uint32_t before = atomicOr(out.status + read, st);
            if ((st & ST_CAND_OVF) && !(before & (ST_SET_OVF | ST_CAND_OVF))) out.ovf_list[atomicAdd(out.n_ovf, 1u)] = read;
          }
        }
        ph = FETCH;
      }
      if (ph == FETCH) {
        if (!next_read_chunked(W.queue, n_jobs, nullptr, chunk, qc, u)) ph = GONE;
        else {
          const bool unit = u < n_units;
          read = unit ? J.unit_read[u] : J.ids ? J.ids[u - n_units] : u - n_units;
          const uint64_t o = qoff[read];
          n = (uint32_t)(qoff[read + 1] - o);
          words = R.words + ((o - first_off) / 32 + read);
          if (R.stride) anchors = R.anchors + ((o - first_off) / (32ull * R.stride) + read);
          i = unit ? J.unit_k[u] * J.seg_len : 0u;
          stop = unit ? min(n, i + J.seg_len) : n;
          first = i > 0;
          nh = 0; st = ST_OK; t0 = touches;
          if (COUNT_TOUCH) touches += 1;
          ph = WINDOW;
        }
      }
      if (ph == WINDOW && min_len && R.stride && i < stop && n - i >= min_len) {
        // to the next window whose anchor occurs
        uint32_t j = (i + R.stride - 1) / R.stride;
        const uint32_t j_was = j, w_end = (n - R.seen_k) / R.stride / 32;
        uint32_t w = j >> 5, bits = __ldg(anchors + w) & (~0u << (j & 31));
        while (!bits && w < w_end) bits = __ldg(anchors + ++w);
        if (!bits) i = n;
        else {
          j = w * 32 + __ffs(bits) - 1;
          if (j != j_was) { i = (j - 1) * R.stride + 1; first = false; }
        }
      }
      if (ph == WINDOW && (min_len == 0 || i >= stop || n - i < min_len)) ph = DONE;
      if (ph == WINDOW || ph == NEXT_START) {
        next = ph == NEXT_START;
        pos = next ? end : i + min_len - 1;
        flo = 0; rlo = 0; sz = Fw.text_len;
        // the window's last seen_k codes (an anchor of its own one time in `stride`), or those
        // that end where the last match ends
        ph = R.stride ? SEEN : k_len ? KMER : next ? NEXT : BACK;
      }
    }
    // one load for every lane that has one to make
    if (ph > TEXT) continue;
    const bool stepping = ph <= LEFT_MAX, left = ph != FORWARD;
    const FmView X{left ? Fw.occ : Rv.occ, left ? Fw.sb : Rv.sb};
    uint32_t lo = left ? flo : rlo, base = left ? rlo : flo;
    const uint4 r = __ldg(words + (pos >> 5));
    const uint4* a = X.occ + (size_t)(lo >> 6) * OCC_NARROW_U4;
    const uint32_t str_len = ph == SEEN ? R.seen_k : k_len, at = pos + 1 - str_len;   // SEEN, KMER: the string that ends at pos
    uint64_t key = 0;
    if (ph == SEEN || ph == KMER) {
      const uint4 r0 = __ldg(words + (at >> 5));
      const uint32_t sh = at & 31, part = (1u << str_len) - 1u;
      const bool two = (at >> 5) != (pos >> 5);
      const uint32_t b0 = two ? __funnelshift_r(r0.x, r.x, sh) : r.x >> sh, b1 = two ? __funnelshift_r(r0.y, r.y, sh) : r.y >> sh;
      const uint32_t odd = two ? __funnelshift_r(r0.z | r0.w, r.z | r.w, sh) : (r.z | r.w) >> sh;
      key = plane_key(b0, b1, str_len);
      a = ph == SEEN ? reinterpret_cast<const uint4*>(A.seen) + (key >> 7) : A.kmer + key;
      if (odd & part) {                                        // a code without a symbol, or with several: by steps
        ph = ph == SEEN && k_len ? KMER : next ? NEXT : BACK;
        continue;
      }
    } else if (ph == PLACE) {
      a = reinterpret_cast<const uint4*>(A.sa) + (flo >> 2);
    } else if (ph == TEXT) {
      a = A.text + ((rlo + pos) >> 5);                         // rlo: text position of code 0 (may wrap below 0)
    }
    const uint4 va = __ldg(a);
    if (COUNT_TOUCH) touches += 1;
    if (stepping) {
      const uint32_t b = pos & 31;
      bool ok = false;
      if ((r.w >> b) & 1) { st = ST_LEAVE; ph = DONE; continue; }
      if (!((r.z >> b) & 1)) {
        ok = acgt_use<COUNT_TOUCH>(X, s_C[left], 1u + ((r.x >> b) & 1) + 2u * ((r.y >> b) & 1), va, a, lo, base, sz, touches);
        if (ok) { flo = left ? lo : base; rlo = left ? base : lo; }
      }
      if (ph == BACK) {
        if (!ok) { i = pos + 1; first = false; ph = WINDOW; }
        else if (pos > i) pos--;
        else {
          pos = i + min_len;
          end = n;
          ph = pos == n ? RESULT : FORWARD;
        }
      } else if (ph == FORWARD) {
        if (ok) pos++;
        if (!ok || pos == n) { end = pos; ph = RESULT; }
        else if (A.text && sz == 1 && pos - i >= min_len + TEXT_AFTER && n - pos >= TEXT_LEFT) ph = PLACE;
      } else if (ph == NEXT) {
        if (!ok) { i = pos + 1; ph = WINDOW; }
        else if (pos <= i + 1) { i = i + 1; ph = WINDOW; }     // q[i, end] is known not to match
        else pos--;
      } else {                                                 // LEFT_MAX
        first = false;
        ph = !ok ? RESULT : end == n ? DONE : NEXT_START;
      }
    } else if (ph == SEEN) {
      // where the string occurs nowhere, no result reaches past it from before its second code
      if ((sel4(va, (uint32_t)(key >> 5) & 3u) >> (key & 31)) & 1) ph = k_len ? KMER : next ? NEXT : BACK;
      else { i = at + 1; first = false; ph = WINDOW; }
    } else if (ph == KMER) {
      if (!va.z) { i = at + 1; first = false; ph = WINDOW; }
      else {
        flo = va.x; rlo = va.y; sz = va.z;
        if (at > i) { pos = at - 1; ph = next ? NEXT : BACK; }
        else {                                                 // k == min_len: the window is matched
          pos = i + min_len;
          end = n;
          ph = pos == n ? RESULT : FORWARD;
        }
      }
    } else if (ph == PLACE) {
      // Directions of an index that disagree give rows whose text ends before the match does:
      // nothing matches at the end.  Further words are compared only when this one is the same,
      // so its codes are in front of the end.
      rlo = min(sel4(va, flo & 3u) - i + pos, Fw.text_len) - pos;
      ph = TEXT;
    } else {
      // the codes of this word against the text
      const uint4 vb = __ldg(a + 1);
      const uint32_t b = pos & 31, sh = (rlo + pos) & 31;
      const uint32_t x0 = __funnelshift_r(va.x, vb.x, sh) ^ (r.x >> b), x1 = __funnelshift_r(va.y, vb.y, sh) ^ (r.y >> b);
      const uint32_t diff = (x0 | x1 | __funnelshift_r(va.z, vb.z, sh) | (r.z | r.w) >> b) & (~0u >> b);
      const uint32_t same = diff ? (uint32_t)__ffs(diff) - 1u : 32u - b;
      pos = min(n, pos + same);
      if (pos == n || diff) {
        const uint32_t c = b + same;
        end = pos;
        ph = RESULT;
        if (pos < n && ((r.w >> c) & 1)) { st = ST_LEAVE; ph = DONE; }
      }
    }
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

// ---- what the search keeps besides the records (DevAux), made when an index is loaded ----

// The text, one code a byte, from the BWT and the whole suffix array; *unknown counts rows
// without a position.  Every byte is TEXT_NONE before: one that stays so (two rows claim
// another position) shows samples that belong to no text.
constexpr uint8_t TEXT_NONE = 0xFF;
__global__ void k_text_bytes(DevFm F, const uint32_t* __restrict__ sa, uint8_t* __restrict__ text,
                             uint32_t* __restrict__ unknown) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < F.text_len; r += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = sa[r];
    if (v == 0xFFFFFFFFu || v >= F.text_len) { atomicAdd(unknown, 1u); continue; }
    uint32_t c, rk;
    row_code_rank<OCC_NARROW>(F, (uint32_t)r, c, rk);
    if (v == 0 && c) atomicAdd(unknown, 1u);
    text[v > 0 ? v - 1 : F.text_len - 1] = (uint8_t)c;
  }
}

// Bit planes of 32 codes a word: the bits of symbol - 1, then the sentinels (and the places
// from n on).  *unknown counts bytes that are TEXT_NONE.
__global__ void k_text_planes(const uint8_t* __restrict__ text, uint64_t n, uint64_t words, uint4* __restrict__ out,
                              uint32_t* __restrict__ unknown) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w < words; w += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint64_t t = w * 32 + lane;
    const uint32_t c = t < n ? text[t] : 0u;
    if (c == TEXT_NONE) atomicAdd(unknown, 1u);
    const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, c && ((c - 1) & 1)), b1 = __ballot_sync(0xFFFFFFFFu, c && ((c - 1) & 2)),
                   z = __ballot_sync(0xFFFFFFFFu, c == 0);
    if (lane == 0) out[w] = make_uint4(b0, b1, z, 0u);
  }
}

// A bit for every string of k codes that occurs in the text (plane_key; k < 32).
__global__ void k_seen_bits(const uint8_t* __restrict__ text, uint32_t n, uint32_t k, uint32_t* __restrict__ seen) {
  const uint64_t from = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 32;
  uint32_t b0 = 0, b1 = 0, run = 0;
  for (uint64_t t = from; t < n && t < from + 32 + k - 1; t++) {       // strings that start in [from, from + 32)
    const uint32_t c = text[t] - 1u;
    run = c < 4 ? run + 1 : 0;
    b0 = b0 >> 1 | (c & 1u) << (k - 1);
    b1 = b1 >> 1 | (c >> 1 & 1u) << (k - 1);
    if (run >= k) {
      const uint64_t key = plane_key(b0, b1, k);
      const uint32_t bit = 1u << (key & 31);
      if (!(seen[key >> 5] & bit)) atomicOr(seen + (key >> 5), bit);
    }
  }
}

}  // namespace hfm
