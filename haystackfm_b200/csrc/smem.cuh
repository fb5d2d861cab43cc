// smem.cuh — SMEM / MEM search, one thread per read or read segment.
//
// What is searched for.  "q[s, e) occurs in the text" (each query code matching its
// compatible text codes) holds for every part of a string that it holds for.  Let LM(e) be
// the smallest s with q[s, e) occurring.  The candidates that find_smems keeps
// (src/fm_index/smem.rs:71-222: right-maximal prefixes of every pivot's sweep, extended
// left maximally, those not contained in another) are exactly the pairs (LM(e), e) with
// e = n or LM(e + 1) > LM(e): an occurrence of such a pair that is not followed by q[e]
// makes the coverage drop at e in the sweep of every pivot inside it, so the sweep records
// it.  find_mems (smem.rs:113-124,250-295: the longest match from every start, kept when it
// does not extend left) gives the same pairs.  The interval set of a pair is the set of SA
// intervals of the text strings that match it, whatever the order it was extended in.  So
// both modes are served by one search that visits only matches of at least min_len:
//
//   window  extend left from i + min_len down to i; where the set empties at position t, no
//           match of min_len starts at or before t: go on with i = t + 1
//   forward extend right from the window while the set is not empty: q[i, e) is a result
//   next    extend left from e + 1; the set empties at t: the next result that reaches past
//           e starts at t + 1 or later
//
// A read costs about 2 min_len + its match lengths in steps; the sweep it replaces extended
// every prefix of every pivot at which the coverage drops (some 15 per pivot) left again.
// Measured on a B200, 256 Mbp ACGT repeat genome, kernel times of the sweep, of this search,
// and with the k-mer table (DevAux) and short segments for small batches: 1M reads of 150 bp
// 58.4 / 11.3 / 8.2 ms; 60,000 mixed reads up to 10 kbp 71.2 / 7.7 / 4.7 ms; 250 of them
// 37.2 / 5.2 / 0.56 ms; find_mems of 20,000 ragged reads 25.9 / 1.9 / 0.9 ms.  With records
// that count from row 32 (32-bit masks, half the popcounts): 5.9, 3.5, 0.38 and 0.70 ms.
//
// Where a window starts.  Codes of several symbols multiply a set, an N fourfold and more, until
// the codes around it have narrowed it down; a window that ended in a run of N was extended from
// that run and had 4^run intervals.  A window whose set grows like that and that holds more than
// SEED_AMBIGUOUS of them starts anew, at the end of its longest run of ACGT (seed_end), goes left
// to i and then right: where the left part empties, the same holds as above; where the right one
// does within the window, no match of min_len starts at i.  B200, 1,000 reads of 150 bp on 64 Mbp
// ACGT, the sweep / from the window's end / so, with ACGT sets of more than ACGT_SET_CAP intervals
// left to the warp kernel: 8 N at a random place 140 / 188 / 90 ms, N from 60 to 69 4.2 / 13.2 / 5.2
// s, N from 13 to 18 18.2 / 12.9 / 9.1 ms, 4 N at a random place 142 / 38 / 7.6 ms.  (Looked for in
// every window before its first step: 3 to 6% for reads with a single N, 4.7 ms for the last.)
//
// Segments.  A result belongs to the segment of a long read in which it starts.  A segment's
// search begins at its first position a: if the window there does not match, everything
// after it is left-maximal by construction; if it does, its match is a result only when it
// does not extend left by q[a - 1].  Segments need nothing from one another, so a long read
// is as many independent jobs.
//
// Execution.  All lanes of a warp run the same loop, one extension step per turn, whatever
// phase their read is in: the step takes its direction, interval and code at run time, so a
// lane that looks backwards and one that goes forward load and count together.
#pragma once
#include "search.cuh"

namespace hfm {

// The jobs of one launch: segments of long reads, then whole reads.  Counts that a
// graph-captured chain does not know on the host are read on the device.
struct SmemJobs {
  const uint32_t* unit_read;      // read of each segment
  const uint32_t* unit_k;         // its index within the read
  uint32_t seg_len;
  uint32_t n_units;
  const uint64_t* n_units_dev;
  const uint32_t* ids;            // whole reads (nullptr: 0..n_ids-1)
  uint32_t n_ids;
  const uint64_t* n_long_dev;     // when set, n_ids counts the long reads too
  const uint32_t* n_ids_dev;      // when set, the number of whole reads
  const uint32_t* jobs;           // when set, only these n_jobs jobs (of the ones above)
  uint32_t n_jobs;
  const uint32_t* n_jobs_dev;     // when set, their number
  const uint32_t* resume;         // per entry of ids: position after a result [0, e) that is already in its read's
                                  // slot (k_trie), or RESUME_START; nullptr: every read from its start
  // Results are written per slot: a read's segments in order (one slot for a read in one
  // piece).  slot_base[i] = first slot of read i; nullptr: slot i.
  const uint64_t* slot_base;
  __device__ __forceinline__ uint32_t units() const { return n_units_dev ? (uint32_t)*n_units_dev : n_units; }
  __device__ __forceinline__ uint32_t whole() const {
    return n_ids_dev ? *n_ids_dev : n_long_dev ? n_ids - (uint32_t)*n_long_dev : n_ids;
  }
};

constexpr uint32_t RESUME_START = 0xFFFFFFFFu;

// One direction of the index as the step needs it.
struct FmView { const uint4* occ; const uint32_t* sb; };

// Extends one interval of an ACGT text by one code s (1..4): rows [lo, lo + n) of the
// extended side become [lo', lo' + n'), `base` (the other side's start) moves past the rows
// of smaller codes.  The border records are those of the first and the last row, so an
// interval within 64 rows (every one-row interval) reads one sector.  Returns false, and
// changes nothing, when no row has the code.
//
// Both borders count from row 32 of their records: 4 popcounts of 32 bits (rows of code s,
// and of the codes from s on, at either border); the masks of s are two words made from its
// bits, so that one form serves every code.  acgt_use takes the first half of the lower
// border's record (at pl) from its caller.
template <bool COUNT_TOUCH>
__device__ __forceinline__ bool acgt_use(const FmView& X, const uint32_t* C, uint32_t s, const uint4& u, const uint4* pl,
                                         uint32_t& lo, uint32_t& base, uint32_t& n, uint64_t& touches) {
  const uint32_t last = lo + n - 1, bl = lo >> 6, bh = last >> 6, sh = 16u * (s - 1u);
  const uint4 v = __ldg(pl + 1);
  const uint32_t sbl = __ldg(X.sb + (size_t)(bl >> SB_BLOCK_SHIFT) * 16 + s);
  uint4 u2 = u, v2 = v;
  if (bh != bl) {
    const uint4* ph = X.occ + (size_t)bh * OCC_NARROW_U4;
    u2 = __ldg(ph); v2 = __ldg(ph + 1);
    if (COUNT_TOUCH) touches += 1;
  }
  Border<OCC_NARROW> L, H;
  L.take(u, v, lo & 63);
  H.take(u2, v2, (last & 63) + 1u);
  const uint32_t k0 = 0u - ((s - 1u) & 1u), k1 = 0u - ((s - 1u) >> 1);      // the bits of code s as masks
  auto eq = [&](const Border<OCC_NARROW>& B) { return (uint32_t)__popc(B.m & ~B.z & ~((B.b0 ^ k0) | (B.b1 ^ k1))) * B.sg; };
  auto ge = [&](const Border<OCC_NARROW>& B) {
    return (uint32_t)__popc(B.m & ~B.z & ((B.b1 & ~k1) | (~(B.b1 ^ k1) & (B.b0 | ~k0)))) * B.sg;
  };
  auto count = [&](const Border<OCC_NARROW>& B) {
    return (uint32_t)((((uint64_t)B.c34 << 32) | B.c12) >> sh) & 0xFFFFu;
  };
  const uint32_t rl = count(L) + eq(L);
  uint32_t d = count(H) + eq(H) - rl;
  // codes from s on: the records' counts differ by u16 fields that never borrow within a
  // superblock
  const uint64_t df = ((((uint64_t)H.c34 << 32) | H.c12) - (((uint64_t)L.c34 << 32) | L.c12)) >> sh;
  uint32_t g = ge(H) - ge(L);
  if ((bh >> SB_BLOCK_SHIFT) == (bl >> SB_BLOCK_SHIFT)) {
    g += (uint32_t)(df & 0xFFFFu) + (uint32_t)(df >> 16 & 0xFFFFu) + (uint32_t)(df >> 32 & 0xFFFFu) + (uint32_t)(df >> 48);
  } else {
    const uint32_t* q = X.sb + (size_t)(bl >> SB_BLOCK_SHIFT) * 16;
    const uint32_t* r = X.sb + (size_t)(bh >> SB_BLOCK_SHIFT) * 16;
    d += __ldg(r + s) - sbl;
    for (uint32_t t = s; t <= 4; t++) g += __ldg(r + t) - __ldg(q + t) + H.delta((int)t) - L.delta((int)t);
  }
  if (!d) return false;
  base += n - g;
  lo = C[s] + sbl + rl;
  n = d;
  return true;
}

template <bool COUNT_TOUCH>
__device__ __forceinline__ bool acgt_step(const FmView& X, const uint32_t* C, uint32_t s, uint32_t& lo, uint32_t& base,
                                          uint32_t& n, uint64_t& touches) {
  const uint4* pl = X.occ + (size_t)(lo >> 6) * OCC_NARROW_U4;
  const uint4 u = __ldg(pl);
  if (COUNT_TOUCH) touches += 1;
  return acgt_use<COUNT_TOUCH>(X, C, s, u, pl, lo, base, n, touches);
}

// A lane's interval set: one interval in registers, or cnt > 1 of them in `cur` (in any
// order), with `alt` as the buffer that the next step writes.
template <class SR>
struct LaneSet {
  uint32_t flo, rlo, sz, cnt;
  SR cur, alt;
};

// One extension of the whole set by the codes of `mask`, to the left or to the right
// (extend_multi_right / extend_multi_left, src/fm_index/smem.rs:332-357).  Returns false,
// and leaves the set as it was, when nothing extends (or, with ovf set, when the set
// outgrows `cap`).
template <bool COUNT_TOUCH, uint32_t FMT, class SR>
__device__ __forceinline__ bool lane_step(const FmView& X, const uint32_t* C, bool left, uint32_t mask,
                                          LaneSet<SR>& L, uint32_t cap, bool& ovf, uint64_t& touches) {
  if (FMT == OCC_NARROW && L.cnt == 1 && (mask & (mask - 1)) == 0) {
    if (!mask) return false;
    uint32_t lo = left ? L.flo : L.rlo, base = left ? L.rlo : L.flo, n = L.sz;
    if (!acgt_step<COUNT_TOUCH>(X, C, 31u - (uint32_t)__clz(mask), lo, base, n, touches)) return false;
    L.flo = left ? lo : base; L.rlo = left ? base : lo; L.sz = n;
    return true;
  }
  if (!mask) return false;
  const uint32_t top = 31u - (uint32_t)__clz(mask);
  uint32_t m = 0, f0 = 0, f1 = 0, f2 = 0;              // children; the first one stays in registers
  auto child = [&](uint32_t lo, uint32_t base, uint32_t d) {
    const uint32_t fl = left ? lo : base, rl = left ? base : lo;
    if (m == 0) { f0 = fl; f1 = rl; f2 = d; m = 1; return; }
    if (m >= cap) { ovf = true; return; }
    if (m == 1) L.alt[0] = BIv{f0, f0 + f2, f1, f1 + f2};
    L.alt[m++] = BIv{fl, fl + d, rl, rl + d};
  };
  const uint32_t cnt = L.cnt;
  for (uint32_t k = 0; k < cnt; k++) {
    uint32_t fl = L.flo, rl = L.rlo, n = L.sz;
    if (cnt > 1) { const BIv v = L.cur[k]; fl = v.flo; rl = v.rlo; n = v.fhi - v.flo; }
    const uint32_t lo = left ? fl : rl, base = left ? rl : fl;
    if (n == 1) {
      // a one-row interval extends by the code of its row alone: one LF step on one record
      uint32_t s0, rk;
      row_code_rank<FMT>(X, lo, s0, rk);
      if (COUNT_TOUCH) touches += 1;
      if ((mask >> s0) & 1) child(C[s0] + rk, base, 1u);
    } else {
      if (COUNT_TOUCH) touches += (lo != 0) + 1;
      uint32_t run = 0;
      // count_smaller_than (src/fm_index/bidir.rs:125-143): the new interval of symbol s on
      // the other strand starts after every code below s, $ included
      split_by_symbol<FMT>(X, lo, lo + n, top, [&](int s, uint32_t d, uint32_t r, uint32_t sbi) {
        if (!ovf && ((mask >> s) & 1) && d)
          child(C[s] + (FMT == OCC_WIDE ? r : sb_count(X, sbi, s) + r), base + run, d);
        run += d;
      });
    }
    if (ovf) return false;
  }
  if (m == 0) return false;
  if (m == 1) { L.flo = f0; L.rlo = f1; L.sz = f2; }
  else { const SR t = L.cur; L.cur = L.alt; L.alt = t; }
  L.cnt = m;
  return true;
}

// Shell sort of an interval set by its forward start (hits of one MEM ascend by it).
template <class SR>
__device__ __forceinline__ void sort_set(const SR& a, uint32_t n) {
  for (uint32_t gap = n / 2; gap > 0; gap /= 2)
    for (uint32_t i = gap; i < n; i++) {
      const BIv t = a[i];
      uint32_t j = i;
      while (j >= gap) {
        const BIv v = a[j - gap];
        if (v.flo <= t.flo) break;
        a[j] = v;
        j -= gap;
      }
      a[j] = t;
    }
}

// Sets that a thread extends on ACGT texts: they have several intervals only behind codes of
// several symbols, in few reads of a batch, and a thread takes them one at a time where the warp
// kernel takes 32.  (64 reads of 150 bp with 4 N, 256 intervals: a thread each 30 ms, a warp 3.0.)
constexpr uint32_t ACGT_SET_CAP = 96;
static_assert(ACGT_SET_CAP <= FAST_SET_CAP, "the sets' areas");

// Persistent search.  KC > 0: hit lists of KC entries in local memory; KC = 0: W.hit_cap
// entries per thread in global memory.  A job that outgrows its sets or its list is queued
// for a later tier (out.ovf_list, once per read).
template <bool COUNT_TOUCH, int STRIDE, int KC, int MINB, uint32_t FMT>
__global__ void __launch_bounds__(128, MINB) k_smem(DevFm Fw, DevFm Rv, const uint16_t* __restrict__ compat_fw,
                                                   const uint16_t* __restrict__ compat_rv,
                                                   const uint8_t* __restrict__ q, const uint64_t* __restrict__ qoff,
                                                   MemsParams P, Pool hitpool, MemsOut out, MemsWork W, SmemJobs J,
                                                   DevAux A) {
  __shared__ SmemFm Sf, Sr;
  smem_fm_init(Sf, Fw, compat_fw);
  smem_fm_init(Sr, Rv, compat_rv);
  __syncthreads();
  // a window's set from which on its seed_end is looked for: three codes of several symbols and
  // more, on texts with such codes more than the usual set
  constexpr uint32_t SEED_SET = FMT == OCC_NARROW ? 16 : 128;
  const uint32_t SCAP = FMT == OCC_NARROW ? ACGT_SET_CAP : STRIDE == 32 ? FAST_SET_CAP : W.set_cap;
  using SR = SetRef<BIv, STRIDE>;
  LaneSet<SR> L;
  L.cur = thread_set<BIv, STRIDE>(W.sets, SCAP, 2, 0);
  L.alt = thread_set<BIv, STRIDE>(W.sets, SCAP, 2, 1);
  uint4 local_h[KC > 0 ? 2 * KC : 1];
  uint4* hits = local_h;
  uint32_t hit_cap = KC;
  if (KC == 0) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    hits = W.hits + tid * W.hit_cap * 2;
    hit_cap = W.hit_cap;
  }
  enum : uint32_t { FETCH, WINDOW, BACK, FORWARD, NEXT_START, NEXT, LEFT_MAX, DONE };
  const uint32_t n_units = J.units(), chunk = W.step(), min_len = P.min_len;
  const uint32_t n_jobs = !J.jobs ? n_units + J.whole() : J.n_jobs_dev ? *J.n_jobs_dev : J.n_jobs;
  const uint32_t sym = Fw.sym_mask;
  QueueCursor qc;
  uint64_t touches = 0, t0 = 0;
  uint32_t ph = FETCH, u = 0, read = 0, st = ST_OK;
  uint32_t n = 0, i = 0, stop = 0, pos = 0, end = 0, nh = 0;
  bool first = false;                     // the left-maximality of i is not known yet
  bool looked = false;                    // BACK: seed_end of this window has been looked for
  const uint8_t* p = q;
  for (;;) {
    if (ph == FETCH) {
      if (!next_read_chunked(W.queue, n_jobs, J.jobs, chunk, qc, u)) break;
      const bool unit = u < n_units;
      read = unit ? J.unit_read[u] : J.ids ? J.ids[u - n_units] : u - n_units;
      const uint64_t o = qoff[read];
      n = (uint32_t)(qoff[read + 1] - o);
      p = q + o;
      i = unit ? J.unit_k[u] * J.seg_len : 0u;
      stop = unit ? min(n, i + J.seg_len) : n;
      first = i > 0;
      nh = 0; st = ST_OK; t0 = touches;
      ph = WINDOW;
      if (!unit && J.resume && J.resume[u - n_units] != RESUME_START) {
        // behind a first result that is already known: its hits lead this read's list
        end = J.resume[u - n_units];
        const uint64_t slot = J.slot_base ? J.slot_base[read] : (uint64_t)read;
        const uint4* src = (const uint4*)hitpool.base + out.hit_start[slot] * 2;
        const uint32_t have = out.hit_count[slot];
        if (have > hit_cap) { st |= ST_CAND_OVF; ph = DONE; }
        else {
          for (uint32_t k = 0; k < 2 * have; k++) hits[k] = src[k];
          nh = have;
          if (end == 0) i = 1;
          else ph = NEXT_START;
        }
      }
    }
    if (ph == WINDOW && (min_len == 0 || i >= stop || n - i < min_len)) ph = DONE;
    if (ph == WINDOW || ph == NEXT_START) {
      // start from the whole text, or from the last k codes at once (k <= min_len): where
      // they do not occur, no result reaches past them from before the second of them
      const bool window = ph == WINDOW;
      L.flo = 0; L.rlo = 0; L.sz = Fw.text_len; L.cnt = 1;
      if (window) { end = i + min_len; looked = false; }
      pos = window ? end - 1 : end;
      ph = window ? BACK : NEXT;
      if (FMT == OCC_NARROW && A.kmer && A.k <= min_len) {
        uint32_t b0 = 0, b1 = 0, bad = 0;
        const uint8_t* b = p + pos + 1 - A.k;
        for (uint32_t k = 0; k < A.k; k++) { const uint32_t c = b[k] - 1u; bad |= c; b0 |= (c & 1u) << k; b1 |= (c >> 1 & 1u) << k; }
        if (bad < 4) {
          const uint4 v = __ldg(A.kmer + (b1 << A.k | b0));
          if (COUNT_TOUCH) touches += 1;
          const uint32_t at = pos + 1 - A.k;               // its first code
          if (!v.z) { i = at + 1; first = false; ph = WINDOW; continue; }
          L.flo = v.x; L.rlo = v.y; L.sz = v.z;
          if (at > i) pos = at - 1;
          else { pos = end; ph = FORWARD; }                // k == min_len: the window is matched
        }
      }
    }
    bool matched = false;                 // q[i, end) is a longest match from i
    if (ph == FORWARD && pos == n) { end = n; matched = true; }
    if (ph != DONE && !matched) {
      const bool left = ph != FORWARD;
      const FmView X{left ? Fw.occ : Rv.occ, left ? Fw.sb : Rv.sb};
      const uint8_t code = p[pos];
      const uint32_t mask = code < 16 ? (uint32_t)Sf.compat_mask[code] & sym : 0u;
      bool ovf = false;
      const bool ok = lane_step<COUNT_TOUCH, FMT>(X, left ? Sf.C : Sr.C, left, mask, L, SCAP, ovf, touches);
      if (ovf) { st |= ST_SET_OVF; ph = DONE; }
      else if (ph == BACK) {
        if (!ok) { i = pos + 1; first = false; ph = WINDOW; }
        else if (pos > i) {
          pos--;
          if (L.cnt > SEED_SET && !looked) {
            looked = true;
            const uint32_t at = seed_end(Sf.compat_mask, p, i, end);
            if (at < end) { end = at; pos = at - 1; L.flo = 0; L.rlo = 0; L.sz = Fw.text_len; L.cnt = 1; }
          }
        } else {
          pos = end;                      // of q[i, end) so far: the window, or up to its seed_end
          ph = FORWARD;
          if (pos == n) matched = true;
        }
      } else if (ph == FORWARD) {
        if (ok) pos++;
        if (!ok && pos < i + min_len) { i = i + 1; first = false; ph = WINDOW; }   // the window at i does not match
        else if (!ok || pos == n) { end = pos; matched = true; }
      } else if (ph == NEXT) {
        if (!ok) { i = pos + 1; ph = WINDOW; }
        else if (pos <= i + 1) { i = i + 1; ph = WINDOW; }      // q[i, end] is known not to match
        else pos--;
      } else {                                                  // LEFT_MAX: the set is still that of q[i, end)
        first = false;
        if (ok) ph = end == n ? DONE : NEXT_START;
        else matched = true;
      }
    }
    if (matched && first) { ph = LEFT_MAX; pos = i - 1; matched = false; }
    if (matched) {
      // one hit per interval of the set, ascending by forward start
      if (nh + L.cnt > hit_cap) { st |= ST_CAND_OVF; ph = DONE; }
      else {
        if (L.cnt > 1) sort_set(L.cur, L.cnt);
        for (uint32_t k = 0; k < L.cnt; k++) {
          uint32_t fl = L.flo, sz = L.sz;
          if (L.cnt > 1) { const BIv v = L.cur[k]; fl = v.flo; sz = v.fhi - v.flo; }
          hits[2 * (nh + k)] = make_uint4(i, end, sz, sz > P.max_hits ? 1u : 0u);
          hits[2 * (nh + k) + 1] = make_uint4(fl, P.resolve ? min(sz, P.max_hits) : 0u, 0u, 0u);
        }
        nh += L.cnt;
        ph = end == n ? DONE : NEXT_START;
      }
    }
    if (ph == DONE) {
      uint64_t hs = 0, hp = 0;
      if (st) nh = 0;
      if (nh) {
        hs = thread_reserve(hitpool, nh);
        if (hs == ~0ull) { st |= ST_POOL_OVF; hs = 0; nh = 0; }
        else {
          uint4* dst = (uint4*)hitpool.base + hs * 2;
          for (uint32_t k = 0; k < 2 * nh; k++) { const uint4 v = hits[k]; dst[k] = v; if (k & 1) hp += v.y; }
        }
      }
      const bool unit = u < n_units;
      const uint64_t slot = (J.slot_base ? J.slot_base[read] : (uint64_t)read) + (unit ? J.unit_k[u] : 0u);
      out.hit_start[slot] = hs; out.hit_count[slot] = nh; out.pos_count[slot] = hp;
      if (!unit && J.slot_base)
        for (uint64_t k = slot + 1; k < J.slot_base[read + 1]; k++) { out.hit_count[k] = 0; out.pos_count[k] = 0; }
      if (COUNT_TOUCH && W.work_log) {
        atomicAdd(W.work_log + 4 * (size_t)read, (uint32_t)(touches - t0));
        if (st & (ST_SET_OVF | ST_CAND_OVF)) atomicOr(W.work_log + 4 * (size_t)read + 3, 1u);
      }
      if (st) {
        const uint32_t before = atomicOr(out.status + read, st);
        const uint32_t tier = ST_SET_OVF | ST_CAND_OVF;
        if ((st & tier) && !(before & tier)) out.ovf_list[atomicAdd(out.n_ovf, 1u)] = read;
      }
      ph = FETCH;
    }
  }
  if (COUNT_TOUCH && touches) atomicAdd(out.touches, (unsigned long long)touches);
}

// ---- DevAux, made when an index is loaded --------------------------------------------

// One more code in front: out[c w] from in[w] for strings w of k codes (in: nullptr for k = 0);
// strings are numbered with their first code in the top digit, in the last level as DevAux has
// them.  *bad counts intervals past the last row, which records that no text gives (a layout
// blob's are not checked) may lead to: they are not gone on with.
__global__ void k_kmer_table(DevFm Fw, const uint4* __restrict__ in, uint32_t k, bool last, uint4* __restrict__ out,
                             uint32_t* __restrict__ bad) {
  const uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >> (2 * (k + 1))) return;
  const uint32_t s = (uint32_t)(x >> (2 * k)) + 1u;
  uint4 v = in ? in[x & ((1ull << (2 * k)) - 1ull)] : make_uint4(0u, 0u, Fw.text_len, 0u);
  uint32_t C[5];
  for (int c = 0; c < 5; c++) C[c] = Fw.C[c];
  uint64_t touches = 0;
  const FmView X{Fw.occ, Fw.sb};
  if (v.z && !acgt_step<false>(X, C, s, v.x, v.y, v.z, touches)) v = make_uint4(0u, 0u, 0u, 0u);
  if ((uint64_t)v.x + v.z > Fw.text_len || (uint64_t)v.y + v.z > Fw.text_len) {
    atomicAdd(bad, 1u);
    v = make_uint4(0u, 0u, 0u, 0u);
  }
  uint64_t at = x;
  if (last) {
    uint32_t b0 = 0, b1 = 0;
    for (uint32_t t = 0; t <= k; t++) {
      const uint32_t d = (uint32_t)(x >> (2 * (k - t))) & 3u;
      b0 |= (d & 1u) << t; b1 |= (d >> 1) << t;
    }
    at = (uint64_t)b1 << (k + 1) | b0;
  }
  out[at] = v;
}

}  // namespace hfm
