// hfm_internal.h — host-side declarations shared by the library's translation units.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/hfm.h"

namespace hfm {

// Thread-local last-error message; returns `status` for `return set_error(...)`.
int set_error(int status, const std::string& msg);

// One FmIndex parsed from bincode (views into the caller's bytes are copied into vectors
// only where the device layout needs a transform).
struct HostFm {
  uint32_t C[16];
  uint8_t num_lanes, num_planes, s2l[16], l2s[16];
  const uint8_t* block_data; uint64_t block_bytes, block_stride;
  uint32_t encoding, occ_text_len;
  const uint8_t* ssa_words; uint64_t ssa_bytes;
  const uint32_t* sa_vals; uint64_t n_sa_vals;     // may be unaligned in the byte stream: copied
  uint32_t sample_rate, ssa_text_len;
  uint32_t text_len, num_sequences;
  std::vector<uint32_t> seq_boundaries;
  std::vector<std::string> headers;
  bool has_lookup; uint32_t lookup_depth;
  std::vector<uint8_t> lookup_core;
  const uint8_t* lookup_intervals; uint64_t n_lookup;
  uint8_t tag;
  std::vector<uint32_t> sa_vals_copy;
};

// Parses and validates FmIndex bincode bytes (src/fm_index/serialize.rs:32-52).  Beyond
// what bincode itself checks, the layout is cross-checked so that no device access can
// leave its buffer.  Returns HFM_OK or HFM_E_FORMAT (message set).
int parse_fm(const uint8_t* p, uint64_t n, HostFm& f);

void suffix_array(const uint8_t* text, uint32_t n, uint32_t* sa);

// One FmIndex in the reference's record layout, ready for the bincode writer: everything but
// the five large sections, which are given by their lengths.
struct FmMeta {
  uint32_t C[16];
  uint8_t num_lanes, num_planes, s2l[16], l2s[16];
  uint64_t n_sb = 0, n_block = 0, n_ssa = 0, n_vals = 0, n_lut = 0;   // u32s, bytes, bytes, u32s, pairs of u32
  uint64_t block_stride;
  uint32_t encoding, text_len;
  uint32_t rate;
  uint32_t num_sequences;
  std::vector<uint32_t> bounds;
  std::vector<std::string> headers;
  uint32_t lookup_depth;
  uint8_t tag;
};

struct BuiltFm : FmMeta {
  std::vector<uint32_t> sb;
  std::vector<uint8_t> block_data;
  std::vector<uint8_t> ssa_words;
  std::vector<uint32_t> sa_vals;
  std::vector<std::pair<uint32_t, uint32_t>> lut;
};

enum FmSection { SEC_SB, SEC_BLOCKS, SEC_SSA, SEC_VALS, SEC_LUT };

// bincode-1 bytes of one FmIndex (fixint, little endian; src/fm_index/serialize.rs:55-67).
// `w` takes bytes by put(p, n) and the large sections by section(id, bytes).
template <class W>
void write_fm(const FmMeta& f, W& w) {
  auto u8 = [&](uint8_t v) { w.put(&v, 1); };
  auto u32 = [&](uint32_t v) { w.put(&v, 4); };
  auto u64 = [&](uint64_t v) { w.put(&v, 8); };
  for (int c = 0; c < 16; c++) u32(f.C[c]);
  // OccTable field order (src/occ/mod.rs:45-78)
  u8(f.num_lanes); u8(f.num_planes); w.put(f.s2l, 16); w.put(f.l2s, 16);
  u64(f.n_sb); w.section(SEC_SB, f.n_sb * 4);
  u64(f.n_block); w.section(SEC_BLOCKS, f.n_block);
  u64(f.block_stride); u32(f.encoding); u32(f.text_len);
  // SampledSuffixArray (src/suffix_array/mod.rs:54-63)
  u64(f.n_ssa); w.section(SEC_SSA, f.n_ssa);
  u64(f.n_vals); w.section(SEC_VALS, f.n_vals * 4);
  u32(f.rate); u32(f.text_len);
  u32(f.text_len); u32(f.num_sequences);
  u64(f.bounds.size()); w.put(f.bounds.data(), f.bounds.size() * 4);
  u64(f.headers.size());
  for (auto& h : f.headers) { u64(h.size()); w.put(h.data(), h.size()); }
  if (f.lookup_depth > 0) {   // Option<LookupTable> (src/fm_index/lookup.rs:19-27)
    u8(1); u32(f.lookup_depth);
    static const uint8_t core[4] = {1, 2, 3, 4};
    u64(4); w.put(core, 4);
    u64(f.n_lut); w.section(SEC_LUT, f.n_lut * 8);
  } else u8(0);
  u8(f.tag);
}

// Joined length, exclusive ends and headers (default "seq_{i}") of the sequences; every code
// is checked to be 1..15 (concatenate_sequences, src/alphabet.rs:375-393).
int sequence_bounds(const uint8_t* codes, const uint64_t* seq_off, uint32_t nseq, const char* const* headers,
                    std::vector<uint32_t>& bounds, std::vector<std::string>& hs);

// Result blocks: pinned host memory from a cache that outlives the calls; hfm_free gives them
// back (api.cu).
void* host_result_alloc(size_t bytes);
void host_result_free(void* p);

}  // namespace hfm

extern "C" int hfm_suffix_array(const uint8_t* text, uint32_t n, uint32_t* sa_out);
