// How a stand-alone launch is cut up, and the workspace that it needs for that: plain host arithmetic, apart from the
// launchers so that it can be checked without a GPU over every call that the entry points accept.
#pragma once
#include "hc_format.h"

namespace hc {

constexpr int kTileBlocks = 128;
constexpr int kTileElems = kTileBlocks * kBlock;  // 4096
constexpr int kMaxDst = 8;
constexpr int kMaxIn = kMaxDst;
constexpr int kMaxCtas = 160;  // CTAs of a launch with one CTA per SM
// exchange of CTA totals (dev::give_total): a word per CTA, a word per group of CTAs, and per CTA what its group's word was
constexpr int kSumGroup = 13, kSumGroups = (kMaxCtas + kSumGroup - 1) / kSumGroup;
constexpr int kSumWords = kMaxCtas + 16 + kMaxCtas;
static_assert(kSumGroups <= 16 && kSumGroup <= 16, "one reduction a lane");

// ---- workspace -----------------------------------------------------------------------------------------------------
// Words in front of the exchange of CTA totals, for calls of up to max_elems values split over up to kMaxDst segments
// (each rounded up to whole chunks of 32768 values).  The steps of a collective use them as three look-back chains (a
// word per tile, a word per 32 tiles), the stand-alone kernels as one array.
HC_HD size_t workspace_tiles(size_t max_elems) {
  return rate_bytes(max_elems) / kTileBlocks + (size_t)kMaxDst * (kBlocksPerChunk / kTileBlocks) + 1;
}
HC_HD size_t workspace_groups(size_t max_elems) { return workspace_tiles(max_elems) / 32 + 1 + kMaxDst; }
HC_HD size_t workspace_words(size_t max_elems) { return 3 * (workspace_tiles(max_elems) + workspace_groups(max_elems)); }

// ---- encode --------------------------------------------------------------------------------------------------------
struct EncodeSplit {
  uint32_t warps;               // compute warps per CTA, the sub-tiles of a chunk
  uint32_t grid;
  uint32_t first[kMaxDst + 1];  // chunk numbers at which the segments start; [n_seg]: number of chunks
  bool one_round;               // one stream, a chunk per CTA
};
// Compute warps per CTA: as many rounds of chunks as the largest CTA needs, then no more warps than fill them (where the
// last round would be half empty, all rounds are narrower instead); at least four at a time.
inline EncodeSplit split_encode(const uint32_t* subs, uint32_t n_seg, uint32_t sms, uint32_t max_warps) {
  EncodeSplit s;
  uint64_t all = 0;
  for (uint32_t g = 0; g < n_seg; ++g) all += subs[g];
  const uint64_t per_round = (uint64_t)sms * max_warps, rounds = (all + per_round - 1) / per_round;
  const uint64_t warps = (all + sms * rounds - 1) / (sms * rounds);
  s.warps = warps < 4 ? 4u : (uint32_t)warps;
  s.first[0] = 0;
  for (uint32_t g = 0; g < n_seg; ++g) s.first[g + 1] = s.first[g] + (subs[g] + s.warps - 1) / s.warps;
  const uint32_t chunks = s.first[n_seg];
  s.grid = chunks < sms ? chunks : sms;
  s.one_round = n_seg == 1 && chunks <= sms;
  return s;
}
// a word per chunk for its payload bytes, and one per chunk and input stream
inline uint64_t encode_words(const EncodeSplit& s, uint32_t n_seg, uint32_t n_in) { return (uint64_t)s.first[n_seg] * (1u + n_in); }

// ---- decode --------------------------------------------------------------------------------------------------------
struct RunSplit {
  uint32_t warps;  // per CTA
  uint32_t grid;
  uint32_t pool;   // sub-tiles at the end of every warp's run that are handed out one by one
};
// Few sub-tiles are spread over the SMs four at a time (fewer CTAs exchange their totals faster).  The pool: an eighth of
// a run; none where a run is a sub-tile or three.
inline RunSplit split_runs(uint64_t subs, uint32_t sms, uint32_t max_warps) {
  RunSplit s;
  const uint64_t warps = (subs + sms - 1) / sms;
  s.warps = warps < 4u ? 4u : warps > max_warps ? max_warps : (uint32_t)warps;
  const uint64_t ctas = (subs + s.warps - 1) / s.warps;
  s.grid = ctas < sms ? (uint32_t)ctas : sms;
  const uint64_t run = subs / ((uint64_t)s.grid * s.warps);
  s.pool = run < 4 ? 0u : run < 8 ? 1u : (uint32_t)(run / 8);
  return s;
}
// Payload bytes, in stream q, of the runs of a CTA's warps before `warp`, of up to 16: the share of lane `part` of eight.  The total of
// one run fits 32 bits; that of a CTA need not, where a large array meets few SMs.
HC_HD uint64_t runs_before(const uint32_t (*totals)[kMaxDst], uint32_t q, uint32_t warp, uint32_t part) {
  return (uint64_t)(part < warp ? totals[part][q] : 0u) + (part + 8u < warp ? totals[part + 8u][q] : 0u);
}
// a word per pooled sub-tile and stream for its payload offset
inline uint64_t run_words(const RunSplit& s, uint32_t streams) { return (uint64_t)s.pool * s.grid * s.warps * streams; }

}  // namespace hc
