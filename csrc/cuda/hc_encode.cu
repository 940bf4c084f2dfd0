// fp32 (+ streams) -> stream (compress and the homomorphic adds, stand-alone): kernel and launcher.
//
// A unit of work is a SUB-TILE, 32 consecutive blocks (1024 values, 4 KB of fp32), one block per lane.  A CHUNK of nc
// sub-tiles, one per compute warp, is what a CTA takes at a time; one CTA per SM.  The compute warps of a CTA do not
// wait for each other: each has a stage for its fp32 rows (TMA tiled load, 128-byte swizzle), for the adds a byte ring
// for incoming payloads (bulk copies up to two jobs ahead), and a byte ring for packed payloads, in which several of
// them wait for their place in the output while the warp goes on.
//
// Where payloads go: the total of every chunk is published as one word; one warp per CTA (the CLERK) adds up the words
// between its CTA's previous chunk and the current one (at most about 150, five loads a lane, one round trip once they
// are there) and hands every compute warp its byte offset.  A clerk only ever waits for chunk totals, never for another
// clerk, so there is no chain of hops as in a decoupled look-back.
// A launch of one round (a chunk per CTA: up to 2220 sub-tiles for the adds, 3404 for compress) pushes its totals instead
// (give_total): its time is start-up and drain, 147 reductions a CTA in all cost nothing there (seven streams of 8 MB
// added and decoded: 31.9 us, 37.1 before).  In longer launches pushing gained nothing for the first chunk alone.
// Where payloads come from (adds): the same sums over the rate bytes of the input streams, four chunks ahead of the
// compute warps.
#include "hc_host.cuh"
#include "hc_launch.h"
#include "hc_timeline.cuh"
#include "hc_warp.cuh"

namespace hc {
namespace dev {

constexpr int kSlots = 8;    // chunks of a CTA between "total known" and "payload copied out"
constexpr int kInSlots = 4;  // chunks whose input offsets are known

// Compute warps of a CTA at most.  Compress: 24 warps with the clerk, 80 registers each (256 MB, two arrays in turn, 51.4 us; 57.1
// with 20 at 96 registers, 64.6 with 25 at 72, which spill; one array again and again takes 54 to 58).  Adds: 16 warps, which is what the shared memory holds (more would not help: 18 and
// 20 with smaller rings took 47.6 and 44.5 us for 64 MB where 16 took 42.9).
constexpr int kEncWarps = 23;
__host__ __device__ constexpr int enc_warps(int op) { return op == kOpCompress ? kEncWarps : 15; }
// packed payloads: a payload of 4096 bytes, 4 bytes pack_block adds, 16 copy_ring looks ahead
__host__ __device__ constexpr int enc_out_ring(int op) { return op == kOpCompress ? 5376 : 5120; }
// rows of the local operand, which stream + stream has not: it takes their room for payloads, so that two of any length are on
// their way (a random walk, 3.3 KB each: 64 MB 53.9 us, 52.4 this way, 16 MB 20.2 and 19.9; payloads of 1 KB no change)
__host__ __device__ constexpr int enc_stage(int op) { return op == kOpAddStream ? 0 : kSubBytes; }
// incoming payloads, and in front of the ring's end what read_planes and sum_add may look at behind one
__host__ __device__ constexpr int enc_in_ring(int op) { return op == kOpCompress ? 0 : op == kOpAddStream ? 4864 + kSubBytes : 4864; }
__host__ __device__ constexpr int enc_in_usable(int op) { return enc_in_ring(op) - 160; }
__host__ __device__ constexpr int enc_warp_bytes(int op) { return enc_stage(op) + enc_out_ring(op) + enc_in_ring(op); }
static_assert(kEncWarps * 4096 < (1 << 24), "EncShared::sum");
static_assert(32 * 132 + 32 <= enc_in_usable(kOpAddF32), "one payload must fit");
static_assert(2 * (32 * 132 + 32) <= enc_in_usable(kOpAddStream), "two payloads are to fit");
static_assert(kSumReads <= enc_in_ring(kOpAddF32) - enc_in_usable(kOpAddF32), "sum_add reads on behind a payload");

struct EncShared {
  uint64_t stage_full[kEncWarps];
  uint64_t in_full[enc_warps(kOpAddF32)][4];
  uint64_t totals[kSlots];                      // tot[] of the chunk is complete (one arrival per compute warp)
  uint64_t placed[kSlots];                      // out_at[] of the chunk is valid
  uint64_t in_known[kInSlots];                  // in_at[] of the chunk is valid (one arrival per stream)
  uint64_t out_at[kSlots][kEncWarps];           // byte offset of the warp's payload; ~0: not to be stored
  uint64_t in_at[kInSlots][kMaxIn][enc_warps(kOpAddF32)];  // byte offsets of the incoming payloads
  uint64_t in_run[kMaxIn];                      // streams: payload bytes before the CTA's next chunk
  uint32_t tot[kSlots][kEncWarps];
  uint32_t sum[kSlots];  // running total of the chunk [23:0] and number of warps that have added theirs [31:24]
  uint32_t dead;         // an earlier launch timed out and nobody has cleared it: no output
};

// chunk number -> segment and chunk inside it
struct Chunk {
  uint32_t seg, lc;
};
template <bool SEGS>
__device__ __forceinline__ Chunk chunk_of(const SoloParams& p, uint32_t t) {
  if (!SEGS) return Chunk{0u, t};
  uint32_t g = 0;
#pragma unroll 1
  while (g + 1 < p.n_seg && t >= p.first[g + 1]) ++g;
  return Chunk{g, t - p.first[g]};
}
// Chunk number k of this CTA: dealt out in turn (the CTAs of a launch keep the same pace; numbers from a counter went
// unevenly to CTAs whose first warp ran ahead of the others: 21 to 26 of 23 chunks at 256 MB).  kNoTile: none left
__device__ __forceinline__ uint32_t ticket(const SoloParams& p, uint32_t k) {
  const uint32_t t = k * gridDim.x + blockIdx.x;
  return t < p.chunks ? t : kNoTile;
}

// Running sum over the totals of consecutive chunks of a launch: brings `base` from chunk `next` to chunk t (one warp)
__device__ __forceinline__ void advance_base(const uint64_t* words, uint32_t& next, uint64_t& base, uint32_t t, const Workspace& ws) {
#pragma unroll 1
  while (next < t) {
    const uint32_t n = t - next < (uint32_t)kMaxCtas ? t - next : (uint32_t)kMaxCtas;
    base += sum_totals(words + next, n, ws);
    next += n;
  }
}

// The clerk's wait for the totals of chunk k.  The hardware suspends the warp for up to kTotalsNap ns a try, so that
// polling does not take issue slots from the compute warps (100 ns to 20 us measure the same).  False: it ran out, or
// another wait of the launch has (recorded).  A hardware barrier (bar.sync) will not do here: it has no time limit, and
// a warp that gave up would have to go on arriving, in step with the others, for the clerk ever to come back.  It answers
// 0.2 us sooner (compress of 4 KB back to back, on the device, when this took its place: 4.0 us, 4.2 this way); in longer
// launches this was no slower (256 MB 63.3 us and 62.3, 64 MB add 47.7 and 47.3).
constexpr uint32_t kTotalsNap = 2000;
__device__ __forceinline__ bool totals_wait(EncShared& sh, uint32_t k, const Workspace& ws) {
  uint64_t* const bar = &sh.totals[k % kSlots];
  const uint32_t parity = (k / kSlots) & 1u;
  if (__all_sync(0xffffffffu, mbar_try_wait_for(bar, parity, kTotalsNap))) return true;
  const long long t0 = clock64();
  const long long limit_clk = (long long)ws.spin_limit_ns * 2;
  for (uint32_t it = 0; it < (1u << 26); ++it) {
    if (__all_sync(0xffffffffu, mbar_try_wait_for(bar, parity, kTotalsNap))) return true;
    if ((it & 15u) == 15u && __any_sync(0xffffffffu, clock64() - t0 > limit_clk || fatal_error(ws.ctrl))) break;
  }
  if ((threadIdx.x & 31u) == 0u) note_timeout(ws, kSiteScannerTotal);
  return false;
}

// ---- the clerk ---------------------------------------------------------------------------------------------------
// Payload bytes of chunk t in the input streams q0, q0 + dq, ..., published for everybody; one warp
__device__ __forceinline__ void publish_inputs(const SoloParams& p, uint32_t nc, uint32_t subs, uint32_t t, uint32_t q0, uint32_t dq) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t a = t * nc, b = a + nc < subs ? a + nc : subs;
#pragma unroll 1
  for (uint32_t q = q0; q < p.n_in; q += dq) {
    const uint32_t all = __reduce_add_sync(0xffffffffu, payload_len16(rates16(p.in[q], p.in_size[q], a, b, lane)));
    if (lane == 0) st_relaxed_gpu_u64(p.in_words + (size_t)q * p.first[1] + t, st_pack(kStAgg, p.ws.epoch, all));
    if (p.one_round) give_total(p.ws.sums + (1u + q) * kSumWords, all);
  }
}
// Payload offsets of the sub-tiles of chunk t in input stream q (slot r of in_at); one warp.  `next`: chunks before it
// are in sh.in_run[q]
__device__ __forceinline__ void input_offsets(const SoloParams& p, EncShared& sh, uint32_t nc, uint32_t subs, uint32_t t,
                                              uint32_t q, uint32_t r, uint32_t next) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t a = t * nc, b = a + nc < subs ? a + nc : subs;
  const uint32_t sum = payload_len16(rates16(p.in[q], p.in_size[q], a, b, lane));  // half a sub-tile per lane
  const uint32_t inc = warp_inclusive_scan(sum);
  const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
  uint64_t base = sh.in_run[q];
  if (p.one_round) base = take_total(p.ws.sums + (1u + q) * kSumWords, p.ws);
  else advance_base(p.in_words + (size_t)q * p.first[1], next, base, t, p.ws);
  if (!(lane & 1u) && (lane >> 1) < nc) sh.in_at[r][q][lane >> 1] = rate_bytes(p.n[0]) + base + inc - sum;
  __syncwarp();
  if (lane == 0) {
    sh.in_run[q] = base + all;
    mbar_arrive(&sh.in_known[r]);
  }
}

// Adds up the chunk totals, places the payloads; keeps the input offsets kInSlots chunks ahead of the compute warps and
// the published input totals two chunks ahead of that (the first chunk's inputs are the compute warps' work).  Leaves when
// a compute warp has given up; what that leaves unplaced runs out in the others' waits.
__device__ __forceinline__ void clerk(const SoloParams& p, EncShared& sh, uint32_t nc, uint32_t subs, bool has_in, bool segs) {
  const uint32_t lane = threadIdx.x & 31u;
  const Workspace& ws = p.ws;
  // section A covers whole chunks of 32768 values: what is behind the blocks
  for (uint32_t g = blockIdx.x; g < p.n_seg; g += gridDim.x)
#pragma unroll 1
    for (uint64_t b = (uint64_t)p.subs[g] * kSubBlocks + lane; b < rate_bytes(p.n[g]); b += 32u) p.out[g][b] = 0;
  constexpr uint32_t kLead = 2;
  auto inputs_ahead = [&](uint32_t k) {  // offsets of chunk k, totals of chunk k + kLead
    const uint32_t lead = ticket(p, k + kLead), t = ticket(p, k);
    if (lead != kNoTile) publish_inputs(p, nc, subs, lead, 0u, 1u);
    if (t == kNoTile) return;
#pragma unroll 1
    for (uint32_t q = 0; q < p.n_in; ++q) input_offsets(p, sh, nc, subs, t, q, k % kInSlots, ticket(p, k - 1) + 1u);
  };
  if (has_in) {
#pragma unroll 1
    for (uint32_t k = 1; k <= kLead; ++k)
      if (ticket(p, k) != kNoTile) publish_inputs(p, nc, subs, ticket(p, k), 0u, 1u);
    if (!warp_wait(&sh.in_known[0], 0u, ws, kSiteLoaderInFree)) return;  // in_run is the compute warps' until then
#pragma unroll 1
    for (uint32_t k = 1; k < (uint32_t)kInSlots; ++k) inputs_ahead(k);
  }
  uint32_t next = 0;  // chunks [first of the segment, next) are in base
  uint64_t base = 0;
  uint32_t seg = 0;
  for (uint32_t k = 0;; ++k) {
    const uint32_t t = ticket(p, k);
    if (t == kNoTile) break;
    const uint32_t r = k % kSlots;
    if (!totals_wait(sh, k, ws)) return;
    const uint32_t tot = lane < nc ? sh.tot[r][lane] : 0u;
    const uint32_t inc = warp_inclusive_scan(tot);
    const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
    const Chunk c = segs ? chunk_of<true>(p, t) : Chunk{0u, t};
    if (c.seg != seg) {  // every segment is a stream of its own
      seg = c.seg;
      base = 0;
      next = p.first[seg];
    }
    if (p.one_round) base = take_total(ws.sums, ws);
    else advance_base(p.out_words, next, base, t, ws);
    const uint64_t start = rate_bytes(p.n[seg]) + base;
    const uint64_t at = start + inc - tot;
    const bool fits = at + tot <= p.out_cap && !fatal_error(ws.ctrl);
    if (tot && !fits) note_error(ws.ctrl, kErrCapacity);
    if (lane < nc) sh.out_at[r][lane] = tot && fits ? at : ~0ull;
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&sh.placed[r]);
      // the last chunk ends where the stream ends: no size for a stream that did not fit
      if (p.size_out && t + 1 == p.first[seg + 1] && start + all <= p.out_cap && !fatal_error(ws.ctrl)) p.size_out[seg] = start + all;
    }
    base += all;
    next = t + 1;
    if (has_in) inputs_ahead(k + kInSlots);  // every compute warp has taken the inputs of chunk k out of the slot
  }
}

// ---- blocks beyond the reach of the subnormal form ------------------------------------------------------------------
// Row `row` of the stage: fp32 values -> deltas in int32, or their sign and magnitude.  Out of line, and through the stage:
// kept inline it took registers and instruction cache from the common path (64 MB add: 56 us inline, 52 out of line), and
// handed over in local memory it went to L2 and back (32 M values of a random walk with most blocks of this kind, add of
// a stream: 236 us, 126 this way; compress 80, 65).
template <int MODE, bool SIGN>
__device__ __noinline__ void cold_local(uint8_t* stage, int row, float recip) {
  uint32_t x[32];
  load_row_swizzled(stage, row, x);
  deltas_int<MODE>(x, recip);
  if (SIGN) {
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = sign_magnitude(x[i]);
  }
  store_row_swizzled(stage, row, x);
}

// Rows that the TMA unit cannot bring (a ragged end, an operand off the 16-byte boundary), past `n` zeros.  Coherent loads: the
// kernel may have started while the one that writes the operand was still at work.
static __device__ __noinline__ void load_rows(uint8_t* stage, const uint32_t* src, uint64_t first, uint64_t n) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 4
  for (int r = 0; r < kSubBlocks; ++r) {
    const uint64_t i = first + r * kBlock + lane;
    sts32((swizzled_row(stage, r) ^ ((lane >> 2) << 4)) | ((lane & 3u) << 2), i < n ? __ldcg(src + i) : 0u);
  }
}

// ---- the kernel --------------------------------------------------------------------------------------------------
// SEGS: several segments in the launch.  A kernel of its own, because a thread has 80 registers and a single array does not pay for
// those that finding the segment of a chunk takes (one kernel for both, as it then was, had spills: compress of 256 MB 54.4 us with
// two arrays in turn, 51.4 with one of its own)
// ONE: one input stream.  Its kernel has no loop over streams (add of 64 MB 40.3 us, 38.8 this way; for the two of
// stream + stream a constant number gained nothing)
template <int OP, int MODE, bool SEGS, bool ONE>
__global__ void __launch_bounds__((enc_warps(OP) + 1) * 32, 1)
hc_encode_solo_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ SoloParams p) {
  constexpr bool kHasLocal = OP != kOpAddStream;
  constexpr bool kHasIn = OP != kOpCompress;
  constexpr bool kFloat = OP != kOpAddI32;  // the subnormal form may apply
  constexpr bool kPlanes = kHasIn && kFloat && !ONE;  // contributions are added as planes (see PlaneSum)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ EncShared sh;
  __shared__ __align__(64) uint32_t masks[kPlanes ? kMaskPitch * kSumMaskRows : 4];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t nc = (blockDim.x >> 5) - 1u;  // compute warps
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Workspace& ws = p.ws;
  HC_TL_DECL(ws.epoch);
  const uint32_t Q = !kHasIn ? 0u : ONE ? 1u : p.n_in;

  if (tid < nc) {
    mbar_init(&sh.stage_full[tid], 1);
    if (kHasIn)
      for (int i = 0; i < 4; ++i) mbar_init(&sh.in_full[tid][i], 1);
  } else if (warp == 1u) {
    if (lane < (uint32_t)kSlots) {
      mbar_init(&sh.totals[lane], nc);
      mbar_init(&sh.placed[lane], 1);
      sh.sum[lane] = 0;
    }
    if (kHasIn && lane < (uint32_t)kInSlots) mbar_init(&sh.in_known[lane], Q);
    if (kHasIn && lane < (uint32_t)kMaxIn) sh.in_run[lane] = 0;
  }
  fence_mbar_init();
  if (kPlanes) fill_masks<kSumMaskRows>(masks);
  if (tid == 0) launch_dependents();
  grid_dependency_wait();  // nothing in global memory is touched before (see launch_overlapped)
  if (tid == 0) {
    sh.dead = fatal_error(ws.ctrl) ? 1u : 0u;
    HC_TL_ZERO();
    HC_STAMP(0);
  }
  __syncthreads();
  if (sh.dead) return;  // (one answer for all warps)
  const uint32_t subs0 = p.subs[0];
  if (warp == nc) {
    clerk(p, sh, nc, subs0, kHasIn, SEGS);
    return;
  }

  // ============================================ compute warps ==========================================================
  uint8_t* const stage = smem + warp * enc_stage(OP);
  uint8_t* const inring = smem + nc * enc_stage(OP) + warp * enc_in_ring(OP);
  const uint32_t oring = smem_u32(smem + nc * (enc_stage(OP) + enc_in_ring(OP)) + warp * enc_out_ring(OP));
  constexpr uint32_t kOutBytes = (uint32_t)enc_out_ring(OP);
  struct Where {
    uint32_t seg, sub;  // segment, sub-tile inside it
  };
  auto where = [&](uint32_t t) -> Where {
    if (kHasIn) return Where{0u, t * nc + warp};
    const Chunk c = chunk_of<SEGS>(p, t);
    return Where{c.seg, c.lc * nc + warp};
  };
  auto n_local = [&](uint32_t g) -> uint64_t { return OP == kOpAddI32 ? num_blocks(p.n[g]) * kBlock : p.n[g]; };
  // whole sub-tiles of an aligned operand come through the TMA unit; the rest is loaded by the warp itself
  auto by_tma = [&](const Where& w) -> bool { return w.sub < p.by_tma[w.seg]; };
  auto fetch_stage = [&](uint32_t t) {
    if (!kHasLocal || t == kNoTile) return;
    const Where w = where(t);
    if (lane == 0) {
      if (by_tma(w)) {
        fence_proxy_async();
        mbar_expect_tx(&sh.stage_full[warp], kSubBytes);
        tma_load_2d(stage, &tmaps.m[w.seg], 0, (int)(w.sub * kSubBlocks), &sh.stage_full[warp]);
      } else {
        mbar_arrive(&sh.stage_full[warp]);
      }
    }
  };

  // ---- incoming payloads: jobs (chunk k, stream q) --------------------------------------------------------------------
  uint32_t pk = 0, pq = 0, pt = kNoTile;  // next job to be staged
  uint32_t praw = 0;                      // rate byte of the lane's block in it
  uint32_t live_at = 0, live_end = 0, jobs = 0, staged = 0;
  uint32_t cur_rate = 0, cur_pos = 0, nxt_rate = 0, nxt_pos = 0;
  auto load_rate = [&]() {
    const uint64_t b = ((uint64_t)pt * nc + warp) * kSubBlocks + lane;
    praw = pt != kNoTile && b < (uint64_t)subs0 * kSubBlocks && b < p.in_size[pq] ? ld_cg_u8(p.in[pq] + b) : 0u;
  };
  // stages the next job unless the ring has no room for it
  auto produce = [&]() {
    if (pq == 0 && !warp_wait(&sh.in_known[pk % kInSlots], (pk / kInSlots) & 1u, ws, kSiteLoaderInFree)) {
      pt = kNoTile;
      return;
    }
    const uint32_t len = payload_len(praw);
    const uint32_t inc = warp_inclusive_scan(len);
    uint32_t tot = __shfl_sync(0xffffffffu, inc, 31), rate = praw;
    uint32_t at = staged ? live_end : 0u;
    if (tot && at + tot + 31u > (uint32_t)enc_in_usable(OP)) {
      at = 0;
      if (tot + 31u > (staged ? live_at : (uint32_t)enc_in_usable(OP))) return;
    }
    const uint64_t off = sh.in_at[pk % kInSlots][pq][warp];
    if (tot && off + tot > p.in_size[pq]) {  // stream shorter than its rate bytes imply
      if (lane == 0) note_error(ws.ctrl, kErrTruncated);
      tot = 0;
      rate = 0;
    }
    const uint8_t* const src = p.in[pq] + off;
    const uint32_t phase = (uint32_t)reinterpret_cast<uintptr_t>(src) & 15u;
    const uint32_t bytes = tot ? (phase + tot + 15u) & ~15u : 0u;
    live_at = at;
    live_end = at + bytes;
    uint64_t* const bar = &sh.in_full[warp][jobs & 3u];
    if (lane == 0) {
      if (tot) {
        fence_proxy_async();
        mbar_expect_tx(bar, bytes);
        bulk_load(inring + at, src - phase, bytes, bar);
      } else {
        mbar_arrive(bar);
      }
    }
    ++jobs;
    const uint32_t pos = at + phase + inc - len;
    if (staged) nxt_rate = rate, nxt_pos = pos;
    else cur_rate = rate, cur_pos = pos;
    ++staged;
    if (++pq == Q) {
      pq = 0;
      ++pk;
      pt = ticket(p, pk);
    }
    load_rate();
  };

  uint32_t t = ticket(p, 0);
  fetch_stage(t);
  if (kHasIn) {
    pt = t;
    load_rate();
    if (t != kNoTile) {
      publish_inputs(p, nc, subs0, t, warp, nc);
#pragma unroll 1
      for (uint32_t q = warp; q < Q; q += nc) input_offsets(p, sh, nc, subs0, t, q, 0u, 0u);
    }
  }

  // ---- packed payloads waiting for their place: lane k % kSlots keeps that of chunk k ----------------------------------
  // SEGS: segment [31:26], length [25:13] and start [12:0] in one register.  In three it had spills (16 bytes stored, 36 loaded;
  // two arrays of 64 MB 38.2 us, 36.1 this way, gradients of a block of width 1024 18.1 and 17.6).  The other kernels have none to
  // lose and are slower for the unpacking (compress of 16 MB 7.04 us, 7.22 this way; add of int32 deltas of 128 MB, whose 12 bytes
  // of spills it would take away, 70.7 and 71.6)
  uint32_t my_start = 0, my_tot = 0;
  static_assert(kOutBytes <= 1u << 13 && kSubBlocks * 128 < 1 << 13 && kMaxDst <= 64, "fields of my_start");
  // ring: free is [head, end) and [0, tail), or, once wrapped (head < tail), [head, tail); all of it when taken == 0
  uint32_t head = 0, tail = 0, taken = 0;
  uint32_t copied = 0;  // chunks [copied, k) wait
  auto room_for = [&](uint32_t tot) -> uint32_t { return tot ? (tot + 20u + 15u) & ~15u : 0u; };
  auto copy_oldest = [&]() {
    const uint32_t r = copied % kSlots;
    const uint32_t mine = __shfl_sync(0xffffffffu, my_start, (int)r), start = SEGS ? mine & 0x1fffu : mine;
    const uint32_t tot = SEGS ? mine >> 13 & 0x1fffu : __shfl_sync(0xffffffffu, my_tot, (int)r);
    const uint64_t at = sh.out_at[r][warp];
    if (tot) {
      if (at != ~0ull) copy_ring(oring + start, p.out[SEGS ? mine >> 26 : 0u] + at, tot);
      tail = start + room_for(tot);
      if (--taken == 0) head = tail = 0;
    }
    ++copied;
  };
  auto placed = [&](uint32_t k) -> bool { return __all_sync(0xffffffffu, mbar_test(&sh.placed[k % kSlots], (k / kSlots) & 1u)); };

  // A warp whose wait ran out (recorded) leaves.  Every wait of the others has a limit of its own, so they follow.
  bool failed = false;
  uint32_t k = 0, rows = 0, read = 0;  // failed: the chunk whose rows, the input job that may still be on their way
  if (tid == 0) HC_PH_START();
  for (;; ++k) {
    if (t == kNoTile) {
#pragma unroll 1
      while (copied < k) {
        if (!warp_wait(&sh.placed[copied % kSlots], (copied / kSlots) & 1u, ws, kSiteCopierBase)) break;
        copy_oldest();
      }
      break;
    }
    if (tid == 0) HC_PH(0);
    const Where w = where(t);
    const uint32_t t_next = ticket(p, k + 1);
    uint32_t d[32];
    PlaneSum sum;
    uint32_t or_tail = 0;
    bool ints = false;  // d holds int32 deltas instead of subnormals
    // ---- local operand: first, because it needs nothing but its rows --------------------------------------------------
    if (kHasLocal) {
      if (!warp_wait(&sh.stage_full[warp], k & 1u, ws, kSiteComputeTile)) {
        failed = true;
        rows = k;
        read = k * Q;
        break;
      }
      if (tid == 0) HC_PH(1);
      if (__builtin_expect(!by_tma(w), 0)) {
        load_rows(stage, reinterpret_cast<const uint32_t*>(p.local[w.seg]), (uint64_t)w.sub * kSubValues, n_local(w.seg));
        __syncwarp();
      }
      load_row_swizzled(stage, (int)lane, d);
      if (kFloat) {
        deltas_sub<MODE>(d, p.recip, p.one);
        // exact when no quantised value of the block reaches 2^24: |q_0| below 2^23 and 31 differences below 2^18
        or_tail = or_tail_of(d);
        if (__builtin_expect(!__all_sync(0xffffffffu, or_tail < (1u << 18) && (d[0] & 0x7fffffffu) < (1u << 23)), 0)) {
          cold_local<MODE, !kHasIn>(stage, (int)lane, p.recip);
          load_row_swizzled(stage, (int)lane, d);
          if (!kHasIn) or_tail = or_tail_of(d);
          else ints = true;
        } else if (kHasIn && !kPlanes) {
          d[0] = sub_to_int(d[0]);
        }
      }
      __syncwarp();
      fetch_stage(t_next);  // every lane holds its row
      if (kPlanes) sum_local(sum, d, or_tail, ints);
    } else {
      sum_clear(sum);
    }
    if (tid == 0) HC_PH(2);
    // ---- incoming streams ----------------------------------------------------------------------------------------------
    if (kHasIn) {
#pragma unroll 1
      for (uint32_t q = 0; q < Q; ++q) {
#pragma unroll 1
        while (staged < 2u && pt != kNoTile) {
          const uint32_t before = staged;
          produce();
          if (staged == before) break;
        }
        const uint32_t v = k * Q + q;
        if (!warp_wait(&sh.in_full[warp][v & 3u], (v >> 2) & 1u, ws, kSiteComputeInFull)) {
          failed = true;
          rows = k + 1u;
          read = v;
          break;
        }
        if (tid == 0) HC_PH(3);
        if (kPlanes) {
          sum_add(sum, inring, masks, cur_pos, cur_rate);
          __syncwarp();
        } else {
          uint32_t T[32], sign, a0;
          decode_rows<-1>(inring, nullptr, cur_pos, cur_rate, plane_width(__reduce_max_sync(0xffffffffu, cur_rate & 31u)), sign, a0, T);
          __syncwarp();
          // |d_1| .. |d_31| small enough for sums in subnormals: so with up to 16 planes, else to be looked at (a
          // plain block may have many planes for the sake of d_0 alone, which is summed in int32)
          bool fits = (cur_rate & 31u) <= 16u;
          if (kFloat && __builtin_expect(!__all_sync(0xffffffffu, fits), 0)) fits = fits || or_rows_tail(T) < (1u << 20);
          if (kFloat && __builtin_expect(__all_sync(0xffffffffu, fits) && !ints, 1)) {
            const uint32_t m = (uint32_t)((int32_t)sign >> 31);
            d[0] += (T[7] ^ m) - m;
            d[1] = as_u(__fadd_rn(as_f(d[1]), as_f(signed_sub(T[6], sign, 1))));
#pragma unroll
            for (int i = 2; i < 32; i += 2)
              unpack2(add2(pack2(d[i], d[i + 1]), pack2(signed_sub(T[i ^ 7], sign, i), signed_sub(T[(i + 1) ^ 7], sign, i + 1))), d[i], d[i + 1]);
          } else {
            if (kFloat && !ints) {
#pragma unroll
              for (int i = 1; i < 32; ++i) d[i] = sub_to_int(d[i]);
              ints = true;
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const uint32_t m = (uint32_t)((int32_t)(sign << i) >> 31);
              d[i] += (T[i ^ 7] ^ m) - m;
            }
          }
        }
        cur_rate = nxt_rate;
        cur_pos = nxt_pos;
        --staged;
        if (tid == 0) HC_PH(4);
      }
      if (failed) break;
      if (!kPlanes) {
        if (!kFloat || __builtin_expect(ints, 0)) {
#pragma unroll
          for (int i = 0; i < 32; ++i) d[i] = sign_magnitude(d[i]);
        } else {
          d[0] = sign_magnitude(d[0]);
        }
        or_tail = or_tail_of(d);
      }
    }

    if (tid == 0) HC_PH(4);
    // ---- encode -----------------------------------------------------------------------------------------------------------
    const BlockCode code = [&]() -> BlockCode {
      if constexpr (kPlanes) return sum_code<MODE>(sum);
      else return code_of<MODE>(d, or_tail);
    }();
    const uint32_t inc = warp_inclusive_scan(code.len);
    const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
    uint32_t before = 0;
    if (lane == 0) {
      const uint32_t r = k % kSlots;
      sh.tot[r][warp] = tot;
      // the last warp publishes the chunk's total, not the clerk: other CTAs wait for it, whatever this one's clerk
      // is waiting for (published by the clerks, the totals moved on in lock step, 4 us a chunk)
      before = atomicAdd(&sh.sum[r], (1u << 24) | tot);
      if (before >> 24 == nc - 1u) {
        st_relaxed_gpu_u64(p.out_words + t, st_pack(kStAgg, ws.epoch, (before & 0xffffffu) + tot));
        sh.sum[r] = 0;
      }
    }
    if (p.one_round) {
      before = __shfl_sync(0xffffffffu, before, 0);
      if (before >> 24 == nc - 1u) give_total(ws.sums, (before & 0xffffffu) + tot);
    }
    if (lane == 0) mbar_arrive(&sh.totals[k % kSlots]);
    __syncwarp();
    const uint32_t subs = p.subs[w.seg];
    uint8_t* const rates = p.out[w.seg];
    if (w.sub < subs) rates[(uint64_t)w.sub * kSubBlocks + lane] = (uint8_t)code.rate;

    if (tid == 0) HC_PH(5);
    // payloads whose place is known leave; the oldest ones have to where this one needs their room
    // (one a turn keeps the pace; a second look pays only where they pile up)
    if (copied < k && placed(copied)) {
      copy_oldest();
#pragma unroll 1
      while (copied + 2u < k && placed(copied)) copy_oldest();
    }
    const uint32_t need = room_for(tot);
    uint32_t start = head;
#pragma unroll 1
    while (true) {
      bool room = true;
      start = head;
      if (need && taken) {
        if (head >= tail && head + need > kOutBytes) {
          start = 0;
          room = need < tail;
        } else if (head < tail) {
          room = head + need < tail;
        }
      }
      if (room && k - copied < (uint32_t)kSlots - 1u) break;
      if (tid == 0) HC_PH(6);
      if (!warp_wait(&sh.placed[copied % kSlots], (copied / kSlots) & 1u, ws, kSiteComputeRing)) {
        failed = true;
        rows = k + 1u;
        read = rows * Q;
        break;
      }
      if (tid == 0) HC_PH(9);
      copy_oldest();
    }
    t = t_next;
    if (failed) break;
    if (tid == 0) HC_PH(6);
    __syncwarp();
    const int W = plane_width(__reduce_max_sync(0xffffffffu, code.rate & 31u));
    if (kPlanes) pack_planes(oring + start, inc - code.len, code, sum.A, W);
    else pack_blocks(oring + start, inc - code.len, code, d, W);
    if (lane == k % kSlots) {
      my_start = SEGS ? start | tot << 13 | w.seg << 26 : start;
      if (!SEGS) my_tot = tot;
    }
    if (need) {
      head = start + need;
      ++taken;
    }
    if (tid == 0) {
      HC_PH(7);
      HC_PH_COUNT();
    }
  }
  if (failed) {  // nothing may land in shared memory once the CTA has left it
    if (kHasLocal && ticket(p, rows) != kNoTile) mbar_wait_bounded(&sh.stage_full[warp], rows & 1u, ws.spin_limit_ns);
    for (; kHasIn && read < jobs; ++read) mbar_wait_bounded(&sh.in_full[warp][read & 3u], (read >> 2) & 1u, ws.spin_limit_ns);
  }
  if (tid == 0) HC_PH(8);
  if (lane == 0) HC_STAMP_MAX(7);
}

}  // namespace dev

// ---- host side ---------------------------------------------------------------------------------------------------

namespace {

template <int OP, int MODE, bool SEGS, bool ONE>
cudaError_t launch_solo_t(const TensorMaps& maps, SoloParams p, cudaStream_t stream) {
  constexpr int kWarps = dev::enc_warps(OP);
  auto smem = [](int nc) { return nc * dev::enc_warp_bytes(OP) + 1024; };
  static thread_local int cache[64] = {};
  const int cap = resident_ctas(dev::hc_encode_solo_kernel<OP, MODE, SEGS, ONE>, 32 * (kWarps + 1), smem(kWarps), cache);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  const EncodeSplit split = split_encode(p.subs, p.n_seg, (uint32_t)(cap < kMaxCtas ? cap : kMaxCtas), (uint32_t)kWarps);
  if (encode_words(split, p.n_seg, p.n_in) > p.ws.words) return cudaErrorInvalidValue;
  const int nc = (int)split.warps;
  memcpy(p.first, split.first, sizeof(p.first));
  p.chunks = p.first[p.n_seg];
  p.one_round = split.one_round;
  p.one = 1.0f;
  p.out_words = p.ws.st_a;
  p.in_words = p.ws.st_a + p.first[p.n_seg];
  return launch_overlapped(dev::hc_encode_solo_kernel<OP, MODE, SEGS, ONE>, (int)split.grid, 32 * (nc + 1), smem(nc), stream, maps, p);
}

template <int OP, bool SEGS = false, bool ONE = false>
cudaError_t launch_solo_m(int mode, const TensorMaps& maps, const SoloParams& p, cudaStream_t stream) {
  switch (mode) {
    case kModeOutlier: return launch_solo_t<OP, kModeOutlier, SEGS, ONE>(maps, p, stream);
    case kModePlain: return launch_solo_t<OP, kModePlain, SEGS, ONE>(maps, p, stream);
    case kModeVec: return launch_solo_t<OP, kModeVec, SEGS, ONE>(maps, p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_encode_solo(int op, int mode, SoloParams p, cudaStream_t stream) {
  if (p.n_seg == 0 || p.n_seg > (uint32_t)kMaxDst || p.n_in > (uint32_t)kMaxIn) return cudaErrorInvalidValue;
  if ((p.n_seg > 1 && op != kOpCompress) || (op == kOpCompress) != (p.n_in == 0)) return cudaErrorInvalidValue;
  TensorMaps maps;
  memset(&maps, 0, sizeof(maps));
  uint64_t total = 0;
  for (uint32_t g = 0; g < p.n_seg; ++g) {
    total += p.n[g];
    p.subs[g] = (uint32_t)((p.n[g] + dev::kSubValues - 1) / dev::kSubValues);
    p.by_tma[g] = 0;
    if (op == kOpAddStream) continue;
    // int32 deltas are stored in whole blocks; fp32 data may end in a ragged row
    const uint64_t whole = (op == kOpAddI32 ? num_blocks(p.n[g]) * kBlock : p.n[g]) / dev::kSubValues;
    if (whole && make_rows_map(&maps.m[g], p.local[g], whole * dev::kSubBlocks, dev::kSubBlocks)) p.by_tma[g] = (uint32_t)whole;
  }
  if (total == 0) return cudaSuccess;
  switch (op) {
    case kOpCompress:
      return p.n_seg > 1 ? launch_solo_m<kOpCompress, true>(mode, maps, p, stream) : launch_solo_m<kOpCompress>(mode, maps, p, stream);
    case kOpAddF32:
      return p.n_in == 1 ? launch_solo_m<kOpAddF32, false, true>(mode, maps, p, stream) : launch_solo_m<kOpAddF32>(mode, maps, p, stream);
    case kOpAddI32: return p.n_in == 1 ? launch_solo_m<kOpAddI32, false, true>(mode, maps, p, stream) : cudaErrorInvalidValue;
    case kOpAddStream: return launch_solo_m<kOpAddStream>(mode, maps, p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hc

HC_TL_READ(hc_debug_timeline_encode)
