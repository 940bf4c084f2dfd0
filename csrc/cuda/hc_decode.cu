// stream -> fp32 (decompress, its flagged and multi-stream forms): kernel and launcher.
//
// A unit of work is a SUB-TILE: 32 consecutive blocks (1024 values, 4 KB of fp32), one block per lane, a quarter
// of a tile.  Every warp works alone: payloads come by bulk copy into a byte ring of its own; the decoded 4 KB go to an output
// buffer (128-byte swizzle) and leave through a TMA tiled store.  Inside the loop no warp waits for another one.
//
// Stand-alone streams (hc_decode_run_kernel; the sum of several: hc_decode_kernel): every warp of the grid owns a contiguous run of
// sub-tiles.  It sums the payload lengths of its run from the rate bytes (700 bytes for a 256 MB array), the CTAs (one per SM, so
// at most 148) exchange their totals once through the workspace, and from there on a warp carries its own running offset: no
// look-back, no second kernel.  The SMs do not run at the same pace (with equal static shares the first warp of a 256 MB launch
// finished at 42 us, the last at 70), so the last eighth of every run goes to whoever is free first; the payload
// offsets of those sub-tiles are written to the workspace after the first one has been decoded.
// What bounds the decode of one stream: 256 MB the memory (60.9 us), 64 MB the memory and the start (21.2; before the masks 22.8, with
// 20.8 without the arithmetic and 19.0 without the stores), smaller ones the way to the first payload: rate bytes, exchange, payload, one trip to
// L2 after the other (8 MB: of 6.1 us on the device 3.3; 5.1 of 7.5 when 64-bit divisions, the status and the offsets of the pool
// stood in between).
//
// Steps of a collective: hc_decode_step.cuh.
#include "hc_decode_step.cuh"
#include "hc_host.cuh"
#include "hc_launch.h"
#include "hc_timeline.cuh"
#include "hc_warp.cuh"

namespace hc {
namespace dev {

// ---- sum of several stand-alone streams ------------------------------------------------------------------------------
// As with one stream (below) every warp has a contiguous run of sub-tiles, and its offset in every stream.  What it stages at a time is a
// BATCH, the payloads of one sub-tile in up to four streams, and everything that goes with one is done for the four at once: lanes
// 8 s .. 8 s + 7 belong to stream s, each with the rate bytes of four blocks.  Staged one by one, every stream of a sub-tile cost a scan,
// room in the ring, bounds and a barrier of its own, 300 of its 470 instructions (four streams of 256 MB 198 us, 143 this way; seven
// of 40 MB 67.6 and 48.1; four of 4 MB 11.0 and 8.7; two of 4 KB 5.2 and 4.9).  So are the totals of a run and the offsets of its pool,
// which stream by stream were 5 to 8 % of seven streams of 40 MB.  A batch whose payloads do not all fit in the ring is staged in parts.
// What bounds it: instructions, at 16 warps an SM (four streams of 256 MB: 84 us of memory traffic); short runs the same trips to L2 as
// one stream's.
constexpr int kSumWarps = 16;
constexpr uint32_t kSumRing = 10112, kSumUsable = kSumRing - 160;  // (see kDecRingUsable)
constexpr int kSumWarpBytes = kSubBytes + (int)kSumRing;
static_assert(32 * 132 + 32 <= kSumUsable, "one payload must fit");
static_assert((uint32_t)kSumReads <= kSumRing - kSumUsable, "sum_add reads on behind a payload");
static_assert(kSumWarps <= 16, "runs_before");

__global__ void __launch_bounds__(kSumWarps * 32, 1)
hc_decode_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ DecParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t s_full[kSumWarps][2];
  __shared__ uint32_t s_tot[kSumWarps][kMaxDst];  // payload bytes of a run
  __shared__ uint64_t s_pre[kMaxDst];
  __shared__ __align__(64) uint32_t masks[kMaskPitch * kSumMaskRows];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n_warps = blockDim.x >> 5;
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* const obuf = smem + warp * kSubBytes;
  uint8_t* const ring = smem + n_warps * kSubBytes + warp * kSumRing;
  const Workspace& ws = p.ws;
  uint64_t* const full = s_full[warp];
  if (lane < 2u) mbar_init(&full[lane], 1);
  fence_mbar_init();
  if (tid == 0) launch_dependents();
  fill_masks<kSumMaskRows>(masks);
  grid_dependency_wait();  // nothing in global memory is touched before (see launch_overlapped)
  __syncwarp();
  const uint32_t Q = p.n_seg;
  const uint32_t gw = blockIdx.x * n_warps + warp, nw = gridDim.x * n_warps;
  const uint32_t status = *((volatile const uint32_t*)(ws.ctrl + 2));
  HC_TL_DECL(ws.epoch);
  if (tid == 0) {
    HC_TL_ZERO();
    HC_STAMP(0);
    HC_PH_START();
  }

  // ---- shares, offsets -----------------------------------------------------------------------------------------------
  auto run_of = [&](uint32_t w) -> uint32_t { return p.run_all * w + (w < p.run_more ? w : p.run_more); };
  const uint32_t pool = p.pool;  // sub-tiles at the end of every run that are handed out one by one
  uint32_t it = run_of(gw);
  const uint32_t run_end = run_of(gw + 1u), own_end = run_end - pool;
  auto sum8 = [&](auto v) {  // over the lanes of a stream
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  // Payload bytes of the run in every stream: eight lanes a stream, 16 rate bytes a lane
  const uint32_t mine = lane >> 3, part = lane & 7u;  // stream of the four
  uint32_t sum = 0, sum_2 = 0;                        // of streams `mine` and 4 + `mine`
  if (p.run_all + (p.run_more ? 1u : 0u) <= 4u) {
    uint4 v = make_uint4(0, 0, 0, 0), v_2 = v;
    if (mine < Q) v = rates16(p.seg[mine].in, p.seg[mine].in_size, it, run_end, part);
    if (mine + 4u < Q) v_2 = rates16(p.seg[mine + 4u].in, p.seg[mine + 4u].in_size, it, run_end, part);
    sum = sum8(payload_len16(v) | payload_len16(v_2) << 16);  // below 2^16 each: 4 * 32 * 132 at most
    sum_2 = sum >> 16;
    sum &= 0xffffu;
  } else {
    // Longer runs: 16 sub-tiles of all streams are asked for before the first is added (one stream after the other: eight of
    // 40 MB 96.0 us, 92.6 with four at a time)
#pragma unroll 1
    for (uint32_t at = it; at < run_end; at += 16u) {
      uint4 v[8];
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) {
        const uint32_t q = mine + 4u * (j & 1u), first = at + 4u * (j >> 1);
        v[j] = q < Q && first < run_end ? rates16(p.seg[q].in, p.seg[q].in_size, first, run_end, part) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (uint32_t j = 0; j < 4u; ++j) {
        if (at + 4u * j >= run_end) break;
        sum += payload_len16(v[2u * j]);
        if (Q > 4u) sum_2 += payload_len16(v[2u * j + 1u]);
      }
    }
    sum = sum8(sum);
    if (Q > 4u) sum_2 = sum8(sum_2);
  }
  if (part == 0u) {
    s_tot[warp][mine] = sum;
    s_tot[warp][mine + 4u] = sum_2;
  }

  // ---- units: a sub-tile in streams 4 half .. 4 half + 3 ------------------------------------------------------------------
  // items: own sub-tiles, then tickets of the pools (kPool set)
  constexpr uint32_t kPool = 0x80000000u;
  uint32_t tk_raw = kNoTile;
  const uint32_t n_tickets = pool * nw;
  auto ask = [&]() {
    if (lane == 0) tk_raw = atomicAdd(ws.tick, 1u);
  };
  auto next_item = [&]() -> uint32_t {
    if (it < own_end) {
      const uint32_t i = it++;
      if (it == own_end && pool) ask();
      return i;
    }
    if (!pool) return kNoTile;
    const uint32_t t = __shfl_sync(0xffffffffu, tk_raw, 0);
    if (t >= n_tickets) return kNoTile;
    ask();
    return t | kPool;
  };
  // ticket t is the (t / nw)-th pool sub-tile of warp t % nw
  auto sub_of = [&](uint32_t item) -> uint32_t {
    if (!(item & kPool)) return item;
    const uint32_t w = (item & ~kPool) % nw, k = (item & ~kPool) / nw;
    return run_of(w + 1u) - pool + k;
  };
  auto pool_flag = [&](uint32_t t, uint32_t q) -> uint64_t* { return p.flags + (size_t)q * pool * nw + (t & ~kPool); };
  struct Unit {
    uint32_t item, half;
    uint32_t sub;
    uint32_t rates;  // of the lane's four blocks
    uint64_t flag;   // pool items: a look at the payload offset
  };
  auto look = [&](Unit& u) {
    const uint32_t q = 4u * u.half + mine;
    u.rates = 0;
    u.flag = 0;
    if (u.item == kNoTile || q >= Q) return;
    u.rates = load_rates4(p.seg[q].in, p.seg[q].in_size, (uint64_t)u.sub * kSubBlocks + 4u * part);
    if (u.item & kPool) u.flag = ld_relaxed_gpu_u64(pool_flag(u.item, q));
  };
  // (an earlier launch that timed out, and nobody has cleared its status: no output)
  Unit next{};
  next.item = status >= (uint32_t)kErrTimeout ? kNoTile : next_item();
  next.sub = sub_of(next.item);
  look(next);

  __syncthreads();
  for (uint32_t q = warp; q < Q; q += n_warps)
    give_total_of(ws.sums + (1u + q) * kSumWords, warp_sum_u64(lane < n_warps ? s_tot[lane][q] : 0ull));
  for (uint32_t q = warp; q < Q; q += n_warps) {
    const uint64_t pre = take_total_of(ws.sums + (1u + q) * kSumWords, ws);
    if (lane == 0) s_pre[q] = pre;
  }
  __syncthreads();
  // offset of the next own sub-tile's payload in the lane's stream of this half, of the other one
  auto before_me = [&](uint32_t q) -> uint64_t {
    return rate_bytes(p.seg[0].n) + (q < Q ? s_pre[q] : 0u) + sum8(runs_before(s_tot, q, warp, part));
  };
  uint64_t own_off = before_me(mine), own_off_2 = Q > 4u ? before_me(mine + 4u) : 0u;

  // ---- staging -------------------------------------------------------------------------------------------------------
  struct Batch {
    uint32_t rates;        // of the lane's four blocks of its stream
    uint32_t pos;          // ring byte of their payload
    uint32_t begin, end;   // its streams of the four
    uint32_t sub;
    bool first, last;      // of the sub-tile's batches
  };
  Batch cur{}, nxt{};
  uint32_t staged = 0, jobs = 0;  // batches in the ring, and so far
  uint32_t live_at = 0, live_end = 0;  // ring bytes of the newest batch
  Unit un{};
  bool open = false;     // `un` has streams [done, many) still to be staged
  uint32_t done = 0, many = 0;
  uint32_t before = 0, bytes = 0;  // payload bytes of the lane's stream in front of its blocks; of the copy
  uint64_t src = 0;                // address of its payload
  auto stage = [&](Batch& b) -> bool {
    if (!open) {
      un = next;
      many = Q - 4u * un.half < 4u ? Q - 4u * un.half : 4u;
      done = 0;
      open = true;
      // the next unit's rate bytes and offsets are on their way while this one is worked on
      if (un.half == 0u && Q > 4u) {
        next.half = 1u;
      } else {
        next.half = 0u;
        next.item = next_item();
        if (next.item != kNoTile) next.sub = sub_of(next.item);
      }
      look(next);
      const uint32_t sum = payload_len4(un.rates);
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o, 8);
        if (part >= (uint32_t)o) inc += v;
      }
      before = inc - sum;
      const uint32_t tot = __shfl_sync(0xffffffffu, inc, 7, 8);
      uint64_t off = own_off;
      if (un.item & kPool) {
        off = un.flag;
        const bool there = mine >= many || flag_matches(off, p.ring_epoch);
        if (__builtin_expect(!__all_sync(0xffffffffu, there), 0)) {
#pragma unroll 1
          for (uint32_t s = 0; s < many; ++s) {
            const uint64_t fw = own_flag_wait(pool_flag(un.item, 4u * un.half + s), p.ring_epoch, ws);
            if (mine == s) off = fw;
          }
        }
        off &= kFlagOffsetMask;
      } else {
        own_off += tot;
      }
      if (Q > 4u) {
        const uint64_t v = own_off;
        own_off = own_off_2;
        own_off_2 = v;
      }
      bytes = 0;
      if (tot) {
        const DecSegment& sg = p.seg[4u * un.half + mine];
        src = reinterpret_cast<uintptr_t>(sg.in) + off;
        if (off + tot <= sg.in_size) {
          bytes = (((uint32_t)src & 15u) + tot + 15u) & ~15u;
        } else {  // stream shorter than its rate bytes imply (or the offset never came)
          if (part == 0u && off != kFlagOffsetMask) note_error(ws.ctrl, kErrTruncated);
          un.rates = 0;
          before = 0;
        }
      }
    }
    // room: the streams that are left, or as many of them as there is room for
    uint32_t ends = mine >= done ? bytes : 0u;
    uint32_t v = __shfl_up_sync(0xffffffffu, ends, 8);
    if (mine >= 1u) ends += v;
    v = __shfl_up_sync(0xffffffffu, ends, 16);
    if (mine >= 2u) ends += v;
    const uint32_t all = __shfl_sync(0xffffffffu, ends, 31);
    uint32_t at = staged ? live_end : 0u, space = kSumUsable - at;
    if (staged && all > space && (all <= live_at || live_at > space)) {
      at = 0;
      space = live_at;
    }
    uint32_t end = many, used = all;
    if (__builtin_expect(all > space, 0)) {
      end = (uint32_t)(__ffs((int)__ballot_sync(0xffffffffu, ends > space)) - 1) >> 3;
      if (end <= done) return false;  // (not with an empty ring)
      used = __shfl_sync(0xffffffffu, ends, 8 * (int)end - 1);
    }
    uint64_t* const bar = &full[jobs & 1u];
    fence_proxy_async();  // what used to be in these bytes has been read
    if (lane == 0) {
      if (used) mbar_expect_tx(bar, used);
      else mbar_arrive(bar);
    }
    __syncwarp();
    const uint32_t start = at + ends - bytes;
    if (part == 0u && bytes && mine >= done && mine < end)
      bulk_load(ring + start, reinterpret_cast<const uint8_t*>(src & ~uint64_t(15)), bytes, bar);
    live_at = at;
    live_end = at + used;
    ++jobs;
    b.rates = un.rates;
    b.pos = start + ((uint32_t)src & 15u) + before;
    b.begin = done;
    b.end = end;
    b.sub = un.sub;
    b.first = un.half == 0u && done == 0u;
    b.last = end == many && 4u * un.half + end == Q;
    done = end;
    open = end < many;
    return true;
  };

  // ---- adding up -----------------------------------------------------------------------------------------------------
  PlaneSum acc;  // of this lane's block
  bool announced = pool == 0u;
  if (tid == 0) HC_PH(0);
  uint32_t landed = 0;  // batches whose payloads have landed
  const uint32_t ahead = (1u << (8u * (lane & 3u))) - 1u;  // rate bytes of the blocks of a word in front of the lane's
  const DecSegment& out = p.seg[0];
  for (;;) {
    if (staged < 2u && (open || next.item != kNoTile)) {
      Batch b;
      if (stage(b)) {
        if (staged == 0u) cur = b;
        else nxt = b;
        ++staged;
        continue;
      }
    }
    if (!announced) {
      // offsets of the sub-tiles of this run that others may take, counted back from its end; after the first bulk
      // copies have been issued, so that it delays nothing
      announced = true;
#pragma unroll 1
      for (uint32_t q = mine; q - mine < Q; q += 4u) {
        uint64_t off = before_me(q) + s_tot[warp][q];
#pragma unroll 2
        for (uint32_t k = pool; k-- > 0u;) {
          const uint32_t r4 = q < Q ? load_rates4(p.seg[q].in, p.seg[q].in_size, (uint64_t)(own_end + k) * kSubBlocks + 4u * part) : 0u;
          off -= sum8(payload_len4(r4));
          if (part == 0u && q < Q) st_relaxed_gpu_u64(pool_flag(k * nw + gw, q), flag_pack(p.ring_epoch, off));
        }
      }
    }
    if (tid == 0) HC_PH(1);
    if (staged == 0u) break;
    uint32_t rates = __shfl_sync(0xffffffffu, cur.rates, (int)(8u * cur.begin + (lane >> 2)));
    uint32_t pos = __shfl_sync(0xffffffffu, cur.pos, (int)(8u * cur.begin + (lane >> 2)));
    if (!warp_wait(&full[landed & 1u], (landed >> 1) & 1u, ws, kSiteDecodeInFull)) break;
    ++landed;
    if (tid == 0) HC_PH(2);
    if (cur.first) sum_clear(acc);
#pragma unroll 1
    for (uint32_t s = cur.begin; s < cur.end; ++s) {
      const uint32_t rate = rates >> (8u * (lane & 3u)) & 0xffu, at = pos + payload_len4(rates & ahead);
      rates = __shfl_sync(0xffffffffu, cur.rates, (int)(8u * s + 8u + (lane >> 2)));  // (past the last one: unused)
      pos = __shfl_sync(0xffffffffu, cur.pos, (int)(8u * s + 8u + (lane >> 2)));
      sum_add(acc, ring, masks, at, rate);
    }
    __syncwarp();
    if (tid == 0) HC_PH(3);
    if (cur.last) {
      uint32_t w[32];
      sum_values(acc, p.scale, p.eb, w);
      if (tid == 0) HC_PH(4);
      const uint64_t first = (uint64_t)cur.sub * kSubValues;
      if (lane == 0) tma_wait_group_read<0>();  // the rows of a turn ago have left the buffer
      __syncwarp();
      store_row_swizzled(obuf, (int)lane, w);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && out.use_tma && first + kBlock <= out.n) {
        tma_store_2d(&tmaps.m[0], 0, (int)(cur.sub * kSubBlocks), obuf);
        tma_commit_group();
      }
      if (!(out.use_tma && first + kSubValues <= out.n) && first < out.n) store_rows(obuf, out, first);
    }
    cur = nxt;
    --staged;
    if (tid == 0) {
      HC_PH(5);
      HC_PH_COUNT();
    }
  }
  // after a wait that ran out: nothing may land in shared memory once the CTA has left it
  for (; landed < jobs; ++landed) mbar_wait_bounded(&full[landed & 1u], (landed >> 1) & 1u, ws.spin_limit_ns);
  if (lane == 0) tma_wait_group<0>();
  if (lane == 0) HC_STAMP_MAX(7);
  if (pool) cta_epilogue(ws.tick);
}

// ---- one stand-alone stream ----------------------------------------------------------------------------------------
// The payloads of a warp's run lie behind one another in the stream, so they are staged as what they are: one sequence of bytes,
// in pieces of kPiece through a ring of four, whatever the sub-tiles in it are.  Staging sub-tile by sub-tile took half of the
// 700 instructions that a sub-tile cost (its own copy, barrier, room in the ring and bounds).  A sub-tile of a pool is a
// sequence of its own and begins at a piece.  Bytes are counted through the ring from 0 on (a "place"), place modulo kRing is
// where they are; the first kMirror bytes of the ring stand once more behind its end, so that a block reads on across it.
constexpr uint32_t kPiece = 1536, kRing = 4 * kPiece, kMirror = 160;
constexpr int kRunWarpBytes = kSubBytes + (int)(kRing + kMirror);
constexpr int kRunWarps = 20;
static_assert(32 * 132 + 15 <= 1 + 3 * kPiece, "a payload touches four pieces at most");
static_assert(132 + 8 <= kMirror, "a block and what read_planes looks at behind it");

template <int MODE>
__global__ void __launch_bounds__(kRunWarps * 32, 1)
hc_decode_run_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ DecParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t s_full[kRunWarps][4];
  __shared__ uint32_t s_tot[kRunWarps];
  __shared__ __align__(64) uint32_t masks[kMaskPitch * kMaskRows];
  __shared__ uint64_t s_pre;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n_warps = blockDim.x >> 5;
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* const obuf = smem + warp * kSubBytes;
  uint8_t* const ring = smem + n_warps * kSubBytes + warp * (kRing + kMirror);
  const Workspace& ws = p.ws;
  uint64_t* const full = s_full[warp];
  if (lane < 4u) mbar_init(&full[lane], 1);
  fence_mbar_init();
  if (tid == 0) launch_dependents();
  fill_masks<kMaskRows>(masks);
  grid_dependency_wait();  // nothing in global memory is touched before (see launch_overlapped)
  __syncwarp();
  const DecSegment& sg = p.seg[0];
  const uint8_t* const in = sg.in;
  const uint32_t gw = blockIdx.x * n_warps + warp, nw = gridDim.x * n_warps;
  HC_TL_DECL(ws.epoch);
  if (tid == 0) {
    HC_TL_ZERO();
    HC_STAMP(0);
    HC_PH_START();
  }

  // ---- shares, offsets -----------------------------------------------------------------------------------------------
  // What the first payload waits for, one after the other: rate bytes, total of the CTA, exchange.  Nothing else stands in
  // between: a 64-bit division by the number of warps, a look at the status and the sums of the pool did, and the first payload of
  // a 64 MB array was asked for after 6.1 us
  const uint32_t pool = p.pool;  // sub-tiles at the end of every run that are handed out one by one
  auto run_of = [&](uint32_t w) -> uint32_t { return p.run_all * w + (w < p.run_more ? w : p.run_more); };
  const uint32_t run_begin = run_of(gw), run_end = run_of(gw + 1u);
  const uint32_t own_end = run_end - pool;
  const uint4 rates = rates16(in, sg.in_size, run_begin, run_end, lane);  // of 16 sub-tiles, and of the next 16
  const uint4 rates_2 = run_end - run_begin > 16u ? rates16(in, sg.in_size, run_begin, run_end, lane + 32u) : make_uint4(0, 0, 0, 0);
  const uint32_t status = *((volatile const uint32_t*)(ws.ctrl + 2));
  auto rate_of = [&](uint32_t sub) -> uint32_t {
    const uint64_t b = (uint64_t)sub * kSubBlocks + lane;
    return b < sg.in_size ? ld_cg_u8(in + b) : 0u;
  };
  // items: own sub-tiles, then tickets of the pools (kPool set)
  constexpr uint32_t kPool = 0x80000000u;
  uint32_t it = run_begin, tk_raw = kNoTile;
  const uint32_t n_tickets = pool * nw;
  auto ask = [&]() {
    if (lane == 0) tk_raw = atomicAdd(ws.tick, 1u);
  };
  auto next_item = [&]() -> uint32_t {
    if (it < own_end) {
      const uint32_t i = it++;
      if (it == own_end && pool) ask();
      return i;
    }
    if (!pool) return kNoTile;
    const uint32_t t = __shfl_sync(0xffffffffu, tk_raw, 0);
    if (t >= n_tickets) return kNoTile;
    ask();
    return t | kPool;
  };
  // ticket t is the (t / nw)-th pool sub-tile of warp t % nw
  auto sub_of = [&](uint32_t item) -> uint32_t {
    if (!(item & kPool)) return item;
    const uint32_t w = (item & ~kPool) % nw, k = (item & ~kPool) / nw;
    return run_of(w + 1u) - pool + k;
  };
  uint32_t sub = run_begin, rate = run_begin < run_end ? rate_of(run_begin) : 0u;  // (a pool is smaller than its run)
  uint32_t sum = payload_len16(rates), own = run_begin + (lane >> 1) < own_end ? sum : 0u;
#pragma unroll 1
  for (uint32_t l = lane + 64u; run_begin * kSubBlocks + 16u * l < run_end * kSubBlocks; l += 32u) {
    const uint32_t s = payload_len16(rates16(in, sg.in_size, run_begin, run_end, l));
    sum += s;
    if (run_begin + (l >> 1) < own_end) own += s;
  }
  const uint32_t sum_2 = payload_len16(rates_2);
  sum += sum_2;
  if (run_begin + 16u + (lane >> 1) < own_end) own += sum_2;
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) s_tot[warp] = sum;
  __syncthreads();
  const uint32_t tot_of = lane < n_warps ? s_tot[lane] : 0u;  // of warp `lane`; sums in two halves of 16 bits
  auto sum64 = [&](uint32_t v) -> uint64_t {
    return __reduce_add_sync(0xffffffffu, v & 0xffffu) + ((uint64_t)__reduce_add_sync(0xffffffffu, v >> 16) << 16);
  };
  if (warp == 0) {
    give_total_of(ws.sums + kSumWords, sum64(tot_of));
    const uint64_t pre = take_total_of(ws.sums + kSumWords, ws);
    if (lane == 0) s_pre = pre;
  }
  uint64_t own_base = rate_bytes(sg.n) + sum64(lane < warp ? tot_of : 0u);  // byte of the stream where this warp's run begins
  const uint32_t own_bytes = __reduce_add_sync(0xffffffffu, own);           // payload bytes of its own sub-tiles
  __syncthreads();
  own_base += s_pre;
  // (an earlier launch that timed out, and nobody has cleared its status: no output)
  uint32_t item = status >= (uint32_t)kErrTimeout ? kNoTile : next_item();

  // ---- staging -------------------------------------------------------------------------------------------------------
  const uint8_t* f_src = in;  // the next bytes to be staged, 16-byte aligned
  uint32_t f_left = 0;        // of the sequence that is being staged
  uint32_t issued = 0, landed = 0, freed = 0;  // pieces asked for, waited for, and read
  auto pump = [&]() {
    if (lane == 0) fence_proxy_async();  // what used to be in the bytes has been read
#pragma unroll 1
    while (f_left && issued - freed < 4u) {
      const uint32_t bytes = f_left < kPiece ? f_left : kPiece;
      if (lane == 0) {
        uint64_t* const bar = &full[issued & 3u];
        uint8_t* const dst = ring + (issued & 3u) * kPiece;
        // (nothing lies in front of the very first piece that could read on into it)
        const uint32_t again = (issued & 3u) || !issued ? 0u : bytes < kMirror ? bytes : kMirror;
        mbar_expect_tx(bar, bytes + again);
        bulk_load(dst, f_src, bytes, bar);
        if (again) bulk_load(ring + kRing, f_src, again, bar);
      }
      f_src += bytes;
      f_left -= bytes;
      ++issued;
    }
  };
  uint32_t limit = 0;  // place up to which the sequence has bytes (the stream may end before its rate bytes say so)
  // a sequence of `bytes` bytes from byte `off` of the stream: place of its first byte
  auto begin = [&](uint64_t off, uint32_t bytes) -> uint32_t {
    const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(in) + off) & 15u;
    const uint32_t place = issued * kPiece + phase;
    const uint32_t there = off >= sg.in_size ? 0u : sg.in_size - off < bytes ? (uint32_t)(sg.in_size - off) : bytes;
    f_src = in + off - phase;
    f_left = there ? (phase + there + 15u) & ~15u : 0u;
    limit = place + there;
    return place;
  };
  uint32_t at = item == kNoTile ? 0u : begin(own_base, own_bytes);  // place of the current item's payload
  pump();
  uint32_t next = item == kNoTile ? kNoTile : next_item(), next_sub = 0, next_rate = 0;
  uint64_t next_flag = 0;  // lane 0's look at the payload offset of a pool item
  auto look = [&]() {
    if (next == kNoTile) return;
    next_sub = sub_of(next);
    next_rate = rate_of(next_sub);
    if (next & kPool && lane == 0) next_flag = ld_relaxed_gpu_u64(p.flags + (next & ~kPool));
  };
  look();
  bool announced = pool == 0u;
  if (tid == 0) HC_PH(0);

  while (item != kNoTile) {
    const uint32_t len = payload_len(rate);
    const uint32_t inc = warp_inclusive_scan(len);
    const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
    if (tot && at + tot > limit) {  // stream shorter than its rate bytes imply
      if (lane == 0) note_error(ws.ctrl, kErrTruncated);
      rate = 0;
    } else {
      bool gave_up = false;
      while (landed * kPiece < at + tot && landed < issued) {
        gave_up = !warp_wait(&full[landed & 3u], (landed >> 2) & 1u, ws, kSiteDecodeInFull);
        if (gave_up) break;
        ++landed;
      }
      if (gave_up) break;
    }
    if (tid == 0) HC_PH(2);
    uint32_t pos = at % kRing + inc - len;
    if (pos >= kRing) pos -= kRing;
    uint32_t T[32], sign, a0;
    decode_rows<12>(ring, masks, pos, rate, plane_width(__reduce_max_sync(0xffffffffu, rate & 31u)), sign, a0, T);
    const bool little = (rate & 31u) <= 16u && a0 < (1u << 23);
    const uint32_t cur = sub;
    __syncwarp();
    if (tid == 0) HC_PH(3);
    // ---- what comes next: its payload begins here, or is a sequence of its own
    item = next;
    if (item != kNoTile) {
      sub = next_sub;
      rate = next_rate;
      if (item & kPool) {
        while (landed < issued && warp_wait(&full[landed & 3u], (landed >> 2) & 1u, ws, kSiteDecodeInFull)) ++landed;
        freed = landed;
        uint64_t fw = __shfl_sync(0xffffffffu, next_flag, 0);
        if (!flag_matches(fw, p.ring_epoch)) fw = own_flag_wait(p.flags + (item & ~kPool), p.ring_epoch, ws);
        at = begin(fw & kFlagOffsetMask, __reduce_add_sync(0xffffffffu, payload_len(rate)));
      } else {
        at += tot;
        freed = at / kPiece;
      }
      pump();
      next = next_item();
      look();
    }
    if (tid == 0) HC_PH(1);

    // ---- signs, prefix sum, scaling --------------------------------------------------------------------------------
    uint32_t w[32];
    constexpr int S = MODE == kModeVec ? 4 : 1;
    if (p.scale != 0.0f && __all_sync(0xffffffffu, little)) {
      float qv[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        qv[i] = __fmaf_rn(as_f(T[i ^ 7]), sign_scale(sign, i), i >= S ? qv[i - S] : 0.0f);
        w[i] = as_u(__fmul_rn(qv[i], p.scale));
      }
    } else {
      int32_t qv[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int32_t m = (int32_t)(sign << i) >> 31;
        qv[i] = (i >= S ? qv[i - S] : 0) + ((int32_t)T[i ^ 7] ^ m) - m;
        w[i] = as_u(__fmul_rn(__fmul_rn((float)qv[i], p.eb), 2.0f));
      }
    }
    if (tid == 0) HC_PH(4);
    // ---- out -------------------------------------------------------------------------------------------------------
    if (lane == 0) tma_wait_group_read<0>();  // the rows of a turn ago have left the buffer
    __syncwarp();
    store_row_swizzled(obuf, (int)lane, w);
    fence_proxy_async();
    __syncwarp();
    const uint64_t first = (uint64_t)cur * kSubValues;
    if (lane == 0 && sg.use_tma && first + kBlock <= sg.n) {
      tma_store_2d(&tmaps.m[0], 0, (int)(cur * kSubBlocks), obuf);
      tma_commit_group();
    }
    if (!(sg.use_tma && first + kSubValues <= sg.n) && first < sg.n) store_rows(obuf, sg, first);
    if (!announced) {
      // offsets of the sub-tiles of this run that others may take, counted back from its end; after the first own one, so that it
      // delays nothing (in front of it, 2.3 us at 256 MB)
      announced = true;
      uint64_t off = own_base + sum;
#pragma unroll 1
      for (uint32_t k = pool; k-- > 0u;) {
        off -= __reduce_add_sync(0xffffffffu, payload_len(rate_of(own_end + k)));
        if (lane == 0) st_relaxed_gpu_u64(p.flags + (k * nw + gw), flag_pack(p.ring_epoch, off));
      }
    }
    if (tid == 0) {
      HC_PH(5);
      HC_PH_COUNT();
    }
  }
  // after a wait that ran out: nothing may land in shared memory once the CTA has left it
  for (; landed < issued; ++landed) mbar_wait_bounded(&full[landed & 3u], (landed >> 2) & 1u, ws.spin_limit_ns);
  if (lane == 0) tma_wait_group<0>();
  if (lane == 0) HC_STAMP_MAX(7);
  if (pool) cta_epilogue(ws.tick);
}

}  // namespace dev

// ---- host side ---------------------------------------------------------------------------------------------

namespace {

template <int MODE, bool SUM>
cudaError_t launch_flagged(const TensorMaps& maps, DecParams p, cudaStream_t stream, bool overlap) {
  const auto kernel = dev::hc_decode_step_kernel<MODE, SUM>;
  constexpr int kWarps = dev::kDecWarps, kSmem = kWarps * dev::kDecWarpBytes + 1024;
  static thread_local int cache[64] = {};
  const int cap = resident_ctas(kernel, 32 * kWarps, kSmem, cache);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  // tickets are quarters of a tile while there is a warp for each
  const uint32_t tiles = SUM ? p.tiles_per_seg : p.n_tiles;
  p.parts = tiles <= (uint32_t)cap ? 4u : 1u;
  const uint32_t ctas = p.parts == 4u ? tiles : (tiles + 3u) / 4u;
  const int grid = (int)(ctas < (uint32_t)cap ? ctas : (uint32_t)cap);
  if (overlap) return launch_overlapped(kernel, grid, 32 * kWarps, kSmem, stream, maps, p);
  kernel<<<grid, 32 * kWarps, kSmem, stream>>>(maps, p);
  return cudaGetLastError();
}

// stand-alone: one stream (hc_decode_run_kernel) or the sum of several (hc_decode_kernel)
template <typename Kernel>
cudaError_t launch_runs(Kernel kernel, int max_warps, int warp_bytes, int (&cache)[64], const TensorMaps& maps, DecParams p, cudaStream_t stream) {
  auto smem = [&](int warps) { return warps * warp_bytes + 1024; };
  const int cap = resident_ctas(kernel, 32 * max_warps, smem(max_warps), cache);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  const uint64_t subs = (p.seg[0].n + dev::kSubValues - 1) / dev::kSubValues;
  const RunSplit split = split_runs(subs, (uint32_t)(cap < kMaxCtas ? cap : kMaxCtas), (uint32_t)max_warps);
  if (run_words(split, p.n_seg) > p.ws.words) return cudaErrorInvalidValue;
  p.pool = split.pool;
  p.flags = p.ws.st_a;
  p.run_all = (uint32_t)(subs / (split.grid * split.warps));
  p.run_more = (uint32_t)(subs % (split.grid * split.warps));
  return launch_overlapped(kernel, (int)split.grid, 32 * (int)split.warps, smem((int)split.warps), stream, maps, p);
}
template <int MODE>
cudaError_t launch_run(const TensorMaps& maps, const DecParams& p, cudaStream_t stream) {
  static thread_local int cache[64] = {};
  return launch_runs(dev::hc_decode_run_kernel<MODE>, dev::kRunWarps, dev::kRunWarpBytes, cache, maps, p, stream);
}
cudaError_t launch_sum(const TensorMaps& maps, const DecParams& p, cudaStream_t stream) {
  static thread_local int cache[64] = {};
  return launch_runs(dev::hc_decode_kernel, dev::kSumWarps, dev::kSumWarpBytes, cache, maps, p, stream);
}
template <int MODE>
cudaError_t launch_one(const TensorMaps& maps, const DecParams& p, cudaStream_t stream, bool overlap) {
  return p.seg[0].in_ready ? launch_flagged<MODE, false>(maps, p, stream, overlap) : launch_run<MODE>(maps, p, stream);
}

}  // namespace

// Either every segment has arrival flags or none has; without flags there is one segment, or `sum`.
cudaError_t launch_decode(int mode, DecParams p, cudaStream_t stream, bool overlap) {
  if (p.n_seg == 0 || p.n_seg > (uint32_t)kMaxDst) return cudaErrorInvalidValue;
  uint64_t n_max = 0;
  for (uint32_t i = 0; i < p.n_seg; ++i) {
    n_max = p.seg[i].n > n_max ? p.seg[i].n : n_max;
    if ((p.seg[i].in_ready != nullptr) != (p.seg[0].in_ready != nullptr)) return cudaErrorInvalidValue;
  }
  if (n_max == 0) return cudaSuccess;
  if (!p.sum && p.n_seg > 1 && !p.seg[0].in_ready) return cudaErrorInvalidValue;
  p.tiles_per_seg = (uint32_t)((n_max + kTileElems - 1) / kTileElems);
  p.n_tiles = p.tiles_per_seg * p.n_seg;
  if (!p.seg[0].in_ready) p.ring_epoch = p.ws.epoch;  // tag of the launch's own flag words
  // (q * eb) * 2 rounds once (the factor 2 is exact) as long as q * eb is a normal number
  p.scale = p.eb >= 0x1p-120f && p.eb <= 0x1p90f ? p.eb * 0x1p24f : 0.0f;
  TensorMaps maps;
  memset(&maps, 0, sizeof(maps));
  const uint32_t outs = p.sum ? 1u : p.n_seg;
  for (uint32_t i = 0; i < outs; ++i)
    p.seg[i].use_tma = make_rows_map(&maps.m[i], p.seg[i].out, p.seg[i].n / kBlock, dev::kSubBlocks) ? 1u : 0u;
  if (p.sum) {
    // one output: every stream must describe the same array
    for (uint32_t i = 1; i < p.n_seg; ++i)
      if (p.seg[i].n != p.seg[0].n) return cudaErrorInvalidValue;
    if (mode == kModeVec) return cudaErrorInvalidValue;
    return p.seg[0].in_ready ? launch_flagged<kModeOutlier, true>(maps, p, stream, overlap) : launch_sum(maps, p, stream);
  }
  switch (mode) {
    case kModeOutlier:
    case kModePlain: return launch_one<kModeOutlier>(maps, p, stream, overlap);
    case kModeVec: return launch_one<kModeVec>(maps, p, stream, overlap);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hc

HC_TL_READ(hc_debug_timeline_decode)
