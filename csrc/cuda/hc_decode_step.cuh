// stream -> fp32 in the steps of a collective: the kernel.
//
// The producer raises one flag word per tile, carrying the tile's payload offset.  Tickets are dealt in the order in which the flags
// rise, round the segments: a tile (all four quarters by one warp, its rate bytes scanned once), or a quarter of a tile while the GPU
// holds a warp for each.  A quarter is a sub-tile (see hc_decode.cu); every warp works alone.
#pragma once
#include "hc_timeline.cuh"
#include "hc_warp.cuh"

namespace hc {
namespace dev {

// CTAs of four warps, which slip into an SM one by one while the CTAs of the step before leave it: 20 warps (96 registers a
// thread) or, in sums, 16 (128) on an SM
constexpr int kDecWarps = 4;
// payload ring of a warp: the largest payload of corrupt rate bytes (32 x 132) with its 16-byte phase, and in
// front of the ring's end what read_planes and sum_add may look at behind a payload
constexpr int kDecRing = 6144;
constexpr int kDecRingUsable = kDecRing - 160;
constexpr int kDecWarpBytes = kSubBytes + kDecRing;
static_assert(32 * 132 + 32 <= kDecRingUsable, "one payload must fit");
static_assert(kSumReads <= kDecRing - kDecRingUsable, "sum_add reads on behind a payload");

// Steps of a collective.  SUM: the n_seg streams hold contributions to ONE array; a warp stages the same sub-tile of every stream in
// turn, adds the deltas in registers, as bit planes, and writes seg[0].out once.
template <int MODE, bool SUM>
__global__ void __launch_bounds__(kDecWarps * 32, SUM ? 4 : 5)
hc_decode_step_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ DecParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t s_full[kDecWarps][4];
  __shared__ __align__(64) uint32_t masks[kMaskPitch * (SUM ? kSumMaskRows : kMaskRows)];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n_warps = blockDim.x >> 5;
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* const obuf = smem + warp * kSubBytes;
  uint8_t* const ring = smem + n_warps * kSubBytes + warp * kDecRing;
  const Workspace& ws = p.ws;
  uint64_t* const full = s_full[warp];
  if (lane < 4u) mbar_init(&full[lane], 1);
  fence_mbar_init();
  if (tid == 0) launch_dependents();
  fill_masks<SUM ? kSumMaskRows : kMaskRows>(masks);
  __syncthreads();

  const uint32_t Q = SUM ? p.n_seg : 1u;  // streams per sub-tile
  const uint32_t gw = blockIdx.x * n_warps + warp, nw = gridDim.x * n_warps;
  const uint32_t status = *((volatile const uint32_t*)(ws.ctrl + 2));

  // A job is a sub-tile of one stream.  Its ITEM is a tile, or a quarter of one; items are known one ahead, so that
  // the next one's rate bytes and flag are asked for a job or more before they are looked at.
  struct Staged {
    uint32_t rate;  // rate byte of this lane's block (0: nothing staged for it)
    uint32_t pos;   // its byte position in the ring
    uint32_t sub;   // sub-tile inside the segment
    uint32_t seg;   // segment; SUM: number of the stream
  };
  uint32_t live_at = 0, live_end = 0;  // ring bytes of the newest staged payload
  uint32_t jobs = 0;                   // staged so far
  // room for a payload of `bytes` bytes, `busy`: the newest staged payload has not been read yet
  auto ring_room = [&](uint32_t bytes, bool busy, uint32_t& at) -> bool {
    at = busy ? live_end : 0u;
    if (at + bytes > (uint32_t)kDecRingUsable) {
      at = 0;
      if (bytes > live_at) return false;
    }
    return true;
  };
  // bulk copy of the payload bytes [off, off + tot) of a stream to ring byte `at`; sets rate and pos of the lane's block
  auto issue = [&](const DecSegment& sg, uint64_t off, uint32_t tot, uint32_t at, Staged& st) {
    const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(sg.in) + off) & 15u;
    const uint32_t bytes = tot ? (phase + tot + 15u) & ~15u : 0u;
    live_at = at;
    live_end = at + bytes;
    uint64_t* const bar = &full[jobs & 3u];
    if (lane == 0) {
      if (tot) {
        fence_proxy_async();  // what used to be in these bytes has been read
        mbar_expect_tx(bar, bytes);
        bulk_load(ring + at, sg.in + off - phase, bytes, bar);
      } else {
        mbar_arrive(bar);
      }
    }
    ++jobs;
    if (!tot) st.rate = 0;
    st.pos += at + phase;
  };

  // ---- tickets: tiles or quarters ---------------------------------------------------------------------------------------
  const bool small = p.parts == 4u;
  const uint32_t n_tickets = (SUM ? p.tiles_per_seg : p.n_tiles) * p.parts;
  const bool dynamic = n_tickets > nw;
  // the first half of the tickets is dealt out in turn, the rest comes from the counter (one address for all
  // warps: it answers a request every few cycles)
  const uint32_t rounds = n_tickets / nw, dealt = rounds > 2u ? rounds / 2u + 1u : rounds;
  uint32_t asked = 0, tk_raw = kNoTile;  // tickets asked for; lane 0 (all lanes if dealt): the newest answer
  auto ask = [&]() {
    if (asked < dealt || !dynamic) tk_raw = asked * nw + gw;
    else if (lane == 0) tk_raw = dealt * nw + atomicAdd(ws.tick, 1u);
    ++asked;
  };
  auto next_item = [&]() -> uint32_t {
    const uint32_t t = __shfl_sync(0xffffffffu, tk_raw, 0);
    if (t >= n_tickets) return kNoTile;
    ask();
    return t;
  };
  auto tile_at = [&](uint32_t t) -> uint32_t { return small ? t >> 2 : t; };
  auto seg_at = [&](uint32_t t, uint32_t qq) -> uint32_t { return SUM ? qq : tile_at(t) % p.n_seg; };
  auto local_tile = [&](uint32_t t) -> uint32_t { return SUM ? tile_at(t) : tile_at(t) / p.n_seg; };

  struct Unit {
    uint64_t flag;  // lane 0's look at the flag
    uint32_t raw;   // the rate bytes of four blocks of the tile
    bool raw_ok;    // raw has been asked for (only once the flag is up)
  };
  auto load_raw = [&](uint32_t t, uint32_t qq) -> uint32_t {
    const DecSegment& sg = p.seg[seg_at(t, qq)];
    return load_rates4(sg.in, sg.in_size, (uint64_t)local_tile(t) * kTileBlocks + 4u * lane);
  };
  auto prime = [&](Unit& u, uint32_t t, uint32_t qq) {
    u = Unit{0ull, 0u, true};
    if (t == kNoTile) return;
    const DecSegment& sg = p.seg[seg_at(t, qq)];
    if ((uint64_t)local_tile(t) * kTileElems >= sg.n) {
      u.flag = ~0ull;  // past the end of a segment shorter than the longest one: nothing to read or to wait for
    } else {
      if (lane == 0) u.flag = ld_acquire_sys_u64(sg.in_ready + local_tile(t));
      u.raw_ok = false;
    }
  };
  HC_TL_DECL(ws.epoch);
  if (threadIdx.x == 0) {
    HC_TL_ZERO();
    HC_STAMP(0);
    HC_PH_START();
  }
  ask();
  // (an earlier launch that timed out, and nobody has cleared its status: no output)
  uint32_t tk = status >= (uint32_t)kErrTimeout ? kNoTile : next_item(), tk_next = tk == kNoTile ? kNoTile : next_item();
  Unit un, un_next{0ull, 0u, true};
  uint32_t r = small ? tk & 3u : 0u, q = 0;  // quarter, stream of the next job
  prime(un, tk, 0u);
  uint64_t fw = 0;              // flag word of the current unit (~0: gave up, or nothing there)
  uint32_t excl = 0, inc = 0;   // scan of the payload lengths of the current tile
  bool scanned = false;

  // stages the next job; false: flag still down (unless `block`), or no room in the ring
  auto produce = [&](Staged& st, bool busy, bool block) -> bool {
    const DecSegment& sg = p.seg[seg_at(tk, q)];
    if (!scanned) {
      fw = __shfl_sync(0xffffffffu, un.flag, 0);
      if (fw != ~0ull && !flag_matches(fw, p.ring_epoch)) {
        const uint64_t* flag = sg.in_ready + local_tile(tk);
        fw = block ? flag_wait_warp(flag, p.ring_epoch, ws) : flag_peek(flag, p.ring_epoch);
        if (fw == 0 && !block) return false;
        if (fw == 0) {
          fw = ~0ull;
          un.raw_ok = true;
        }
      }
      if (!un.raw_ok) un.raw = load_raw(tk, q);
      const uint32_t sum = payload_len4(un.raw);
      inc = warp_inclusive_scan(sum);
      excl = inc - sum;
      scanned = true;
      // the next unit's flag and rate bytes are on their way while this one is worked on
      if (SUM && q + 1 < Q) prime(un_next, tk, q + 1);
      else if (SUM && !small && r < 3u) prime(un_next, tk, 0u);
      else prime(un_next, tk_next, 0u);
    } else if (!un_next.raw_ok && r >= 2u) {
      const uint64_t f = __shfl_sync(0xffffffffu, un_next.flag, 0);
      if (flag_matches(f, p.ring_epoch)) {
        un_next.raw = load_raw(tk_next, 0u);
        un_next.raw_ok = true;
      }
    }
    const uint32_t before = __shfl_sync(0xffffffffu, excl, 8 * (int)r);
    const uint32_t tot = __shfl_sync(0xffffffffu, inc, 8 * (int)r + 7) - before;
    const int src = 8 * (int)r + (int)(lane >> 2);
    const uint32_t k8 = 8u * (lane & 3u);
    const uint32_t r4 = __shfl_sync(0xffffffffu, un.raw, src);
    st.pos = __shfl_sync(0xffffffffu, excl, src) - before + payload_len4(r4 & ((1u << k8) - 1u));
    st.rate = (r4 >> k8) & 0xffu;
    st.sub = local_tile(tk) * 4u + r;
    const uint64_t off = (fw & kFlagOffsetMask) + before;
    uint32_t at;
    if (!ring_room(tot ? tot + 31u : 0u, busy, at)) return false;
    uint32_t take = tot;
    if ((fw & kFlagOffsetMask) == kFlagOffsetMask) {
      take = 0;  // the producer gave up on the tile
    } else if (tot && off + tot > sg.in_size) {  // stream shorter than its rate bytes imply
      if (lane == 0) note_error(ws.ctrl, kErrTruncated);
      take = 0;
    }
    st.seg = seg_at(tk, q);
    issue(sg, off, take, at, st);
    // advance: next stream, next quarter, next item
    if (SUM && q + 1 < Q) {
      ++q;
      scanned = false;
    } else {
      q = 0;
      scanned = !SUM;
      if (!small && r < 3u) {
        ++r;
      } else {
        scanned = false;
        tk = tk_next;
        r = small ? tk & 3u : 0u;
        if (tk != kNoTile) tk_next = next_item();
      }
    }
    if (!scanned) un = un_next;
    return true;
  };

  // ---- consumer side -----------------------------------------------------------------------------------------------
  // one sub-tile is decoded while the payload of the next one lands; the one after is staged as soon as the first
  // has been read
  Staged cur{}, nxt{};
  uint32_t staged = 0;
  PlaneSum acc;  // SUM: of this lane's block
  if (threadIdx.x == 0) HC_PH(0);
  uint32_t v = 0;  // jobs whose payload has landed
  for (;;) {
    if (staged < 2u && tk != kNoTile) {
      Staged st;
      if (produce(st, staged != 0u, staged == 0u)) {
        if (staged == 0u) cur = st;
        else nxt = st;
        ++staged;
        continue;
      }
    }
    if (threadIdx.x == 0) HC_PH(1);
    if (staged == 0u) break;
    if (!warp_wait(&full[v & 3u], (v >> 2) & 1u, ws, kSiteDecodeInFull)) break;
    ++v;
    if (threadIdx.x == 0) HC_PH(2);
    bool last = true;
    uint32_t w[32];
    if constexpr (SUM) {
      if (cur.seg == 0) sum_clear(acc);
      sum_add(acc, ring, masks, cur.pos, cur.rate);
      __syncwarp();
      if (threadIdx.x == 0) HC_PH(3);
      last = cur.seg + 1 == Q;
      if (last) sum_values(acc, p.scale, p.eb, w);
    } else {
      constexpr int S = MODE == kModeVec ? 4 : 1;
      const int W = plane_width(__reduce_max_sync(0xffffffffu, cur.rate & 31u));
      uint32_t T[32], sign, a0;
      decode_rows<16>(ring, masks, cur.pos, cur.rate, W, sign, a0, T);
      __syncwarp();
      if (threadIdx.x == 0) HC_PH(3);
      // ---- signs, prefix sum, scaling ------------------------------------------------------------------------------
      const bool little = (cur.rate & 31u) <= 16u && a0 < (1u << 23);
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
    }
    if (last) {
      if (threadIdx.x == 0) HC_PH(4);
      // ---- out -------------------------------------------------------------------------------------------------------
      const uint32_t sgo = SUM ? 0u : cur.seg;
      const DecSegment& sg = p.seg[sgo];
      const uint64_t first = (uint64_t)cur.sub * kSubValues;
      if (lane == 0) tma_wait_group_read<0>();  // the rows of a turn ago have left the buffer
      __syncwarp();
      store_row_swizzled(obuf, (int)lane, w);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && sg.use_tma && first + kBlock <= sg.n) {
        tma_store_2d(&tmaps.m[sgo], 0, (int)(cur.sub * kSubBlocks), obuf);
        tma_commit_group();
      }
      if (!(sg.use_tma && first + kSubValues <= sg.n) && first < sg.n) store_rows(obuf, sg, first);
    }
    cur = nxt;
    --staged;
    if (threadIdx.x == 0) {
      HC_PH(5);
      HC_PH_COUNT();
    }
  }
  // after a wait that ran out: nothing may land in shared memory once the CTA has left it
  for (; v < jobs; ++v) mbar_wait_bounded(&full[v & 3u], (v >> 2) & 1u, ws.spin_limit_ns);
  if (lane == 0) tma_wait_group<0>();
  if (lane == 0) HC_STAMP_MAX(7);
  if (dynamic) cta_epilogue(ws.tick);
}


}  // namespace dev
}  // namespace hc
