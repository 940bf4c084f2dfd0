// stream -> fp32 (decompress, its flagged and multi-stream forms): kernel and launcher.
//
// A unit of work is a SUB-TILE: 32 consecutive blocks (1024 values, 4 KB of fp32), one block per lane, a quarter
// of a tile.  Every warp works alone: payloads come by bulk copy into a byte ring of its own; the decoded 4 KB go to an output
// buffer (128-byte swizzle) and leave through a TMA tiled store.  Inside the loop no warp waits for another one.
//
// Stand-alone streams (hc_decode_run_kernel; RUNS, the sum of several): every warp of the grid owns a contiguous run of
// sub-tiles.  It sums the payload lengths of its run from the rate bytes (700 bytes for a 256 MB array), the CTAs (one per SM, so
// at most 148) exchange their totals once through the workspace, and from there on a warp carries its own running offset: no
// look-back, no second kernel.  The SMs do not run at the same pace (with equal static shares the first warp of a 256 MB launch
// finished at 42 us, the last at 70), so the last eighth of every run goes to whoever is free first; the payload
// offsets of those sub-tiles are written to the workspace after the first one has been decoded.
// What bounds the decode of one stream: 256 MB the memory (62.1 us; 61.9 with the arithmetic left out, 50.4 without the stores), 64 MB
// the memory and the start (22.8; 20.8, 19.0), smaller ones the way to the first payload: rate bytes, exchange, payload, one trip to
// L2 after the other (8 MB: of 6.1 us on the device 3.3; 5.1 of 7.5 when 64-bit divisions, the status and the offsets of the pool
// stood in between).  Sums take their streams one after the other in every warp and add them as bit planes (four streams of 256 MB
// 233 us by way of a row for every stream, 198 this way; seven of 40 MB 80 and 67; four of 4 MB 12.0 and 10.7).
//
// Steps of a collective (!RUNS): the producer raises one flag word per tile, carrying the tile's payload offset.
// Tickets are dealt in the order in which the flags rise, round the segments: a tile (all four quarters by one
// warp, its rate bytes scanned once), or a quarter of a tile while the GPU holds a warp for each.
#include "hc_host.cuh"
#include "hc_launch.h"
#include "hc_timeline.cuh"
#include "hc_warp.cuh"

namespace hc {
namespace dev {

// Warps of a CTA at most, 20 (96 registers a thread) or 16 (128) on an SM.  Stand-alone: one CTA per SM, so that the totals
// of at most 148 CTAs are exchanged.  Steps of a collective: CTAs of four warps, which slip into an SM one by one
// while the CTAs of the step before leave it.
__host__ __device__ constexpr int dec_max_warps(bool runs) { return runs ? 16 : 4; }
__host__ __device__ constexpr int dec_ctas(bool sum, bool runs) { return runs ? 1 : sum ? 4 : 5; }
// payload ring of a warp: the largest payload of corrupt rate bytes (32 x 132) with its 16-byte phase, and in
// front of the ring's end what read_planes may look at behind a payload
constexpr int kDecRing = 6144;
constexpr int kDecRingUsable = kDecRing - 160;
constexpr int kDecWarpBytes = kSubBytes + kDecRing;
static_assert(32 * 132 + 32 <= kDecRingUsable, "one payload must fit");

// What the TMA unit cannot store of a sub-tile: the ragged last row (not part of the tensor map), or everything when the array is
// not 16-byte aligned
static __device__ __noinline__ void store_rows(const uint8_t* rows, const DecSegment& sg, uint64_t first) {
  const uint32_t len = sg.n - first < kSubValues ? (uint32_t)(sg.n - first) : (uint32_t)kSubValues;
#pragma unroll 1
  for (uint32_t e = (sg.use_tma ? len / kBlock * kBlock : 0u) + (threadIdx.x & 31u); e < len; e += 32u)
    sg.out[first + e] = as_f(lds32((swizzled_row(rows, (int)(e >> 5)) ^ ((e & 28u) << 2)) | ((e & 3u) << 2)));
  __syncwarp();
}

// SUM: the n_seg streams hold contributions to ONE array; a warp stages the same sub-tile of every stream in
// turn, adds the deltas in registers, as bit planes, and writes seg[0].out once.
template <int MODE, bool SUM, bool RUNS>
__global__ void __launch_bounds__(dec_max_warps(RUNS) * 32, dec_ctas(SUM, RUNS))
hc_decode_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ DecParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t s_full[dec_max_warps(RUNS)][4];
  __shared__ uint32_t s_tot[dec_max_warps(RUNS)][kMaxDst];  // payload bytes of a run; RUNS
  __shared__ uint64_t s_pre[kMaxDst];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n_warps = blockDim.x >> 5;
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* const obuf = smem + warp * kSubBytes;
  uint8_t* const ring = smem + n_warps * kSubBytes + warp * kDecRing;
  const Workspace& ws = p.ws;
  uint64_t* const full = s_full[warp];
  if (lane < 4u) mbar_init(&full[lane], 1);
  fence_mbar_init();
  if (tid == 0) launch_dependents();
  if (RUNS) grid_dependency_wait();  // nothing in global memory is touched before (see launch_overlapped)
  __syncwarp();

  const uint32_t Q = SUM ? p.n_seg : 1u;  // streams per sub-tile
  const uint32_t gw = blockIdx.x * n_warps + warp, nw = gridDim.x * n_warps;
  static_assert(SUM || !RUNS, "one stand-alone stream: hc_decode_run_kernel");
  const uint32_t status = *((volatile const uint32_t*)(ws.ctrl + 2));

  // A job is a sub-tile of one stream.  Its ITEM is a sub-tile (RUNS) or a tile; items are known one ahead, so that
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

  // ---- RUNS: shares, offsets -----------------------------------------------------------------------------------------
  auto run_of = [&](uint32_t w) -> uint32_t { return p.run_all * w + (w < p.run_more ? w : p.run_more); };
  const uint32_t pool = p.pool;  // sub-tiles at the end of every run that are handed out one by one
  uint32_t it = 0, it_end = 0;   // this warp's own sub-tiles still to be staged
  uint64_t run_base = 0;         // lane q: payload offset of the next one in stream q
  uint32_t run_end = 0;
  if (RUNS) {
    it = run_of(gw);
    run_end = run_of(gw + 1u);
    it_end = run_end - pool;
    // Payload bytes of the run in every stream.  Runs of up to four sub-tiles: eight lanes a stream, four streams at a time (a
    // load per stream, its code eight times over, took 0.5 us more where all is start-up)
    if (p.run_all + (p.run_more ? 1u : 0u) <= 4u) {
      const uint32_t l = lane & 7u, q0 = lane >> 3, q1 = q0 + 4u;
      uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
      if (q0 < Q) v0 = rates16(p.seg[q0].in, p.seg[q0].in_size, it, run_end, l);
      if (q1 < Q) v1 = rates16(p.seg[q1].in, p.seg[q1].in_size, it, run_end, l);
      uint32_t s0 = payload_len16(v0), s1 = payload_len16(v1);  // below 2^16 each: 4 * 32 * 132 at most
      s0 |= s1 << 16;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (l == 0) {
        s_tot[warp][q0] = s0 & 0xffffu;
        s_tot[warp][q1] = s0 >> 16;
      }
    } else {
      // Longer runs: 16 sub-tiles of four streams are asked for before the first is added (one stream after the other: eight of
      // 40 MB 96.0 us, 92.6 this way; four of 256 MB 240.9 and 237.1; two of 128 MB 70.4 and 70.0)
#pragma unroll 1
      for (uint32_t q4 = 0; q4 < Q; q4 += 4u) {
        uint32_t sum[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (uint32_t l = lane; it * kSubBlocks + 16u * l < run_end * kSubBlocks; l += 32u) {
          uint4 v[4];
#pragma unroll
          for (uint32_t u = 0; u < 4u; ++u)
            v[u] = q4 + u < Q ? rates16(p.seg[q4 + u].in, p.seg[q4 + u].in_size, it, run_end, l) : make_uint4(0, 0, 0, 0);
#pragma unroll
          for (uint32_t u = 0; u < 4u; ++u) sum[u] += payload_len16(v[u]);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
          sum[u] = __reduce_add_sync(0xffffffffu, sum[u]);
          if (lane == 0) s_tot[warp][q4 + u] = sum[u];  // (room for kMaxDst streams, a multiple of four)
        }
      }
    }
  }
  // ---- tickets: sub-tiles of the pools (RUNS), tiles or quarters (!RUNS) -----------------------------------------------
  const bool small = p.parts == 4u;
  const uint32_t n_tickets = RUNS ? pool * nw : (SUM ? p.tiles_per_seg : p.n_tiles) * p.parts;
  const bool dynamic = RUNS ? pool != 0u : n_tickets > nw;
  // !RUNS: the first half of the tickets is dealt out in turn, the rest comes from the counter (one address for all
  // warps: it answers a request every few cycles)
  const uint32_t rounds = n_tickets / nw, dealt = RUNS ? 0u : (rounds > 2u ? rounds / 2u + 1u : rounds);
  uint32_t asked = 0, tk_raw = kNoTile;  // tickets asked for; lane 0 (all lanes if dealt): the newest answer
  auto ask = [&]() {
    if (asked < dealt || (!RUNS && !dynamic)) tk_raw = asked * nw + gw;
    else if (lane == 0) tk_raw = dealt * nw + atomicAdd(ws.tick, 1u);
    ++asked;
  };
  auto answer = [&]() -> uint32_t {
    const uint32_t t = __shfl_sync(0xffffffffu, tk_raw, 0);
    return t < n_tickets ? t : kNoTile;
  };
  // items: RUNS: own sub-tiles, then pool tickets (kPool set); !RUNS: tickets
  constexpr uint32_t kPool = 0x80000000u;
  auto next_item = [&]() -> uint32_t {
    if (RUNS && it < it_end) {
      const uint32_t i = it++;
      if (it == it_end && dynamic) ask();
      return i;
    }
    if (RUNS && !dynamic) return kNoTile;
    const uint32_t t = answer();
    if (t == kNoTile) return t;
    if (!RUNS || dynamic) ask();
    return RUNS ? t | kPool : t;
  };
  auto tile_at = [&](uint32_t t) -> uint32_t { return small ? t >> 2 : t; };
  auto seg_at = [&](uint32_t t, uint32_t qq) -> uint32_t { return SUM ? qq : tile_at(t) % p.n_seg; };
  auto local_tile = [&](uint32_t t) -> uint32_t { return SUM ? tile_at(t) : tile_at(t) / p.n_seg; };
  // RUNS: sub-tile and flag word of pool ticket t: the (t / nw)-th pool sub-tile of warp t % nw
  auto pool_sub = [&](uint32_t t) -> uint32_t {
    const uint32_t w = (t & ~kPool) % nw, k = (t & ~kPool) / nw;
    return run_of(w + 1u) - pool + k;
  };
  auto pool_flag = [&](uint32_t t, uint32_t qq) -> uint64_t* { return p.flags + (size_t)qq * pool * nw + (t & ~kPool); };

  struct Unit {
    uint64_t flag;  // lane 0's look at the flag
    uint32_t raw;   // RUNS: the rate byte of the lane's block; !RUNS: those of four blocks of the tile
    uint32_t sub;   // RUNS: the sub-tile
    bool raw_ok;    // raw has been asked for (behind a collective's flag only once it is up)
  };
  auto load_raw = [&](uint32_t t, uint32_t qq, uint32_t sub) -> uint32_t {
    const DecSegment& sg = p.seg[seg_at(t, qq)];
    if (RUNS) {
      const uint64_t b = (uint64_t)sub * kSubBlocks + lane;
      return b < sg.in_size ? ld_cg_u8(sg.in + b) : 0u;
    }
    return load_rates4(sg.in, sg.in_size, (uint64_t)local_tile(t) * kTileBlocks + 4u * lane);
  };
  auto prime = [&](Unit& u, uint32_t t, uint32_t qq) {
    u = Unit{0ull, 0u, 0u, true};
    if (t == kNoTile) return;
    const DecSegment& sg = p.seg[seg_at(t, qq)];
    if (RUNS) {
      u.sub = t & kPool ? pool_sub(t) : t;
      if (t & kPool && lane == 0) u.flag = ld_relaxed_gpu_u64(pool_flag(t, qq));
      u.raw = load_raw(t, qq, u.sub);
    } else if ((uint64_t)local_tile(t) * kTileElems >= sg.n) {
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
  if (!RUNS) ask();
  // (an earlier launch that timed out, and nobody has cleared its status: no output)
  uint32_t tk = status >= (uint32_t)kErrTimeout ? kNoTile : next_item(), tk_next = tk == kNoTile ? kNoTile : next_item();
  Unit un, un_next{0ull, 0u, 0u, true};
  uint32_t r = small ? tk & 3u : 0u, q = 0;  // !RUNS: quarter; stream of the next job
  prime(un, tk, 0u);
  if (RUNS) {
    __syncthreads();
    for (uint32_t qq = warp; qq < Q; qq += n_warps)
      give_total_of(ws.sums + (1u + qq) * kSumWords, warp_sum_u64(lane < n_warps ? s_tot[lane][qq] : 0ull));
    for (uint32_t qq = warp; qq < Q; qq += n_warps) {
      const uint64_t pre = take_total_of(ws.sums + (1u + qq) * kSumWords, ws);
      if (lane == 0) s_pre[qq] = pre;
    }
    __syncthreads();
    if (lane < Q) {
      run_base = rate_bytes(p.seg[0].n) + s_pre[lane];
      for (uint32_t w = 0; w < warp; ++w) run_base += s_tot[w][lane];
    }
  }
  uint64_t fw = 0;              // flag word of the current unit (~0: gave up, or nothing there)
  uint32_t excl = 0, inc = 0;   // !RUNS: scan of the payload lengths of the current tile
  bool scanned = false;

  // stages the next job; false: flag still down (unless `block`), or no room in the ring
  auto produce = [&](Staged& st, bool busy, bool block) -> bool {
    const DecSegment& sg = p.seg[seg_at(tk, q)];
    uint32_t tot, at;
    uint64_t off;
    if (!scanned) {
      if (RUNS) {
        if (tk & kPool) {
          fw = __shfl_sync(0xffffffffu, un.flag, 0);
          if (!flag_matches(fw, p.ring_epoch)) fw = own_flag_wait(pool_flag(tk, q), p.ring_epoch, ws);
        }
        const uint32_t len = payload_len(un.raw);
        inc = warp_inclusive_scan(len, (int)lane);
        excl = inc - len;
      } else {
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
        if (!un.raw_ok) un.raw = load_raw(tk, q, 0u);
        const uint32_t sum = payload_len4(un.raw);
        inc = warp_inclusive_scan(sum, (int)lane);
        excl = inc - sum;
      }
      scanned = true;
      // the next unit's flag and rate bytes are on their way while this one is worked on
      if (SUM && q + 1 < Q) prime(un_next, tk, q + 1);
      else if (SUM && !RUNS && !small && r < 3u) prime(un_next, tk, 0u);
      else prime(un_next, tk_next, 0u);
    } else if (!RUNS && !un_next.raw_ok && r >= 2u) {
      const uint64_t f = __shfl_sync(0xffffffffu, un_next.flag, 0);
      if (flag_matches(f, p.ring_epoch)) {
        un_next.raw = load_raw(tk_next, 0u, 0u);
        un_next.raw_ok = true;
      }
    }
    if (RUNS) {
      tot = __shfl_sync(0xffffffffu, inc, 31);
      st.rate = un.raw;
      st.pos = excl;
      st.sub = un.sub;
      off = tk & kPool ? fw & kFlagOffsetMask : __shfl_sync(0xffffffffu, run_base, (int)q);
    } else {
      const uint32_t before = __shfl_sync(0xffffffffu, excl, 8 * (int)r);
      tot = __shfl_sync(0xffffffffu, inc, 8 * (int)r + 7) - before;
      const int src = 8 * (int)r + (int)(lane >> 2);
      const uint32_t k8 = 8u * (lane & 3u);
      const uint32_t r4 = __shfl_sync(0xffffffffu, un.raw, src);
      st.pos = __shfl_sync(0xffffffffu, excl, src) - before + payload_len4(r4 & ((1u << k8) - 1u));
      st.rate = (r4 >> k8) & 0xffu;
      st.sub = local_tile(tk) * 4u + r;
      off = (fw & kFlagOffsetMask) + before;
    }
    if (!ring_room(tot ? tot + 31u : 0u, busy, at)) return false;
    if (RUNS && !(tk & kPool) && lane == q) run_base += tot;
    uint32_t take = tot;
    if ((RUNS ? (tk & kPool) != 0u : true) && (fw & kFlagOffsetMask) == kFlagOffsetMask) {
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
      scanned = !SUM && !RUNS;
      if (!RUNS && !small && r < 3u) {
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
  bool announced = !RUNS || pool == 0u;
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
    if (!announced) {
      // offsets of the sub-tiles of this run that others may take, counted back from its end; after the first bulk
      // copies have been issued, so that it delays nothing
      announced = true;
      for (uint32_t qq = 0; qq < Q; ++qq) {
        const DecSegment& sg = p.seg[qq];
        uint64_t off = rate_bytes(sg.n) + s_pre[qq];
        for (uint32_t w = 0; w <= warp; ++w) off += s_tot[w][qq];
        for (uint32_t k = pool; k-- > 0u;) {
          const uint32_t len = payload_len(load_raw(0u, qq, run_end - pool + k));
          off -= __reduce_add_sync(0xffffffffu, len);
          if (lane == 0) st_relaxed_gpu_u64(pool_flag(k * nw + gw, qq), flag_pack(p.ring_epoch, off));
        }
      }
    }
    if (threadIdx.x == 0) HC_PH(1);
    if (staged == 0u) break;
    if (!warp_wait(&full[v & 3u], (v >> 2) & 1u, ws, kSiteDecodeInFull)) break;
    ++v;
    if (threadIdx.x == 0) HC_PH(2);
    constexpr int S = MODE == kModeVec ? 4 : 1;
    bool last = true;
    uint32_t w[32];
    if (SUM) {
      if (cur.seg == 0) sum_clear(acc);
      sum_add(acc, ring, cur.pos, cur.rate);
      __syncwarp();
      if (threadIdx.x == 0) HC_PH(3);
      last = cur.seg + 1 == Q;
      if (last) sum_values<S>(acc, p.scale, p.eb, w);
    } else {
      const int W = plane_width(__reduce_max_sync(0xffffffffu, cur.rate & 31u));
      uint32_t T[32], sign, a0;
      decode_rows(ring, cur.pos, cur.rate, W, sign, a0, T);
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
      if (!(sg.use_tma && first + kSubValues <= sg.n) && first < sg.n) {
        // the ragged last row (not part of the tensor map), or everything when the array is not 16-byte aligned
        const uint32_t len = sg.n - first < kSubValues ? (uint32_t)(sg.n - first) : (uint32_t)kSubValues;
#pragma unroll 1
        for (uint32_t e = (sg.use_tma ? len / kBlock * kBlock : 0u) + lane; e < len; e += 32u)
          sg.out[first + e] = as_f(lds32((swizzled_row(obuf, (int)(e >> 5)) ^ ((e & 28u) << 2)) | ((e & 3u) << 2)));
        __syncwarp();
      }
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
    const uint32_t inc = warp_inclusive_scan(len, (int)lane);
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
    decode_rows(ring, pos, rate, plane_width(__reduce_max_sync(0xffffffffu, rate & 31u)), sign, a0, T);
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

constexpr int dec_smem(int warps) { return warps * dev::kDecWarpBytes + 1024; }

template <int MODE, bool SUM, bool RUNS>
cudaError_t launch_t(const TensorMaps& maps, DecParams p, cudaStream_t stream, bool overlap) {
  constexpr int kWarps = dev::dec_max_warps(RUNS);
  static thread_local int cache[64] = {};
  const int cap = resident_ctas(dev::hc_decode_kernel<MODE, SUM, RUNS>, 32 * kWarps, dec_smem(kWarps), cache);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  uint32_t warps;
  int grid;
  if (RUNS) {
    const uint64_t subs = (p.seg[0].n + dev::kSubValues - 1) / dev::kSubValues;
    const RunSplit split = split_runs(subs, (uint32_t)(cap < kMaxCtas ? cap : kMaxCtas), (uint32_t)kWarps);
    if (run_words(split, p.n_seg) > p.ws.words) return cudaErrorInvalidValue;
    warps = split.warps;
    grid = (int)split.grid;
    p.run_all = (uint32_t)(subs / (split.grid * split.warps));
    p.run_more = (uint32_t)(subs % (split.grid * split.warps));
    p.pool = split.pool;
    p.flags = p.ws.st_a;
  } else {
    // tickets are quarters of a tile while there is a warp for each
    const uint32_t tiles = SUM ? p.tiles_per_seg : p.n_tiles;
    warps = (uint32_t)kWarps;
    p.parts = tiles <= (uint32_t)cap ? 4u : 1u;
    const uint32_t ctas = p.parts == 4u ? tiles : (tiles + 3u) / 4u;
    grid = (int)(ctas < (uint32_t)cap ? ctas : (uint32_t)cap);
  }
  const int block = 32 * (int)warps, smem = dec_smem((int)warps);
  if (overlap || RUNS) return launch_overlapped(dev::hc_decode_kernel<MODE, SUM, RUNS>, grid, block, smem, stream, maps, p);
  dev::hc_decode_kernel<MODE, SUM, RUNS><<<grid, block, smem, stream>>>(maps, p);
  return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_run(const TensorMaps& maps, DecParams p, cudaStream_t stream) {
  static thread_local int cache[64] = {};
  auto smem = [](int warps) { return warps * dev::kRunWarpBytes + 1024; };
  const int cap = resident_ctas(dev::hc_decode_run_kernel<MODE>, 32 * dev::kRunWarps, smem(dev::kRunWarps), cache);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  const uint64_t subs = (p.seg[0].n + dev::kSubValues - 1) / dev::kSubValues;
  const RunSplit split = split_runs(subs, (uint32_t)(cap < kMaxCtas ? cap : kMaxCtas), (uint32_t)dev::kRunWarps);
  if (run_words(split, 1) > p.ws.words) return cudaErrorInvalidValue;
  p.pool = split.pool;
  p.flags = p.ws.st_a;
  p.run_all = (uint32_t)(subs / (split.grid * split.warps));
  p.run_more = (uint32_t)(subs % (split.grid * split.warps));
  return launch_overlapped(dev::hc_decode_run_kernel<MODE>, (int)split.grid, 32 * (int)split.warps, smem((int)split.warps), stream, maps, p);
}

template <int MODE, bool SUM>
cudaError_t launch_solo(const TensorMaps& maps, const DecParams& p, cudaStream_t stream) {
  if constexpr (SUM) return launch_t<MODE, true, true>(maps, p, stream, false);
  else return launch_run<MODE>(maps, p, stream);
}
template <int MODE, bool SUM>
cudaError_t launch_f(const TensorMaps& maps, const DecParams& p, cudaStream_t stream, bool overlap) {
  return p.seg[0].in_ready ? launch_t<MODE, SUM, false>(maps, p, stream, overlap)
                           : launch_solo<MODE, SUM>(maps, p, stream);
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
    return launch_f<kModeOutlier, true>(maps, p, stream, overlap);
  }
  switch (mode) {
    case kModeOutlier:
    case kModePlain: return launch_f<kModeOutlier, false>(maps, p, stream, overlap);
    case kModeVec: return launch_f<kModeVec, false>(maps, p, stream, overlap);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hc

HC_TL_READ(hc_debug_timeline_decode)
