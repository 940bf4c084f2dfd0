// stream -> fp32 (decompress, its flagged and multi-stream forms): kernel and launcher.
//
// A unit of work is a SUB-TILE: 32 consecutive blocks (1024 values, 4 KB of fp32), one block per lane, a quarter
// of a tile.  Every warp works alone: payloads come by bulk copy into a byte ring of its own (two or three
// typical payloads fit, one of the worst kind), up to two sub-tiles ahead; the decoded 4 KB go to an output
// buffer (128-byte swizzle) and leave through a TMA tiled store.  Inside the loop no warp waits for another one.
//
// Stand-alone streams (RUNS): every warp of the grid owns a contiguous run of sub-tiles.  It sums the payload lengths
// of its run from the rate bytes (700 bytes for a 256 MB array), the CTAs (one per SM, so at most 148) exchange their
// totals once through the workspace (about 2 us), and from there on a warp carries its own running offset: no
// look-back, no second kernel.  The SMs do not run at the same pace (with equal static shares the first warp of a 256 MB launch
// finished at 42 us, the last at 70), so the last eighth of every run goes to whoever is free first; the payload
// offsets of those sub-tiles are written to the workspace at the start.
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

// Warps of a CTA at most, 20 (96 registers a thread) or 16 (128) on an SM.  RUNS: one CTA per SM, so that the totals
// of at most 148 CTAs are exchanged.  Steps of a collective: CTAs of four warps, which slip into an SM one by one
// while the CTAs of the step before leave it.
__host__ __device__ constexpr int dec_max_warps(bool sum, bool runs) { return !runs ? 4 : sum ? 16 : 20; }
__host__ __device__ constexpr int dec_ctas(bool sum, bool runs) { return runs ? 1 : sum ? 4 : 5; }
// payload ring of a warp: the largest payload of corrupt rate bytes (32 x 132) with its 16-byte phase, and in
// front of the ring's end what read_planes may look at behind a payload
constexpr int kDecRing = 6144;
constexpr int kDecRingUsable = kDecRing - 160;
constexpr int kDecWarpBytes = kSubBytes + kDecRing;
static_assert(32 * 132 + 32 <= kDecRingUsable, "one payload must fit");

// SUM: the n_seg streams hold contributions to ONE array; a warp stages the same sub-tile of every stream in
// turn, adds the signed deltas in registers and writes seg[0].out once.
template <int MODE, bool SUM, bool RUNS>
__global__ void __launch_bounds__(dec_max_warps(SUM, RUNS) * 32, dec_ctas(SUM, RUNS))
hc_decode_kernel(const __grid_constant__ TensorMaps tmaps, const __grid_constant__ DecParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t s_full[dec_max_warps(SUM, RUNS)][4];
  __shared__ uint64_t s_tot[dec_max_warps(SUM, RUNS)][SUM ? kMaxDst : 1];
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
  const bool dead = fatal_error(ws.ctrl);  // an earlier launch timed out and nobody has cleared it: no output

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
  const uint32_t subs = (uint32_t)((p.seg[0].n + kSubValues - 1) / kSubValues);
  const uint32_t pool = p.pool;  // sub-tiles at the end of every run that are handed out one by one
  uint32_t it = 0, it_end = 0;   // this warp's own sub-tiles still to be staged
  uint64_t run_base = 0;         // lane q: payload offset of the next one in stream q
  uint32_t run_end = 0;
  uint4 rates[SUM && RUNS ? kMaxDst : 1];
  if (RUNS) {
    it = (uint32_t)((uint64_t)subs * gw / nw);
    run_end = (uint32_t)((uint64_t)subs * (gw + 1) / nw);
    it_end = run_end - pool;
#pragma unroll
    for (uint32_t qq = 0; qq < (SUM ? kMaxDst : 1); ++qq) rates[qq] = qq < Q ? rates16(p.seg[qq].in, p.seg[qq].in_size, it, run_end, lane) : make_uint4(0, 0, 0, 0);
  }
  const uint32_t run_begin = it;
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
  auto seg_at = [&](uint32_t t, uint32_t qq) -> uint32_t { return SUM ? qq : (RUNS ? 0u : tile_at(t) % p.n_seg); };
  auto local_tile = [&](uint32_t t) -> uint32_t { return SUM ? tile_at(t) : tile_at(t) / p.n_seg; };
  // RUNS: sub-tile and flag word of pool ticket t: the (t / nw)-th pool sub-tile of warp t % nw
  auto pool_sub = [&](uint32_t t) -> uint32_t {
    const uint32_t w = (t & ~kPool) % nw, k = (t & ~kPool) / nw;
    return (uint32_t)((uint64_t)subs * (w + 1) / nw) - pool + k;
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
  uint32_t tk = dead ? kNoTile : next_item(), tk_next = tk == kNoTile ? kNoTile : next_item();
  Unit un, un_next{0ull, 0u, 0u, true};
  uint32_t r = small ? tk & 3u : 0u, q = 0;  // !RUNS: quarter; stream of the next job
  prime(un, tk, 0u);
  if (RUNS) {
#pragma unroll
    for (uint32_t qq = 0; qq < (SUM ? kMaxDst : 1); ++qq) {
      if (qq >= Q) break;
      uint32_t sum = payload_len16(rates[qq]);
      for (uint32_t l = lane + 32u; run_begin * kSubBlocks + 16u * l < run_end * kSubBlocks; l += 32u)
        sum += payload_len16(rates16(p.seg[qq].in, p.seg[qq].in_size, run_begin, run_end, l));
      sum = __reduce_add_sync(0xffffffffu, sum);
      if (lane == 0) s_tot[warp][qq] = sum;
    }
    __syncthreads();
    for (uint32_t qq = warp; qq < Q; qq += n_warps)
      give_total(ws.sums + (1u + qq) * kMaxCtas, warp_sum_u64(lane < n_warps ? s_tot[lane][qq] : 0ull));
    for (uint32_t qq = warp; qq < Q; qq += n_warps) {
      const uint64_t pre = take_total(ws.sums + (1u + qq) * kMaxCtas, ws);
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
  float acc[32];       // SUM: deltas * 2^-23, or int32 bits once `ints`
  bool ints = false;
  uint32_t bound = 0;  // of |sum of the deltas| of this lane's block
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
    const int W = plane_width(__reduce_max_sync(0xffffffffu, cur.rate & 31u));
    uint32_t T[32], sign, a0;
    decode_rows(ring, cur.pos, cur.rate, W, sign, a0, T);
    __syncwarp();

    if (threadIdx.x == 0) HC_PH(3);
    // ---- signs, sum over the streams, prefix sum, scaling ----------------------------------------------------------
    uint32_t w[32];
    const bool little = (cur.rate & 31u) <= 16u && a0 < (SUM ? 1u << 20 : 1u << 23);
    bool exact = p.scale != 0.0f && __all_sync(0xffffffffu, little);
    constexpr int S = MODE == kModeVec ? 4 : 1;
    bool last = true;
    if (SUM) {
      if (cur.seg == 0) {
        ints = !exact;
        bound = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
      } else if (!ints && !exact) {
        ints = true;
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = __int_as_float(__float2int_rn(__fmul_rn(acc[i], 8388608.0f)));
      }
      if (!ints) {
        bound += a0 + (31u << (cur.rate & 31u));
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = __fmaf_rn(as_f(T[i ^ 7]), sign_scale(sign, i), acc[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int32_t m = (int32_t)(sign << i) >> 31;
          acc[i] = __int_as_float(__float_as_int(acc[i]) + ((int32_t)T[i ^ 7] ^ m) - m);
        }
      }
      last = cur.seg + 1 == Q;
      if (last && !ints && !__all_sync(0xffffffffu, bound < (1u << 24))) {
        ints = true;
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = __int_as_float(__float2int_rn(__fmul_rn(acc[i], 8388608.0f)));
      }
      exact = !ints;
    }
    if (last) {
      if (exact) {
        float qv[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float before = i >= S ? qv[i - S] : 0.0f;
          if (SUM) qv[i] = i >= S ? __fadd_rn(before, acc[i]) : acc[i];
          else qv[i] = __fmaf_rn(as_f(T[i ^ 7]), sign_scale(sign, i), before);
          w[i] = as_u(__fmul_rn(qv[i], p.scale));
        }
      } else {
        int32_t qv[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int32_t before = i >= S ? qv[i - S] : 0;
          if (SUM) {
            qv[i] = before + __float_as_int(acc[i]);
          } else {
            const int32_t m = (int32_t)(sign << i) >> 31;
            qv[i] = before + ((int32_t)T[i ^ 7] ^ m) - m;
          }
          w[i] = as_u(__fmul_rn(__fmul_rn((float)qv[i], p.eb), 2.0f));
        }
      }
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

}  // namespace dev

// ---- host side ---------------------------------------------------------------------------------------------

namespace {

constexpr int dec_smem(int warps) { return warps * dev::kDecWarpBytes + 1024; }

template <int MODE, bool SUM, bool RUNS>
cudaError_t launch_t(const TensorMaps& maps, DecParams p, cudaStream_t stream, bool overlap) {
  constexpr int kWarps = dev::dec_max_warps(SUM, RUNS);
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

template <int MODE, bool SUM>
cudaError_t launch_f(const TensorMaps& maps, const DecParams& p, cudaStream_t stream, bool overlap) {
  return p.seg[0].in_ready ? launch_t<MODE, SUM, false>(maps, p, stream, overlap)
                           : launch_t<MODE, SUM, true>(maps, p, stream, false);
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
