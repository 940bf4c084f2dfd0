// Warp- and CTA-level helpers of the codec kernels: status words, bounded waits, rate bytes -> payload offsets.
#pragma once
#include "hc_block.cuh"
#include "hc_kernels.cuh"

namespace hc {
namespace dev {

constexpr uint32_t kNoTile = 0xffffffffu;
// sub-tile: 32 consecutive blocks, one per lane; what a warp works on at a time
constexpr int kSubBlocks = 32;
constexpr int kSubValues = kSubBlocks * kBlock;
constexpr int kSubBytes = kSubValues * 4;  // 4096

__device__ __forceinline__ void note_error(uint32_t* ctrl, uint32_t code) { atomicMax(ctrl + 2, code); }
// timeouts and peer failures end the launch early; capacity / truncation errors only skip data
__device__ __forceinline__ bool fatal_error(const uint32_t* ctrl) {
  return *((volatile const uint32_t*)(ctrl + 2)) >= (uint32_t)kErrTimeout;
}

// which wait ran out; the first one is kept in ctrl[3] (hc_codec_status_site), because every later time-out of
// the launch is only a consequence of it
enum WaitSite : uint32_t {
  kSiteLoaderStageFree = 1, kSiteLoaderInFree = 2, kSiteComputeInFull = 3, kSiteComputeTile = 4, kSiteComputeRing = 5,
  kSiteScannerTotal = 6, kSiteCopierBase = 7, kSiteDecodeInFull = 10, kSiteLookBack = 11,  // (8 and 9 belonged to roles that no longer exist)
};
__device__ __forceinline__ void note_timeout(const Workspace& ws, uint32_t site) {
  if (!fatal_error(ws.ctrl)) atomicCAS(ws.ctrl + 3, 0u, site);
  note_error(ws.ctrl, kErrTimeout);
}
// Bounded mbarrier wait of a whole warp; false: gave up (recorded).  The lanes try together and vote, so that the loop is the same
// for all of them: as a loop per lane every wait carried the code for lanes that leave it apart (a sub-tile of an add 1237 warp
// instructions, 1206 this way; compress of 4 KB 3.84 us and 3.75, of 256 MB 63.6 and 62.4, decode of 64 MB 22.8 and 22.4).  Compress of
// 16 MB takes 7.35 us, 7.2 with a loop per lane in the wait for the rows alone, but then 4 KB 3.84 and 256 MB 63.2; from 8 to 32 MB no
// other size was found to lose.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, const Workspace& ws, uint32_t site) {
  if (__builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, parity)), 1)) return true;
  long long t0 = 0;
#pragma unroll 1
  for (uint32_t it = 0; !__all_sync(0xffffffffu, mbar_try_wait(bar, parity)); ++it) {
    if ((it & 63u) == 0u) {
      const long long now = clock64();
      if (it == 0u) t0 = now;
      else if (__any_sync(0xffffffffu, now - t0 > (long long)ws.spin_limit_ns * 2) || it >= (1u << 26)) {
        if ((threadIdx.x & 31) == 0) note_timeout(ws, site);
        return false;
      }
    }
  }
  return true;
}

// collective steps: one non-blocking look at the tile's arrival flag; 0 = not raised yet
__device__ __forceinline__ uint64_t flag_peek(const uint64_t* flag, uint32_t call) {
  uint64_t w = 0;
  if ((threadIdx.x & 31) == 0) {
    w = ld_acquire_sys_u64(flag);
    if (!flag_matches(w, call)) w = 0;
  }
  return __shfl_sync(0xffffffffu, w, 0);
}
// collective steps: bounded wait for the tile's arrival flag; 0 = the peer never delivered
__device__ __forceinline__ uint64_t flag_wait_warp(const uint64_t* flag, uint32_t call, const Workspace& ws) {
  uint64_t w = 0;
  if ((threadIdx.x & 31) == 0) {
    w = wait_tile_flag(flag, call, ws.spin_limit_ns, ws.ctrl + 2);
    if (w == 0) note_error(ws.ctrl, kErrPeer);
  }
  return __shfl_sync(0xffffffffu, w, 0);
}

// bounded wait for a flag that some CTA of the same launch writes; ~0: gave up
__device__ __forceinline__ uint64_t own_flag_wait(const uint64_t* flag, uint32_t tag, const Workspace& ws) {
  uint64_t w = 0;
  if ((threadIdx.x & 31) == 0) {
    const long long t0 = clock64();
    const long long limit_clk = (long long)ws.spin_limit_ns * 2;
    for (uint32_t it = 0; it < (1u << 24); ++it) {
      w = ld_relaxed_gpu_u64(flag);
      if (flag_matches(w, tag)) break;
      w = ~0ull;
      __nanosleep(100);
      if ((it & 15u) == 15u && (clock64() - t0 > limit_clk || fatal_error(ws.ctrl))) break;
    }
    if (w == ~0ull) note_timeout(ws, kSiteLookBack);
  }
  return __shfl_sync(0xffffffffu, w, 0);
}

// ---- rate bytes -> offsets ------------------------------------------------------------------------------
// rate bytes b .. b+3 of a stream as a word; bytes past the end of the stream count as 0
__device__ __forceinline__ uint32_t load_rates4(const uint8_t* in, uint64_t in_size, uint64_t b) {
  if (b + 4 <= in_size && ((reinterpret_cast<uintptr_t>(in) + b) & 3u) == 0)
    return __ldcg(reinterpret_cast<const uint32_t*>(in + b));
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (b + k < in_size) r |= ld_cg_u8(in + b + k) << (8 * k);
  return r;
}

// the 16 rate bytes at `at` of a stream that is not aligned, or that ends among them (out of line: every caller has the code
// for aligned ones next to the call)
static __device__ __noinline__ uint4 rates16_any(const uint8_t* in, uint64_t in_size, uint64_t at) {
  return make_uint4(load_rates4(in, in_size, at), load_rates4(in, in_size, at + 4u), load_rates4(in, in_size, at + 8u),
                    load_rates4(in, in_size, at + 12u));
}
// rate bytes [16 l, 16 l + 16) of the sub-tiles [a, b) of a stream; 0 past b and past the end of the stream
__device__ __forceinline__ uint4 rates16(const uint8_t* in, uint64_t in_size, uint32_t a, uint32_t b, uint32_t l) {
  const uint64_t at = (uint64_t)a * kSubBlocks + 16u * l;
  if (at >= (uint64_t)b * kSubBlocks) return make_uint4(0, 0, 0, 0);
  if ((reinterpret_cast<uintptr_t>(in) & 15u) == 0 && at + 16u <= in_size) return ld_cg_u4(in + at);
  return rates16_any(in, in_size, at);
}
__device__ __forceinline__ uint32_t payload_len16(const uint4& v) {
  return payload_len4(v.x) + payload_len4(v.y) + payload_len4(v.z) + payload_len4(v.w);
}

// Sum of the totals words[0 .. n) of chunks of this launch (n <= kMaxCtas, a total below 2^24 each), one warp; polls until all
// are there (bounded).  Out of line, because it is the clerk's in more than one place and compute warps share its cache.
static __device__ __noinline__ uint32_t sum_totals(const uint64_t* words, uint32_t n, const Workspace& ws) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t tag = (uint32_t)(st_pack(kStAgg, ws.epoch, 0) >> 32);
  long long t0 = 0;
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 24); ++it) {
    uint64_t w[kMaxCtas / 32];
    uint32_t sum = 0;
    bool ready = true;
#pragma unroll
    for (int u = 0; u < kMaxCtas / 32; ++u) w[u] = lane + 32u * u < n ? ld_relaxed_gpu_u64(words + lane + 32u * u) : (uint64_t)tag << 32;
#pragma unroll
    for (int u = 0; u < kMaxCtas / 32; ++u) {
      ready = ready && (uint32_t)(w[u] >> 32) == tag;
      sum += (uint32_t)w[u];
    }
    if (__all_sync(0xffffffffu, ready)) return __reduce_add_sync(0xffffffffu, sum);
    if (it == 0u) t0 = clock64();
    if ((it & 15u) == 15u && __any_sync(0xffffffffu, clock64() - t0 > (long long)ws.spin_limit_ns * 2 || fatal_error(ws.ctrl))) break;
  }
  if (lane == 0) note_timeout(ws, kSiteLookBack);
  return 0;
}

// Exclusive sum over one total per CTA, by pushing: each CTA adds its total to a word of every later CTA (at most 147
// reductions, five a lane; sum in [47:0], number of totals in [63:48]), and polls nothing but its own word until it is
// complete.  Everybody reading everybody's published word instead costs 2.7 us from the last store to the last reader
// at 148 CTAs, because the polls of all of them queue up on ten L2 lines; this way decode of 256 MB went from 67.4 us to
// 63.3, a sum of four 4 MB streams from 16.9 to 14.4.  It is right for one exchange per launch only: with a push for every
// chunk of a compress of 256 MB the reductions themselves are the queue (70 us, 63 with published words).
__device__ __forceinline__ void give_total(uint64_t* sums, uint64_t total) {
  for (uint32_t j = blockIdx.x + 1u + (threadIdx.x & 31u); j < gridDim.x; j += 32u)
    atomicAdd(reinterpret_cast<unsigned long long*>(sums + j), (1ull << 48) | total);
}
// sum of the totals of all CTAs before this one; leaves the word zero for the next launch
__device__ __forceinline__ uint64_t take_total(uint64_t* sums, const Workspace& ws) {
  uint64_t* const word = sums + blockIdx.x;
  uint64_t w = 0;
  if ((threadIdx.x & 31u) == 0u && blockIdx.x) {
    w = ld_relaxed_gpu_u64(word);
    if (w >> 48 != blockIdx.x) {
      const long long t0 = clock64();
      const long long limit_clk = (long long)ws.spin_limit_ns * 2;
      for (uint32_t it = 0; it < (1u << 26); ++it) {
        w = ld_relaxed_gpu_u64(word);
        if (w >> 48 == blockIdx.x) break;
        if ((it & 15u) == 15u && (clock64() - t0 > limit_clk || fatal_error(ws.ctrl))) {
          note_timeout(ws, kSiteLookBack);
          break;
        }
      }
    }
    st_relaxed_gpu_u64(word, 0);
  }
  return __shfl_sync(0xffffffffu, w & ((1ull << 48) - 1), 0);
}

// The same for more than kDirect CTAs, in groups of kSumGroup: a total goes to the later CTAs of its group and to one word for
// each later group, at most one reduction a lane where the direct form has up to 147 words to add to, whose 10900 reductions a
// launch queue up (148 CTAs: the last one had given 1.5 us after it knew its total, 0.4 us this way; decode of 8 MB 7.2 us and
// 6.4, sum of four 4 MB streams 13.4 and 12.7).  In a launch of few CTAs, and in the one-round launches of the encode kernel, it
// is no faster and its longer code costs 0.2 to 0.4 us (seven streams of 8 MB added 18.7 us, 19.5 this way; sum of two streams
// in 56 CTAs 6.7 us, 7.3 this way; in 123 CTAs 9.2 and 7.9).
// The word of a group has several readers and is never reset: what counts is by how much it has grown since the launch
// before, whose end every CTA notes for itself (the last one of a launch also for those of its group that the launch does not have).
constexpr uint32_t kDirect = 64;
__device__ __forceinline__ void give_total_grouped(uint64_t* sums, uint64_t total) {
  const uint32_t lane = threadIdx.x & 31u, g = blockIdx.x / kSumGroup;
  const uint32_t cta = blockIdx.x + 1u + lane, group = lane - 16u;
  uint64_t* const to = lane < 16u ? sums + cta : sums + kMaxCtas + group;
  if (lane < 16u ? cta < (g + 1u) * kSumGroup && cta < gridDim.x : group > g && group * kSumGroup < gridDim.x)
    atomicAdd(reinterpret_cast<unsigned long long*>(to), (1ull << 48) | total);
}
__device__ __forceinline__ uint64_t take_total_grouped(uint64_t* sums, const Workspace& ws) {
  const uint32_t lane = threadIdx.x & 31u, g = blockIdx.x / kSumGroup;
  uint64_t* const word = lane ? sums + kMaxCtas + g : sums + blockIdx.x;
  uint64_t* const noted = sums + kMaxCtas + 16;
  const uint32_t want = lane == 0u ? blockIdx.x - g * kSumGroup : lane == 1u ? g * kSumGroup : 0u;
  const uint64_t before = lane == 1u ? ld_relaxed_gpu_u64(noted + blockIdx.x) : 0ull;
  uint64_t w = before;
  if (want) {
    long long t0 = 0;
#pragma unroll 1
    for (uint32_t it = 0;; ++it) {
      w = ld_relaxed_gpu_u64(word);
      if ((w - before) >> 48 == want) break;
      if (it == 0u) t0 = clock64();
      if ((it & 15u) == 15u && (clock64() - t0 > (long long)ws.spin_limit_ns * 2 || it >= (1u << 26) || fatal_error(ws.ctrl))) {
        note_timeout(ws, kSiteLookBack);
        break;
      }
    }
    st_relaxed_gpu_u64(lane ? noted + blockIdx.x : word, lane ? w : 0ull);
  }
  const uint64_t all = (w - before) & ((1ull << 48) - 1);
  if (blockIdx.x + 1u == gridDim.x) {
    const uint64_t group = __shfl_sync(0xffffffffu, w, 1);
    const uint32_t cta = blockIdx.x + 1u + lane;
    if (g && cta < (g + 1u) * kSumGroup && cta < (uint32_t)kMaxCtas) st_relaxed_gpu_u64(noted + cta, group);
  }
  return __shfl_sync(0xffffffffu, all, 0) + __shfl_sync(0xffffffffu, all, 1);
}
// decode: by the number of CTAs
__device__ __forceinline__ void give_total_of(uint64_t* sums, uint64_t total) {
  if (gridDim.x <= kDirect) give_total(sums, total);
  else give_total_grouped(sums, total);
}
__device__ __forceinline__ uint64_t take_total_of(uint64_t* sums, const Workspace& ws) {
  return gridDim.x <= kDirect ? take_total(sums, ws) : take_total_grouped(sums, ws);
}

// What the TMA unit cannot store of a sub-tile: the ragged last row (not part of the tensor map), or everything when the array is
// not 16-byte aligned
static __device__ __noinline__ void store_rows(const uint8_t* rows, const DecSegment& sg, uint64_t first) {
  const uint32_t len = sg.n - first < kSubValues ? (uint32_t)(sg.n - first) : (uint32_t)kSubValues;
#pragma unroll 1
  for (uint32_t e = (sg.use_tma ? len / kBlock * kBlock : 0u) + (threadIdx.x & 31u); e < len; e += 32u)
    sg.out[first + e] = as_f(lds32((swizzled_row(rows, (int)(e >> 5)) ^ ((e & 28u) << 2)) | ((e & 3u) << 2)));
  __syncwarp();
}

// the last CTA to leave re-arms the ticket counter for the next launch (true in thread 0 of that CTA)
__device__ __forceinline__ bool cta_epilogue(uint32_t* tick) {
  __syncthreads();
  bool last = false;
  if (threadIdx.x == 0) {
    __threadfence();
    uint32_t done = atomicAdd(tick + 1, 1u);
    if (done == gridDim.x - 1) {
      tick[0] = 0;
      tick[1] = 0;
      __threadfence();
      last = true;
    }
  }
  return last;
}

}  // namespace dev
}  // namespace hc
