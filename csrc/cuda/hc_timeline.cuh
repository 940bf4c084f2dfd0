#pragma once
#include <cuda_runtime.h>

namespace hc {
namespace dev {

// Optional per-CTA timeline (compile with -DHC_TIMELINE): nanosecond stamps of the first tile's way
// through the roles (slots 0-15) and, for the first compute warp, SM-clock cycles accumulated per
// phase of the tile loop (slots 16-30) with the number of tiles in slot 31, for finding where a
// launch spends its time.  Not part of a normal build.  Every file with kernels has stamps of its own and a function
// (HC_TL_READ) that brings them to the host.
#ifdef HC_TIMELINE
constexpr int kTlSlots = 32;
static __device__ unsigned long long g_timeline[4 * 1024 * kTlSlots];  // [launch epoch & 3][CTA][slot]
__device__ __forceinline__ unsigned long long timeline_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define HC_TL_DECL(epoch)                                                                                      \
  unsigned long long* const hc_tl =                                                                            \
      g_timeline + (((epoch)&3u) * 1024u + (blockIdx.x < 1024u ? blockIdx.x : 1023u)) * (unsigned)kTlSlots;     \
  long long hc_ph_t = 0
#define HC_TL_ZERO()                                \
  do {                                              \
    hc_tl[7] = hc_tl[14] = hc_tl[15] = 0;           \
    for (int i_ = 16; i_ < kTlSlots; ++i_) hc_tl[i_] = 0; \
  } while (0)
#define HC_STAMP(i) hc_tl[i] = timeline_now()
#define HC_STAMP_MAX(i) atomicMax(&hc_tl[i], timeline_now())
#define HC_TIC() const unsigned long long hc_tic = timeline_now()
#define HC_TOC(i) hc_tl[i] += timeline_now() - hc_tic
// phase accounting of one thread: HC_PH_START() once, then HC_PH(i) charges the cycles since the
// previous mark to phase i
#define HC_PH_START() hc_ph_t = clock64()
#define HC_PH(i)                                  \
  do {                                            \
    const long long now_ = clock64();             \
    hc_tl[16 + (i)] += (unsigned long long)(now_ - hc_ph_t); \
    hc_ph_t = now_;                               \
  } while (0)
#define HC_PH_COUNT() hc_tl[kTlSlots - 1] += 1
// copies the stamps of the last four launches (4 x 1024 CTAs x 32 slots) to the host (synchronises) and clears them
#define HC_TL_READ(name)                                                                                       \
  extern "C" int name(unsigned long long* host) {                                                              \
    using hc::dev::g_timeline;                                                                                 \
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;                                                     \
    if (cudaMemcpyFromSymbol(host, g_timeline, sizeof(g_timeline)) != cudaSuccess) return -1;                  \
    void* sym = nullptr;                                                                                       \
    if (cudaGetSymbolAddress(&sym, g_timeline) == cudaSuccess) cudaMemset(sym, 0, sizeof(g_timeline));         \
    return 0;                                                                                                  \
  }
#else
#define HC_TL_READ(name)
#define HC_TL_DECL(epoch)
#define HC_TL_ZERO()
#define HC_STAMP(i)
#define HC_STAMP_MAX(i)
#define HC_TIC()
#define HC_TOC(i)
#define HC_PH_START()
#define HC_PH(i)
#define HC_PH_COUNT()
#endif

}  // namespace dev
}  // namespace hc
