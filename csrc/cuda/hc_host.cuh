// Host-side pieces that the launchers share: tensor maps, grid sizes, launches with programmatic serialisation.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>

#include "hc_kernels.cuh"

namespace hc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// 2-D view {32, rows} of a 4-byte-element array, box {32, box_rows}, 128-byte swizzle
inline bool make_rows_map(CUtensorMap* map, const void* base, uint64_t rows, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn || rows == 0 || (reinterpret_cast<uintptr_t>(base) & 15u)) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kBlock, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kBlock * 4};
  cuuint32_t box[2] = {(cuuint32_t)kBlock, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

struct DeviceInfo {
  int sms = 0;
  bool ready = false;
};
inline DeviceInfo& device_info() {
  static thread_local DeviceInfo info[64];
  int dev = 0;
  cudaGetDevice(&dev);
  DeviceInfo& d = info[dev & 63];
  if (!d.ready) {
    cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    d.ready = true;
  }
  return d;
}

template <typename K>
cudaError_t set_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Launch with programmatic stream serialisation: the kernel may start while the one before it drains.  The steps of a
// collective order their data by arrival flags; every other kernel launched this way executes griddepcontrol.wait
// before it touches global memory, and only its launch and set-up overlap (a 4 KB compress back to back: 6.1 us a call
// without).
template <typename... Params, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), int grid, int block, int smem, cudaStream_t stream,
                              const Args&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  memset(&attr, 0, sizeof(attr));
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// CTAs of `kernel` that one GPU holds at the same time, asked of the runtime once per device.  The
// kernels are written for a grid that is resident as a whole (CTA i owns tile i, and every look-back
// waits for tiles held by other CTAs of the grid), so the grid is cut to this number, never assumed.
template <typename K>
int resident_ctas(K kernel, int threads, int smem, int* cache) {
  int dev = 0;
  cudaGetDevice(&dev);
  int& c = cache[dev & 63];
  if (c == 0) {
    if (set_smem(kernel, smem) != cudaSuccess) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, (size_t)smem) != cudaSuccess) return 0;
    c = per_sm * device_info().sms;
  }
  return c;
}

}  // namespace hc
