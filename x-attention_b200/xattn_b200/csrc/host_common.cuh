// Host-side helpers shared by the launchers: status codes, TMA tensor-map encoding through the
// driver entry point (no link-time dependency on libcuda), device checks.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../../include/xattn_b200.h"

namespace xb {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(p);
  return fn;
}

// Tensor seen as up to 5 dimensions, innermost first.  `strides_bytes` has rank-1 entries
// (the innermost stride is one element).  128-byte swizzle, zero fill outside the tensor.
inline int make_tmap(CUtensorMap* map, const void* base, CUtensorMapDataType type, int rank, const uint64_t* dims,
                     const uint64_t* strides_bytes, const uint32_t* box) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return XATTN_B200_ERR_CUDA;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return XATTN_B200_ERR_ARG;
  cuuint64_t gdim[5];
  cuuint64_t gstr[4];
  cuuint32_t gbox[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    gbox[i] = box[i];
    estr[i] = 1;
    if (i > 0) {
      if (strides_bytes[i - 1] % 16 != 0 || strides_bytes[i - 1] == 0) return XATTN_B200_ERR_ARG;
      gstr[i - 1] = strides_bytes[i - 1];
    }
  }
  CUresult r = enc(map, type, static_cast<cuuint32_t>(rank), const_cast<void*>(base),
                   gdim, gstr, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? XATTN_B200_OK : XATTN_B200_ERR_CUDA;
}

// What has to be set up or asked once per kernel and device, and costs microseconds of every call otherwise: `ask` runs at
// the first use (its positive answer is kept; a failure is not).  A few dozen kernels and up to 16 devices; safe to use
// from several threads (two may ask at once, and get the same answer).
template <typename F>
inline int once_per_device(const void* kernel, F&& ask) {
  struct Slot {
    std::atomic<const void*> key{nullptr};
    std::atomic<int> answer[16] = {};
  };
  static Slot slots[128];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 0;
  if (dev >= 16) return ask();
  for (size_t i = (reinterpret_cast<uintptr_t>(kernel) >> 4) % 128, n = 0; n < 128; ++n, i = (i + 1) % 128) {
    const void* k = slots[i].key.load(std::memory_order_acquire);
    if (k == nullptr && slots[i].key.compare_exchange_strong(k, kernel)) k = kernel;
    if (k != kernel) continue;
    int a = slots[i].answer[dev].load(std::memory_order_acquire);
    if (a <= 0) {
      a = ask();
      if (a > 0) slots[i].answer[dev].store(a, std::memory_order_release);
    }
    return a;
  }
  return ask();
}
inline int check_sm100() {
  static const char key = 0;
  const int major = once_per_device(&key, [] {
    int dev = 0, m = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    return cudaDeviceGetAttribute(&m, cudaDevAttrComputeCapabilityMajor, dev) == cudaSuccess ? m : 0;
  });
  return major == 10 ? XATTN_B200_OK : (major > 0 ? XATTN_B200_ERR_ARCH : XATTN_B200_ERR_CUDA);
}
inline int sm_count() {
  static const char key = 0;
  const int n = once_per_device(&key, [] {
    int dev = 0, m = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&m, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? m : 0;
  });
  return n > 0 ? n : 148;
}
// lets `kernel` take `bytes` of dynamic shared memory on the current device
template <typename K>
inline bool allow_smem(K kernel, size_t bytes) {
  return once_per_device(reinterpret_cast<const void*>(kernel), [&]() {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess ? 1 : 0;
  }) > 0;
}

// Kernel launches issued by this library in this process (every launcher calls launch_status() right after its
// <<<>>>): a diagnostic the benchmark reads through xattn_b200_launch_count().
inline std::atomic<unsigned long long>& launch_counter() {
  static std::atomic<unsigned long long> n{0};
  return n;
}

inline int launch_status() {
  launch_counter().fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError() == cudaSuccess ? XATTN_B200_OK : XATTN_B200_ERR_CUDA;
}

// Launches `kernel`, in clusters of `cluster` CTAs, so that it may start while the kernel before it in the stream is still running (programmatic
// stream serialization): the kernel must execute pdl_wait() before it touches anything that kernel writes.
// (Every kernel of a call is launched like this, and lets the next one start early: a prefill is three to six short
// kernels in a row, and the launch of one then runs under the one before it.)
template <typename... KArgs, typename... Args>
inline int launch_dependent_clusters(void (*kernel)(KArgs...), unsigned cluster, dim3 grid, dim3 block, size_t smem_bytes,
                                     cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  const int rc = launch_status();         // (in every case: it also clears the error, which the next launch would report as its own)
  return e == cudaSuccess ? rc : XATTN_B200_ERR_CUDA;
}
template <typename... KArgs, typename... Args>
inline int launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem_bytes, cudaStream_t stream,
                            Args&&... args) {
  return launch_dependent_clusters(kernel, 1, grid, block, smem_bytes, stream, std::forward<Args>(args)...);
}

// Division of numbers below 2^31 by a divisor known on the host (the round-up method of Granlund and Montgomery, "Division by
// invariant integers using multiplication"): a multiplication and a shift instead of the ~25
// instructions of an integer division, which add up in code that every role of a kernel has to decode its work with.
struct FastDiv {
  uint32_t d, mul, shift;
};
static inline FastDiv make_fast_div(uint32_t d) {
  FastDiv f;
  f.d = d;
  f.shift = 0;
  while ((1ull << f.shift) < d) ++f.shift;
  f.mul = static_cast<uint32_t>((((1ull << f.shift) - d) << 32) / d + 1);
  return f;
}
__device__ __forceinline__ int fast_div(int n, const FastDiv& f, int& rem) {
  const uint32_t q = (__umulhi(static_cast<uint32_t>(n), f.mul) + static_cast<uint32_t>(n)) >> f.shift;
  rem = n - static_cast<int>(q * f.d);
  return static_cast<int>(q);
}

}  // namespace xb
