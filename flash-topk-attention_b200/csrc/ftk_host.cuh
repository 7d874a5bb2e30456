// Host-side helpers shared by the launchers: error codes, tensor-map encoding
// through the driver entry point (no link-time dependency on libcuda, so the
// library also loads on machines without a driver).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace ftk {

// C-ABI return codes (mirrored in include/ftk_api.h)
enum : int {
  FTK_OK = 0,
  FTK_ERR_BAD_ARG = -1,
  FTK_ERR_UNSUPPORTED = -2,
  FTK_ERR_WORKSPACE = -3,
  FTK_ERR_CUDA = -4,
  FTK_ERR_DRIVER = -5,
  FTK_ERR_CAPACITY = -6,
};

enum : int { FTK_DTYPE_F16 = 0, FTK_DTYPE_BF16 = 1 };

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Tensor map over a 16-bit tensor addressed as [b][n][h][d] with element
// strides (sb, sn, sh) and unit stride along d.  Box = box_d x 1 x box_rows x 1
// (d, h, n, b), 128-byte swizzle, out-of-range elements read as zero.
// Coordinates at load time are (d0, h, n0, b).
inline int encode_tmap_bnhd(CUtensorMap* out, const void* base, int dtype, int64_t B, int64_t N,
                            int64_t H, int64_t D, int64_t sb, int64_t sn, int64_t sh, int box_d,
                            int box_rows) {
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return FTK_ERR_BAD_ARG;
  if (((sb * 2) & 15) || ((sn * 2) & 15) || ((sh * 2) & 15)) return FTK_ERR_BAD_ARG;
  if (box_d * 2 > 128 || box_rows > 256 || box_rows < 1) return FTK_ERR_BAD_ARG;
  // The stride of a dimension of one is never used for addressing but must be a legal
  // value, and a tensor map cannot repeat a dimension: a stride of 0 (an expanded
  // tensor) replaced by another would read rows that are not there.
  if ((B > 1 && sb <= 0) || (N > 1 && sn <= 0) || (H > 1 && sh <= 0)) return FTK_ERR_BAD_ARG;
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return FTK_ERR_DRIVER;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)N, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)(sh > 0 ? sh : D) * 2, (cuuint64_t)(sn > 0 ? sn : D) * 2,
                           (cuuint64_t)(sb > 0 ? sb : D) * 2};
  cuuint32_t box[4] = {(cuuint32_t)box_d, 1u, (cuuint32_t)box_rows, 1u};
  cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  CUtensorMapDataType dt =
      dtype == FTK_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  auto encode = [&]() {
    return fn(out, dt, 4, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // a thread that has made no runtime call yet (autograd's): bind its device's context
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess)
      return FTK_ERR_CUDA;
    r = encode();
  }
  return r == CUDA_SUCCESS ? FTK_OK : FTK_ERR_DRIVER;
}

// Dynamic shared memory of a kernel, raised once per device and size instead of
// at every launch (the attribute call costs about a microsecond of host time).
// The runtime sets the limit, it does not raise it: threads that ask for two sizes at once take
// turns at looking, setting and recording, or the smaller one could be set behind the record of
// the larger, and launches of that kernel would fail from then on.  A size that is on record
// needs no turn: the limit was set before and never goes down.
template <auto KERNEL>
inline int allow_smem(size_t bytes) {
  constexpr int MAX_DEVICES = 64;
  static std::atomic<size_t> allowed[MAX_DEVICES];
  static std::mutex turn;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return FTK_ERR_CUDA;
  const bool known = dev >= 0 && dev < MAX_DEVICES;
  if (known && allowed[dev].load(std::memory_order_acquire) >= bytes) return FTK_OK;
  std::lock_guard<std::mutex> lock(turn);
  if (known && allowed[dev].load(std::memory_order_relaxed) >= bytes) return FTK_OK;
  if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(bytes)) != cudaSuccess)
    return FTK_ERR_CUDA;
  if (known) allowed[dev].store(bytes, std::memory_order_release);
  return FTK_OK;
}

// A kernel as a type, for code that is generic over kernels of one signature
template <auto KERNEL>
struct Kernel {
  static constexpr auto kernel = KERNEL;
};

// A run-time value 0 .. N - 1 as a compile-time one: f(std::integral_constant<int, value>)
template <int N, typename F>
inline int choose(int value, F&& f) {
  if constexpr (N > 1) {
    if (value < N - 1) return choose<N - 1>(value, f);
  }
  return f(std::integral_constant<int, N - 1>{});
}

// Kernels that this library has enqueued (or captured), for ftk_launch_count.
inline std::atomic<long long> g_launches{0};

// Result of launching `kernels` kernels: FTK_OK, and they are counted, or FTK_ERR_CUDA.
inline int launched(cudaError_t e, int kernels = 1) {
  if (e != cudaSuccess) return FTK_ERR_CUDA;
  g_launches.fetch_add(kernels, std::memory_order_relaxed);
  return FTK_OK;
}

// Launch that may overlap the tail of the stream's previous kernel.  Only for
// kernels that call pdl_wait() in every block before they touch global memory; the one
// launch that does so later is described at pdl_wait().
template <typename... Params, typename... Args>
inline int launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                      cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return launched(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

// The same as clusters of `cluster` CTAs along x (1: no clusters).
template <typename... Params, typename... Args>
inline int launch_clusters(void (*kernel)(Params...), int cluster, dim3 grid, dim3 block,
                           size_t smem, cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return launched(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

// Clusters of that size that can run at once, 0 if the device does not say.
template <typename... Params>
inline int max_clusters(void (*kernel)(Params...), int cluster, dim3 block, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster));
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(cluster);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

inline int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// Dynamic shared memory for a grid of few CTAs that may start under its predecessor: so much that
// no SM takes more than its share.  Otherwise the SMs that the predecessor leaves idle take as many
// as fit, and the work of those waits while the others have none (select of 32000 rows behind 128
// scoring CTAs: 12.0 us, 9.6 with this; score, merge and forward of 4096 tokens, H = 2, head dim 64,
// 32 picks 82 and 64).  `bytes`: the dynamic part that the kernel needs; `fixed`: its static
// part, or a bound of it.
// What runs on other streams finds less room beside such a grid.  That costs where several of them
// would share the SMs: 64 forward tiles of 8 blocks on each of four streams at once 17.4 us, 23.3
// with this, the whole pass of 1024 tokens, H = 8, q-blocks of 32 on four 83.8, 85.4; on one and two
// streams, and on four for the selects and merges, this is the faster one.  To leave half of
// an SM to others (114 KB and one CTA per SM) gains nothing there.
inline size_t spread_smem(int64_t ctas, size_t bytes, size_t fixed) {
  const int64_t share = (ctas + sm_count() - 1) / sm_count();
  if (share > 8) return bytes;
  const size_t most = static_cast<size_t>(227 * 1024 / share) / 1024 * 1024 - 1024;   // 1 KB of each CTA's is reserved
  return std::max(bytes, most > fixed ? most - fixed : 0);
}

}  // namespace ftk
