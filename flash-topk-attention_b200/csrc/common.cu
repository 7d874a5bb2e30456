// Version and error-text entry points of the C ABI, and the conversion of float32
// activations.
#include <algorithm>

#include "ftk_host.cuh"
#include "ftk_sm100.cuh"

extern "C" int ftk_version(void) { return 100; }  // 0.1.0

extern "C" int64_t ftk_launch_count(void) { return ftk::g_launches.load(); }

extern "C" const char* ftk_error_string(int code) {
  switch (code) {
    case ftk::FTK_OK: return "ok";
    case ftk::FTK_ERR_BAD_ARG: return "bad argument (shape, range or alignment)";
    case ftk::FTK_ERR_UNSUPPORTED: return "configuration not supported by this build";
    case ftk::FTK_ERR_WORKSPACE: return "workspace missing or too small";
    case ftk::FTK_ERR_CUDA: return "CUDA runtime call or kernel launch failed";
    case ftk::FTK_ERR_DRIVER: return "tensor-map encoding unavailable or failed";
    case ftk::FTK_ERR_CAPACITY:
      return "problem exceeds the fixed buffer of a no-allocation entry point";
    case ftk::FTK_DEV_TIMEOUT_TMA: return "device: TMA producer wait timed out";
    case ftk::FTK_DEV_TIMEOUT_MMA: return "device: UMMA issuer wait timed out";
    case ftk::FTK_DEV_TIMEOUT_CONSUMER: return "device: consumer wait timed out";
    case ftk::FTK_DEV_TIMEOUT_EPILOGUE: return "device: epilogue wait timed out";
    case ftk::FTK_DEV_BAD_INDEX: return "device: block index out of range";
    default: return "unknown code";
  }
}

namespace ftk {

// float -> bf16, 8 elements per thread and step (two 16-byte loads, one 16-byte
// store); blockIdx.y = which array.  Bound by memory: 6 bytes per element.
struct CastArgs {
  const float4* src[3];
  uint4* dst[3];
  int64_t vecs[3];
};

__global__ void __launch_bounds__(256) cast_bf16_kernel(const CastArgs a) {
  pdl_wait();
  pdl_launch();
  const int t = blockIdx.y;
  const float4* src = t == 0 ? a.src[0] : t == 1 ? a.src[1] : a.src[2];
  uint4* dst = t == 0 ? a.dst[0] : t == 1 ? a.dst[1] : a.dst[2];
  const int64_t n = t == 0 ? a.vecs[0] : t == 1 ? a.vecs[1] : a.vecs[2];
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  auto pack = [](float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
  };
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) {
    const float4 x = src[2 * i], y = src[2 * i + 1];
    dst[i] = make_uint4(pack(x.x, x.y), pack(x.z, x.w), pack(y.x, y.y), pack(y.z, y.w));
  }
}

}  // namespace ftk

extern "C" int ftk_cast_bf16(const float* a, int64_t na, void* to_a, const float* b, int64_t nb,
                             void* to_b, const float* c, int64_t nc, void* to_c, void* stream) {
  using namespace ftk;
  const float* src[3] = {a, b, c};
  const int64_t n[3] = {na, nb, nc};
  void* dst[3] = {to_a, to_b, to_c};
  CastArgs args{};
  int64_t most = 0;
  int count = 0;
  for (int i = 0; i < 3; i++) {
    if (!src[i]) continue;
    if (!dst[i] || n[i] < 0 || n[i] % 8 != 0 ||
        ((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i])) & 15u))
      return FTK_ERR_BAD_ARG;
    args.src[count] = reinterpret_cast<const float4*>(src[i]);
    args.dst[count] = static_cast<uint4*>(dst[i]);
    args.vecs[count++] = n[i] / 8;
    most = std::max(most, n[i] / 8);
  }
  if (count == 0 || most == 0) return FTK_OK;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((most + 255) / 256, sm_count() * 16));
  return launch_pdl(cast_bf16_kernel, dim3(grid, count), 256, 0, static_cast<cudaStream_t>(stream),
                    args);
}
