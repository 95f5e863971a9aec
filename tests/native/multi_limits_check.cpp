// multi_limits_check.cpp -- TEST INFRASTRUCTURE ONLY: the argument checks of
// kg_launch_multi_device (capi_multi.cpp) on the host.  The call ends at its
// first allocation, which fails here; what lies behind it is not linked.
#include "../../supergwas_b200/csrc/capi_multi.cpp"

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }

namespace kg {
bool mp_supported(int, int, int) { return true; }
}  // namespace kg

extern "C" int multi_call(uint64_t m) {
  kg_ctx ctx;
  ctx.mp.np = 1;
  ctx.mp.n_row = 100;
  uint64_t x[16] = {};
  return kg_launch_multi_device(&ctx, x, m, 16, nullptr, 0, nullptr);
}
