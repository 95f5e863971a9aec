// pairs_launch_check.cpp -- TEST INFRASTRUCTURE ONLY: kg_pairs_run_host
// (capi_pairs.cpp) on the host, with stand-ins for the CUDA runtime calls that it
// makes and for the kernel launches, whose results the caller chooses.
#include <cstdlib>
#include <cstring>

#include "../../supergwas_b200/csrc/capi_pairs.cpp"

static cudaError_t pair_result, refine_result;
static int screened, refined;

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }

unsigned long long kgctx::open_base() { return kg::FS_OPEN_BASE; }
int kgctx::ensure_cand(kg_ctx* ctx, unsigned long long cap) {
  ctx->cand_cap = cap;
  return cudaMalloc((void**)&ctx->dCand, cap * sizeof(unsigned long long)) == cudaSuccess ? KG_OK : KG_ERR_NOMEM;
}

namespace kg {
bool pairs_supported(int, int, int, int, int) { return true; }
bool fsp_supported(int, int, int, int, unsigned long long) { return true; }
cudaError_t launch_fs_pairs(const LaunchFsPairs&, cudaStream_t) {
  ++screened;
  return pair_result;
}
cudaError_t launch_pairs(const LaunchPairs&, cudaStream_t) { return pair_result; }
cudaError_t launch_pair_refine(const LaunchPairRefine&, cudaStream_t) {
  ++refined;
  return refine_result;
}
}  // namespace kg

// One call on 200 rows of one word pair; fs: the structure has a 4-bit screen.
// Returns kg_pairs_run_host's code; ran[0]: screen launches, ran[1]: refinements.
extern "C" int pairs_call(int fs, int pair_code, int refine_code, int* ran) {
  kg_ctx ctx;
  unsigned long long counters[64] = {};
  ctx.have_structure = true;
  ctx.opts.precision = KG_PREC_SPLIT_I8;
  ctx.n_row = 100;
  ctx.num_sms = 148;
  ctx.dCounters = counters;
  ctx.P.yyM = 1.0;
  ctx.fs_N = fs ? 16 : 0;
  pair_result = (cudaError_t)pair_code;
  refine_result = (cudaError_t)refine_code;
  screened = refined = 0;
  uint64_t x[400] = {};
  const int rc = kg_pairs_run_host(&ctx, x, 200, 2, 0, 200, nullptr);
  ran[0] = screened;
  ran[1] = refined;
  cudaFree(ctx.dPX);
  cudaFree(ctx.dPairs);
  cudaFree(ctx.dCand);
  cudaFree(ctx.dUnitOff);
  return rc;
}
