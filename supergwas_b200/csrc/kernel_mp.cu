// kernel_mp.cu -- parts shared by the many-phenotype kernels: the FP64
// refinement of their candidates, the supported shapes and the TMA map of
// packed rows.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "device.cuh"
#include "kernels.hpp"

namespace kg {

constexpr unsigned long long MP_KMER_MASK = (1ull << 47) - 1;  // bit 47: CAND_OPEN_MP

// Adds the screen's counts to the launch's, unless it gave up, and clears them for
// the next launch.  A call: inlined, it changes the registers that the compiler
// gives the candidates' loop (8 phenotypes at n = 5000: 65 -> 101 us).
static __device__ __noinline__ void mp_add_counts(const DevOutMP& O, unsigned nc) {
  const bool fs = !*O.over;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < nc; i += gridDim.x * blockDim.x) {
    const unsigned long long c = O.fs_tested[i];
    if (!c) continue;
    if (fs) atomicAdd(O.tested + i, c);
    O.fs_tested[i] = 0;
  }
}

// FP64 recomputation of the candidates of a multi-phenotype launch: one
// warp per (k-mer, phenotype), the phenotype's byte tables at T + p*tstride
// (lanes own the FP64 columns, one table row per byte of the packed row).
template <int CM>
__global__ void __launch_bounds__(256) mp_refine_kernel(const uint64_t* __restrict__ x, int wpk, int nwords,
                                                        const double* __restrict__ T, unsigned long long tstride,
                                                        const double* __restrict__ V, unsigned long long vstride,
                                                        const MPheno* __restrict__ ph, const DevOutMP O) {
  const int lane = threadIdx.x & 31;
  const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
  const unsigned nc = O.over ? (unsigned)O.n_shards * (unsigned)O.n_pheno : 0u;
  if (blockIdx.x * blockDim.x < nc) mp_add_counts(O, nc);
  const bool fs = O.over && !*O.over;  // the 4-bit screen's candidates
  unsigned long long ncand = O.counters[fs ? CNT_FS_OPEN : 3];
  if (ncand > O.cand_cap) ncand = O.cand_cap;
  for (unsigned long long w = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < ncand;
       w += warps) {
    const unsigned long long ent = O.cand[w];
    const unsigned long long gk = ent & MP_KMER_MASK;
    const int p = (int)(ent >> 48);
    const EpiParams& P = ph[p].P;
    const uint64_t* row = x + (gk - O.kmer_offset) * (unsigned long long)wpk;
    double acc[(CM + 31) / 32];
    table_row_sums<CM>(row, nwords, T + (size_t)p * tstride, lane, acc);
    int c;
    double ss, ey;
    refine_reduce<CM>(P, acc, lane, c, ss, ey);
    if (ent & CAND_OPEN_MP) {
      if (!refine_gate<CM>(P, ph[p].LM, V + (size_t)p * vstride, row, nwords, acc, lane, c, ey)) continue;
      if (lane == 0)
        atomicAdd(O.tested + (size_t)mp_shard(O, gk) * O.n_pheno + p, O.weight ? (unsigned long long)O.weight[gk] : 1ull);
    }
    if (lane == 0) {
      const double xxM = (double)c - ss, xyM = P.b * (double)c + ey;
      double effect = 0, Tq = 0, pv = 1;
      if (xxM > 1e-12 && P.yyM > 1e-12) {
        double r2 = (xyM * xyM) / (xxM * P.yyM);
        if (r2 < 0) r2 = 0;
        if (r2 >= 1) r2 = 1 - 1e-15;
        Tq = (double)P.n * log(1.0 / (1.0 - r2));
        pv = erfc(sqrt(0.5 * Tq));
        effect = xyM / (xxM * P.yyM);
      }
      if (pv <= P.p_thresh) {
        const unsigned long long slot = atomicAdd(O.counters + 1, 1ull);
        if (slot < O.hit_cap) {
          kg_phit h;
          h.kmer = gk;
          h.pheno = p;
          h.shard = mp_shard(O, gk);
          h.effect = effect;
          h.pval = pv;
          h.chisq = Tq;
          O.hits[slot] = h;
        } else {
          atomicOr(O.counters + 2, (unsigned long long)ERR_HIT_OVERFLOW);
        }
      }
    }
  }
}

// ------------------------------------------------------------------- host

static PFN_cuTensorMapEncodeTiled_v12000 mp_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

bool mp_supported(int NP, int PPG, int wpk) {
  if (NP < 16 || NP > 128 || NP % 16 || PPG < 1 || NP * PPG > 128) return false;
  if (wpk * 8 < 128) return false;
  return mp_encode_fn() != nullptr;
}

bool mp_tmap(const uint64_t* x, unsigned long long m, int wpk, CUtensorMap* tm, int rows) {
  auto enc = mp_encode_fn();
  if (!enc) return false;
  const cuuint64_t rowbytes = (cuuint64_t)wpk * 8;
  cuuint64_t gdim[2] = {rowbytes, (cuuint64_t)m};
  cuuint64_t gstride[1] = {rowbytes};
  // rows shorter than a 128-byte box: whole rows, not swizzled
  const bool wide = rowbytes >= 128;
  cuuint32_t box[2] = {wide ? 128u : (cuuint32_t)rowbytes, (cuuint32_t)rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)x, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CM>
static cudaError_t launch_mp_refine_t(const LaunchMpRefine& L, cudaStream_t st) {
  static int per_sm = 0;  // every warp of the grid resident at once (candidates are dealt round-robin)
  if (per_sm < 1 &&
      (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mp_refine_kernel<CM>, 256, 0) != cudaSuccess ||
       per_sm < 1))
    per_sm = 1;
  mp_refine_kernel<CM><<<(unsigned)(L.num_sms * per_sm), 256, 0, st>>>(
      L.x, L.wpk, L.vrows / 64, L.T, (unsigned long long)refine_table_len(L.vrows, L.cm), L.V, L.vstride, L.ph, *L.O);
  return cudaGetLastError();
}

cudaError_t launch_mp_refine(const LaunchMpRefine& L, cudaStream_t st) {
  if (!L.T) return cudaErrorInvalidValue;
  switch (L.cm) {
    case 8: return launch_mp_refine_t<8>(L, st);
    case 12: return launch_mp_refine_t<12>(L, st);
    case 16: return launch_mp_refine_t<16>(L, st);
    case 20: return launch_mp_refine_t<20>(L, st);
    case 24: return launch_mp_refine_t<24>(L, st);
    case 28: return launch_mp_refine_t<28>(L, st);
    case 36: return launch_mp_refine_t<36>(L, st);
    case 44: return launch_mp_refine_t<44>(L, st);
    case 52: return launch_mp_refine_t<52>(L, st);
    case 68: return launch_mp_refine_t<68>(L, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kg
