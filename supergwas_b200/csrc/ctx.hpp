// ctx.hpp -- the context behind the C ABI (private to the library).
#pragma once
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/kgwas_cuda.h"
#include "kernels.hpp"
#include "prep.hpp"

namespace kgctx {

constexpr int NBUF = 2;  // host-run chunk buffers in flight

template <class T>
inline void dfree(T*& p) {
  if (p) cudaFree((void*)p);
  p = nullptr;
}

// Smallest r2 that can still give p = erfc(sqrt(T/2)) <= p_thresh with
// T = n log(1/(1-r2)) (src/kgwas.cpp:51-52), lowered by a relative margin of
// 1e-9 so that k-mers below it are certainly not emitted.  -1 when every
// tested k-mer may be emitted.
inline double r2_candidate(double p_thresh, int n) {
  if (!(p_thresh < 1.0)) return -1.0;
  if (p_thresh <= 0.0) return 2.0;
  double lo = 0.0, hi = 1.0;
  while (std::erfc(std::sqrt(0.5 * hi)) > p_thresh && hi < 1e7) hi *= 2;
  for (int it = 0; it < 200; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (std::erfc(std::sqrt(0.5 * mid)) > p_thresh) lo = mid; else hi = mid;
  }
  const double r2 = -std::expm1(-lo / (double)n);
  return r2 * (1.0 - 1e-9);
}

// Epilogue constants of one prepared phenotype.
inline void fill_epi(kg::EpiParams& P, const kg::Prepared& p, const kg_opts& o, bool refine) {
  std::memset(&P, 0, sizeof(P));
  P.n = p.n;
  P.k = p.k;
  P.b = p.b;
  P.kappa = p.kappa;
  P.yyM = p.yyM;
  P.ynorm = p.ynorm;
  P.corr_thr = o.corr_threshold;
  P.p_thresh = std::pow(10.0, -o.log10_thresh);
  P.r2_cand = r2_candidate(P.p_thresh, p.n);
  P.thr2_ynorm2 = o.corr_threshold * o.corr_threshold * p.ynorm * p.ynorm;
  for (int j = 0; j < p.k; ++j) {
    P.a[j] = p.a[j];
    P.g[j] = p.g[j];
  }
  if (refine) {
    P.refine = 1;
    P.r2_ref = -std::expm1(-kg::REFINE_CHISQ / (double)p.n);
  }
}

// Constants of the 4-bit screen for one phenotype (fs_verdict).  False where
// the screen does not apply: the intercept has limbs or is not of unit norm (the
// screen takes c (n - c) / n for c - s_0^2: within 1e-9 c), the structure or the
// phenotype is degenerate, or so much may pass (thresholds at which rows of
// chi-square below REFINE_CHISQ are emitted, residuals that leave the cut or the
// gate vague) that refining it would cost more than the screen saves: a
// refinement reads n / 8 table rows, 20 KB at n = 1000, r = 16+1, so 1e-3 of the
// k-mers cost as much as the screen of all of them (1e8: 1e5 and 2.2 ms).
inline bool fill_fs(kg::FsPheno& F, const kg::EpiParams& P, const kg::Prepared& p, const kg::FsCols& C, int lu,
                    bool gate) {
  F = kg::FsPheno();
  const double r2_ref = -std::expm1(-kg::REFINE_CHISQ / (double)p.n);
  const double yv = P.yyM / (P.ynorm * P.ynorm);
  if (!p.drop0 || p.k < 1 || !(std::fabs(P.a[0] * P.a[0] * p.n - 1.0) <= 1e-9) || p.n >= 65536 || !(P.ynorm >= 1e-12) || !(P.ynorm < 1e150) || !(yv > 1e-6) ||
      !(P.r2_cand >= r2_ref) || !(P.r2_cand < 1.0))
    return false;
  F.n = (float)p.n;
  F.inv_n = (float)(1.0 / p.n);
  const double cut = P.r2_cand * yv;
  F.cut = (float)(cut * (1.0 - 1e-4));
  F.b = (float)(P.b / P.ynorm);
  F.kappa = (float)(P.kappa / P.ynorm);
  F.thr = (float)P.corr_thr;
  // the columns' norms, for the rounding of single-precision sums and scales
  // (a few 2^-24 of each term): 1e-5 of them
  double fu = 0, fy = 0, fg = P.ynorm;
  for (int j = 1; j < p.k; ++j)
    for (int i = 0; i < p.n; ++i) fu += p.d[(size_t)j * p.n + i] * p.d[(size_t)j * p.n + i];
  for (int i = 0; i < p.n; ++i) fy += p.d[(size_t)p.k * p.n + i] * p.d[(size_t)p.k * p.n + i];
  const double up = 1.0 + 1e-5;
  const double bu = C.nu * up + 1e-5 * std::sqrt(fu), by = (C.ny * up + 1e-5 * std::sqrt(fy)) / P.ynorm;
  const double bg = (C.ng * up + 1e-5 * fg) / P.ynorm;
  if (!(bu <= 0.25) || !(by <= 0.2 * std::sqrt(cut)) || (gate && !(bg <= 2e-3))) return false;
  const double tiny = 1e-12;
  F.bu = (float)bu;
  F.mu = (float)(C.mu * up + tiny);
  F.by = (float)by;
  F.my = (float)(C.my * up / P.ynorm + tiny);
  F.bg = (float)bg;
  F.mg = (float)((C.mg + 1.01 * P.gate_unit) * up / P.ynorm + tiny);  // the limb sums decide alike outside it
  for (int l = 0; l < 3; ++l) F.sy[l] = (float)(C.sy[l] / P.ynorm);
  if (gate)
    for (int l = 0; l < 4; ++l) F.sg[l] = (float)(C.sg[l] / P.ynorm);
  for (int j = 0; j + 1 < p.k; ++j)
    for (int l = 0; l < lu; ++l) F.su[lu * j + l] = (float)C.su[(size_t)j * lu + l];
  return true;
}

// State of the many-phenotype path.
struct Multi {
  int np = 0, n_row = 0, NP = 0, G = 0, kpad = 0, cm = 0, nsteps = 0;
  int PPG = 1;          // phenotypes per group (one MMA of NP * PPG columns)
  bool stationary = false;  // the group image fits in shared memory: kernel_mpb.cu
  bool pair_ok = false;     // kernel_mpb2.cu can run these phenotypes (PPG = 1 images)
  int kern = 0;             // chosen kernel: 0 image streamed (tb), 1 image resident (mpb), 2 SM pair (mpb2), 3 4-bit screen (fs)
  int bt_scale = 2;         // tile-iterations per L2 block: the 48 MB rule times bt_scale / 2
  // 4-bit screen: group images and, behind them, the phenotypes' constants;
  // columns per slot (0: not used), slots per group, groups, samples per image
  uint8_t* dFs = nullptr;
  int fs_NP = 0, fs_PPG = 1, fs_G = 0, fs_kpad = 0;
  int8_t* dB = nullptr;
  kg::MPheno* dPh = nullptr;
  double* dV = nullptr;
  double* dT = nullptr;  // byte tables of V (refinement), one block per phenotype
  size_t vstride = 0;
  unsigned long long* dCounters = nullptr;
  unsigned long long* dTested = nullptr;  // counts, and behind them the screen's
  size_t tested_cap = 0;
  kg_phit* dHits = nullptr;
  unsigned long long hit_cap = 0;
  unsigned long long* dShard = nullptr;
  int shard_cap = 0;
  int n_shards = 1;
  std::vector<unsigned long long> shard_host;
  std::vector<kg_phit> hits;
  std::vector<uint64_t> tested;
  unsigned long long counters[kg::NCOUNT] = {};
  // shape of the last streamed-image launch: tiles per item, image chunks in the ring
  int xs = 1, nb = 4;
  int bt = 0;  // B-stationary kernel: tile-iterations per L2 block of the last launch
  bool tuned = false;
  int tuned_nbox = -1;
  // pending device launch and its captured graph
  bool pending = false;
  const uint64_t* pend_x = nullptr;
  uint64_t pend_m = 0;
  uint32_t pend_wpk = 0;
  cudaStream_t pend_stream = nullptr;
  cudaGraphExec_t graph = nullptr;
  const uint64_t* g_x = nullptr;
  uint64_t g_m = 0;
  uint32_t g_wpk = 0;
  cudaStream_t g_stream = nullptr;
  int g_seen = 0, g_launches = 0;
};

}  // namespace kgctx

struct kg_ctx {
  kg_opts opts{};
  int num_sms = 0;
  cudaStream_t stream = nullptr, copy_stream = nullptr;
  std::string err;
  bool have_structure = false;
  int n_row = 0;  // samples per packed row
  kg::Prepared prep;
  kg::LimbCols limbs;
  kg::EpiParams P{};
  kg::LimbMap LM{};
  // structure on the device
  double* dV = nullptr;
  double* dT = nullptr;      // byte tables of V for the split form's FP64 refinement
  int cm = 0, nsteps = 0;
  int8_t* dB = nullptr;      // B image of the smem-A kernel
  int8_t* dBts = nullptr;    // B image of the TMEM-A kernels
  kg::MPheno* dPh1 = nullptr;  // the phenotype's constants for the streamed-image kernel
  // 4-bit screen: image, the phenotype's constants; columns (0: not used), limbs
  // per U column, samples of the image
  uint8_t* dFs = nullptr;
  kg::FsPheno fsF{};
  int fs_N = 0, fs_lu = 0, fs_kpad = 0;
  // FP64 form behind the screen: the gathered rows of undecided k-mers
  uint64_t* dGather = nullptr;
  size_t gather_bytes = 0;
  int nchunk = 0;
  int f64_N = 0;             // limb columns of the FP64 form (dBts holds image and constants); 0: CUDA cores
  // outputs on the device
  unsigned long long* dCounters = nullptr;
  kg_hit* dHits = nullptr;
  unsigned long long hit_cap = 0;
  unsigned long long* dCand = nullptr;  // FP64 refinement candidates (split form)
  unsigned long long cand_cap = 0;
  uint8_t* dTested = nullptr;
  double* dStat[7] = {};
  size_t stat_cap = 0;
  // host result
  std::vector<kg_hit> hits;
  unsigned long long counters[kg::NCOUNT] = {};
  // pending device launch
  bool pending = false;
  const uint64_t* pend_x = nullptr;
  uint64_t pend_m = 0;
  uint32_t pend_wpk = 0;
  bool pend_stats = false;
  cudaStream_t pend_stream = nullptr;
  int launches = 0;
  const char* last_kernel = "";
  int last_screen = 0;       // limbs per U column of the last launch's 4-bit screen, negative where it gave up
  // bounded device waits: pipeline wait limit (0: the default) and the
  // one-launch stall of the row producer that the failure tests use
  unsigned long long wait_ns = 0;
  unsigned long long stall_once = 0;
  // host-run buffers
  uint64_t* dChunk[kgctx::NBUF] = {};
  void* hStage[kgctx::NBUF] = {};
  size_t chunk_bytes = 0;
  cudaEvent_t ev_h2d[kgctx::NBUF] = {}, ev_k[kgctx::NBUF] = {};
  // runs of equal adjacent rows (kg_run_host): first row and length of each
  // run; the device copy of the lengths weighs the tested count
  std::vector<uint64_t> run_first;
  std::vector<uint32_t> run_len;
  uint32_t* dWeight = nullptr;
  size_t weight_cap = 0;
  uint32_t* hWeight[kgctx::NBUF] = {};  // pinned staging of one chunk's run lengths
  size_t hweight_cap = 0;
  const uint32_t* cur_weight = nullptr;  // set while a deduplicated run is in flight
  uint64_t unique_rows = 0;              // rows the last kg_run_host tested (0: no deduplication)
  // many phenotypes
  kgctx::Multi mp;
  // 2-D pair test
  uint64_t* dPX = nullptr;        // packed rows on the device
  size_t px_bytes = 0;
  kg_pair* dPairs = nullptr;
  unsigned long long pair_cap = 0;
  unsigned long long* dUnitOff = nullptr;
  size_t unit_cap = 0;
  std::vector<kg_pair> pairs;

  int fail(int code, const std::string& m) {
    err = m;
    return code;
  }
  int cuda_fail(cudaError_t e, const char* what) {
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return KG_ERR_CUDA;
  }
};

#define KG_CUDA(call, what)                                    \
  do {                                                         \
    cudaError_t e__ = (call);                                  \
    if (e__ != cudaSuccess) return ctx->cuda_fail(e__, what);  \
  } while (0)

namespace kgctx {
void free_multi(kg_ctx* ctx);  // capi_multi.cpp
void drop_graph(Multi& M);
}  // namespace kgctx

namespace kgctx {

// Runs of equal adjacent host rows.  Real batches are sorted by bit pattern
// (src/convert_matrix.cpp:366-368), so equal rows sit next to each other; an
// equal row has equal statistics, so one row per run is tested and counts as
// many tested k-mers as the run has rows.
//
// use_runs: whether to test one row per run.  Finding the runs reads every
// row on the host, which pays only where the rows are copied through the host
// anyway (pageable memory): there, at least 10 % of 4096 sampled adjacent
// pairs must be equal.  KG_DEDUP=0 never, KG_DEDUP=1 always (pinned too).
bool use_runs(const uint64_t* x, uint64_t m, uint32_t wpk, bool pageable);
inline bool rows_equal(const uint64_t* a, const uint64_t* b, uint32_t wpk) {
  uint64_t d = 0;
  for (uint32_t w = 0; w < wpk; ++w) d |= a[w] ^ b[w];
  return d == 0;
}
// A slice of a staging buffer: `rows` rows from row `stage_row` on.
struct StageSeg {
  uint64_t stage_row, rows;
};
// Rows [s0, s0 + cnt) of x in one pass: a row starts a run when it is the
// first of the range, differs from its predecessor or is in `bounds`
// (ascending row indices).  Host threads copy the first row of each run into
// their own slices of dst (listed in segs, in row order), the runs' first rows
// and lengths are appended to first / len; returns the number of runs.
uint64_t scan_gather(const uint64_t* x, uint64_t s0, uint64_t cnt, uint32_t wpk, void* dst,
                     const std::vector<unsigned long long>& bounds, std::vector<uint64_t>& first,
                     std::vector<uint32_t>& len, std::vector<StageSeg>& segs);
// All runs of x at once (kg_run_multi_host): fills ctx->run_first / run_len
// and returns true when use_runs holds and the runs save at least 10 % of the
// rows; `bounds` (shard starts) also start runs.
bool find_runs(kg_ctx* ctx, const uint64_t* x, uint64_t m, uint32_t wpk, const std::vector<unsigned long long>& bounds,
               bool pageable);
bool is_pinned(const void* p);
// What a launch does about rows that the 4-bit screen cannot place: it is repeated
// without the screen once its counters have been read (rows in buffers of the
// context), or the kernel for that case is launched behind the screen (rows that a
// caller, or the next chunk, may overwrite as soon as the launch is done).
enum Screen { SCREEN_REPEAT, SCREEN_BEHIND, SCREEN_OFF };
// The base of kg::fs_open_limit: FS_OPEN_BASE, or KG_SCREEN_OPEN (0: the shares
// alone; 16777216: never reached).
unsigned long long open_base();
// The candidate list, at least cap entries (all paths share it; what it held is lost).
int ensure_cand(kg_ctx* ctx, unsigned long long cap);
// Copies the run lengths to the device and makes them the tested-count
// weights of the following launches (ctx->cur_weight).
int upload_run_lengths(kg_ctx* ctx, cudaStream_t st);
// Pageable memory to the device through a pinned buffer of as many bytes, in
// several host threads.
cudaError_t stage_h2d(void* dst, void* stage, const void* src, size_t bytes, cudaStream_t st);
// Gathers rows sel[0..cnt) of x into dst (row bytes each).
void par_gather(void* dst, const uint64_t* x, const uint64_t* sel, uint64_t cnt, size_t row);
// Repeats each hit of a distinct row for every row of its run, in row order.
void expand_runs(const kg_ctx* ctx, std::vector<kg_hit>& hits);
void expand_runs(const kg_ctx* ctx, std::vector<kg_phit>& hits);

}  // namespace kgctx

