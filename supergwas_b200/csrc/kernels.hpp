// kernels.hpp -- host-side launch interface of the association kernels.
#pragma once
#include <cuda_runtime.h>

#include "params.hpp"

struct CUtensorMap_st;

namespace kg {

struct LaunchFp64 {
  const uint64_t* x;          // packed rows (device)
  unsigned long long m;       // k-mers in this launch
  int wpk;                    // words per k-mer
  const double* V;            // nsteps*128 x cm FP64, sample-major, zero padded (device)
  int nsteps, cm;             // sample steps of 128; padded column count
  const EpiParams* P;
  const DevOut* O;
  int num_sms;
  const double* T = nullptr;  // refinement byte tables of V (refine_table_len doubles; device)
  const LimbMap* LM = nullptr;  // refinement: the int8 limb columns
};

struct LaunchTc {
  const uint64_t* x;
  unsigned long long m;
  int wpk;
  int nchunk;                 // K chunks of tc_kc() samples
  const int8_t* Bimg;         // B operand shared-memory image, chunk after chunk (device)
  const EpiParams* P;
  const LimbMap* LM;
  const DevOut* O;
  int num_sms;
};

int fp64_cm(int C);           // padded column count for C contraction columns (-1: too many)
int fp64_steps(int n);        // 128-sample steps covering n samples
cudaError_t launch_fp64(const LaunchFp64& L, cudaStream_t st);
// FP64 recomputation of the split form's refinement candidates from the
// byte tables of V (LaunchFp64::T).
cudaError_t launch_refine(const LaunchFp64& L, cudaStream_t st);

// Byte tables of the FP64 columns, one block per phenotype: for the 8-sample
// group g of a packed row and a byte value b, entry (g*256 + b)*cm + j is the
// sum of column j of V over the samples of g whose bit is set in b.
struct LaunchTable {
  const double* V;            // nblocks blocks of vrows x cm FP64 (vstride doubles apart)
  int vrows, cm;              // vrows a multiple of 128
  unsigned long long vstride;
  int nblocks;
  double* T;                  // nblocks blocks of refine_table_len(vrows, cm) doubles
};
size_t refine_table_len(int vrows, int cm);
cudaError_t launch_refine_table(const LaunchTable& L, cudaStream_t st);

struct LaunchTs {
  const uint64_t* x;          // packed rows (device), 16-byte aligned
  unsigned long long m;
  int wpk;
  int kpad;                   // samples covered by the B image (multiple of 128)
  bool drop0;                 // U column 0 has no limbs (intercept handled in FP64)
  const int8_t* Bimg;         // make_b_image_ts layout (device)
  const EpiParams* P;
  const LimbMap* LM;
  const DevOut* O;
  int num_sms;
};

// TMEM-A kernel: 3 limbs per U column, 5 for y', N <= 128, B resident in smem.
bool ts_supported(int N, int limbs_u, int limbs_y, int kpad, int wpk);
cudaError_t launch_ts(const LaunchTs& L, cudaStream_t st);

// (columns per phenotype slot, phenotypes per group) pairs with a compiled
// many-phenotype kernel; the group width NP * PPG is at most 128.
#define KG_MP_GROUPS(X)                                                                      \
  X(16, 1) X(16, 2) X(16, 4) X(16, 8) X(32, 1) X(32, 2) X(32, 4) X(48, 1) X(48, 2) X(64, 1) \
  X(64, 2) X(80, 1) X(96, 1) X(112, 1) X(128, 1)

// Streamed image (kernel_tb.cu): tiles in pairs against a limb image that does
// not fit shared memory, one phenotype (O1) or many (O).
struct LaunchTb {
  const uint64_t* x;          // packed rows (device), 16-byte aligned
  unsigned long long m;
  int wpk;
  int kpad;                   // samples per group image (multiple of 128)
  int NP, PPG, G;             // columns per phenotype slot, phenotypes per group (KG_MP_GROUPS), groups
  const int8_t* Bimg;         // G images of kpad x NP*PPG bytes in the make_b_image_ts layout (device)
  const MPheno* ph;           // per-phenotype constants (device)
  const DevOutMP* O;
  const DevOut* O1;           // one phenotype: its outputs (O unused)
  int num_sms;
  bool fp64 = false;          // one phenotype in the FP64 form (image of launch_f64_image)
};
// The FP64 form on the tensor cores: U columns in 7 limbs, y' in 8.
struct LaunchF64Image {
  const double* V;            // FP64 columns (LaunchFp64::V), vrows x cm
  int vrows, cm, k;
  bool drop0;                 // U column 0 has a single limb
  int kpad, N;                // f64_limb_cols columns
  const double* up;           // k + 1 scales 2^s (powers of two) of the columns, y' last
  int8_t* img;                // kpad x N bytes (device)
};
int f64_limb_cols(int k, bool drop0);
bool f64_limbs_supported(int N, int n_row, int wpk);
cudaError_t launch_f64_image(const LaunchF64Image& L, cudaStream_t st);
bool tb_supported(int N, int wpk);
int tb_tiles(unsigned long long m, int num_sms);  // tiles per item of a launch
int tb_ring(int N);                               // image chunks in the ring
cudaError_t launch_tb(const LaunchTb& L, cudaStream_t st);

// 4-bit screen (kernel_fs.cu), one phenotype (O1) or many (O).
struct LaunchFs {
  const uint64_t* x;          // packed rows (device), 16-byte aligned
  unsigned long long m;
  int wpk;
  int kpad;                   // samples per image (multiple of 256)
  int NP, PPG, G;             // columns per phenotype slot, phenotypes per group, groups
  int lu;                     // limbs per U column
  bool gate;                  // the columns hold y - mean(y)
  int bt;                     // tiles of a CTA per pass over the groups (G > 1)
  const uint8_t* Bimg;        // G images of kpad * NP * PPG / 2 bytes (put_fs_image; device)
  const FsPheno* F1;          // one phenotype: its constants (host)
  const FsPheno* ph;          // many: per-phenotype constants (device)
  const DevOutMP* O;
  const DevOut* O1;
  int num_sms;
};
// (columns per phenotype slot, phenotypes per group) with a many-phenotype
// screen: groups of at most 112 columns.
#define KG_FS_GROUPS(X)                                                                                    \
  X(8, 1) X(8, 3) X(8, 8) X(16, 1) X(16, 2) X(16, 4) X(16, 6) X(24, 1) X(24, 2) X(24, 4) X(32, 1) X(32, 2) \
  X(32, 3) X(40, 1) X(40, 2) X(48, 1) X(48, 2) X(56, 1) X(56, 2) X(64, 1) X(72, 1)
// (columns, limbs per U column) with a single-phenotype screen.
#define KG_FS_SINGLE(X)                                                                                         \
  X(8, 1) X(16, 1) X(24, 1) X(32, 1) X(40, 1) X(48, 1) X(56, 1) X(64, 1) X(72, 1) X(80, 1) X(16, 2) X(32, 2) \
  X(48, 2) X(64, 2) X(80, 2) X(96, 2) X(112, 2)
// Columns of one phenotype's slot: a width that has a kernel.
inline int fs_width(bool gate, int lu, int ku) {
  const int q = lu == 2 ? 16 : 8, w = (4 + (gate ? 4 : 0) + lu * ku + q - 1) / q * q;
  return w > 80 ? (w + 15) / 16 * 16 : w;
}
bool fs_supported(int N, int kpad, int wpk);
cudaError_t launch_fs(const LaunchFs& L, cudaStream_t st);
// The rows of x (16-byte aligned, wpk words each; indices from `offset`) that a
// screen with these counters has listed in cand, to dst.
cudaError_t launch_fs_gather(const uint64_t* x, int wpk, const unsigned long long* cand,
                             const unsigned long long* counters, unsigned long long offset, uint64_t* dst, int num_sms,
                             cudaStream_t st);

// Launches k, with `behind` so that its start overlaps the end of the launch before
// it in the stream (programmatic dependent launch; k then calls wait_for_previous
// first).  A kernel that ends at once behind the screen costs a call 2 us so, 6 us
// otherwise.  Not for the refinement: its tables go through the L1 cache, which the
// kernel before it leaves little of (8 phenotypes at n = 5000: 1.06 -> 1.11 ms).
template <class... P, class... A>
cudaError_t launch_behind(bool behind, void (*k)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st,
                          A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = behind ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

struct LaunchMpRefine {
  const uint64_t* x;
  int wpk;
  const double* V;            // n_pheno blocks of vrows x cm FP64 (device)
  int vrows, cm;
  unsigned long long vstride;
  const MPheno* ph;
  const DevOutMP* O;
  int num_sms;
  const double* T = nullptr;  // byte tables of V, refine_table_len(vrows, cm) doubles per phenotype
};
bool mp_supported(int NP, int PPG, int wpk);  // shapes of the many-phenotype kernels
// 2-D TMA map of packed rows: boxes of 128 bytes x `rows` rows, 128-byte swizzle.
bool mp_tmap(const uint64_t* x, unsigned long long m, int wpk, CUtensorMap_st* tm, int rows = 128);

// B-stationary many-phenotype kernel (kernel_mpb.cu): each group's image
// (make_b_image_ts layout, kpad x NP*PPG bytes) resident in shared memory for
// a pass over `bt` tile-iterations of every CTA.
struct LaunchMpb {
  const uint64_t* x;
  unsigned long long m;
  int wpk;
  int kpad;
  int NP, PPG, G;
  int bt;                     // tile-iterations per L2 block
  const int8_t* Bimg;         // G images of kpad x NP*PPG bytes (device)
  const MPheno* ph;
  const DevOutMP* O;
  int num_sms;
};
bool mpb_supported(int NP, int PPG, int kpad, int wpk);  // the image and the x ring fit in shared memory
size_t mpb_smem_bytes(int N, int kpad);
cudaError_t launch_mpb(const LaunchMpb& L, cudaStream_t st);
cudaError_t launch_mp_refine(const LaunchMpRefine& L, cudaStream_t st);

// Pair-of-SMs many-phenotype kernel (kernel_mpb2.cu): a cluster of two CTAs
// issues M = 256 tcgen05 MMAs (cta_group::2) over two phenotypes at once
// (N = 2 * NP), each CTA holding one phenotype's image (kpad x NP, the
// one-phenotype-per-group image of LaunchMpb with PPG = 1; L.G = phenotypes)
// and 128 k-mers of each 256-k-mer pair-tile.
bool mpb2_supported(int NP, int kpad, int wpk);
size_t mpb2_smem_bytes(int NP, int kpad);
cudaError_t launch_mpb2(const LaunchMpb& L, cudaStream_t st);

// 2-D pair test (kernel_pairs.cu): the TMEM-A pipeline on x_i AND x_j.
struct LaunchPairs {
  const uint64_t* x;          // packed rows (device), 16-byte aligned, wpk >= 16
  int wpk;
  int kpad;
  bool drop0;
  PairSched S;
  const int8_t* Bimg;         // make_b_image_ts layout (device)
  const EpiParams* P;
  const LimbMap* LM;
  const DevOutPairs* O;
  int num_sms;
};
struct LaunchPairRefine {
  const uint64_t* x;
  int wpk;
  const double* T;            // byte tables of V (refine_table_len(vrows, cm) doubles)
  int vrows, cm;
  const EpiParams* P;
  const DevOutPairs* O;
  int num_sms;
  const LimbMap* LM;          // behind the 4-bit screen: the int8 limb columns,
  const double* V;            // and the FP64 columns, vrows x cm
};
// The pair test with the 4-bit screen (kernel_fsp.cu).
struct LaunchFsPairs {
  const uint64_t* x;          // packed rows (device), 16-byte aligned, wpk >= 16
  int wpk;
  int kpad;                   // samples of the image (multiple of 256)
  int N, lu;                  // its columns and limbs per U column
  bool gate;                  // it holds y - mean(y)
  PairSched S;
  const uint8_t* Bimg;
  const FsPheno* F;           // host
  const DevOutPairs* O;
  int num_sms;
};
bool fsp_supported(int N, int lu, int kpad, int wpk, unsigned long long ic);
cudaError_t launch_fs_pairs(const LaunchFsPairs& L, cudaStream_t st);
bool pairs_supported(int N, int limbs_u, int limbs_y, int kpad, int wpk);
cudaError_t launch_pairs(const LaunchPairs& L, cudaStream_t st);
cudaError_t launch_pair_refine(const LaunchPairRefine& L, cudaStream_t st);

int tc_kc();                  // samples per K chunk of the tensor-core kernel
bool tc_supported_n(int N);
cudaError_t launch_tc(const LaunchTc& L, cudaStream_t st);

}  // namespace kg
