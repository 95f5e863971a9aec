// params.hpp -- kernel parameter blocks shared by host and device code.
#pragma once
#include <cmath>
#include <cstdint>

#include "../../include/kgwas_cuda.h"
#include "prep.hpp"

namespace kg {

// Single-precision screen of one k-mer (screen_kmer in device.cuh): decides
// from the limb sums, with room for its own rounding, that a k-mer is not
// tested, or is tested and cannot reach the emit or the refinement cut.
// Everything about y is relative to ||y - mean(y)||.
struct alignas(16) ScreenParams {
  int on;            // 0: every k-mer takes the FP64 statistic
  int shift;         // limb sums are shifted right by this into 32 bits
  float inv_n;       // 1 / n
  float b, kappa;    // b / ynorm, kappa / ynorm
  float cut;         // 0.9 x the lowest r2 that matters x yyM / ynorm^2
  float gate_lo, gate_hi;  // (corr_thr -+ margin)^2
  float sy;          // y' limb sums -> e_y / ynorm
  int gate;          // corr_thr > 0
  int pad[2];
  float su[KMAX];    // limb sums of U column j + 1 -> e_(j+1) (column 0: the intercept)
  float g[KMAX];     // g_(j+1) / ynorm
};

// Per-phenotype constants of the epilogue (prep.hpp notation).
struct EpiParams {
  int n, k;
  double b, kappa, yyM, ynorm, corr_thr, p_thresh;
  double r2_cand;   // r2 below this cannot give p <= p_thresh (log/erfc skipped)
  int refine;       // 1: k-mers with r2 >= r2_ref go to the FP64 refinement list
  double r2_ref;
  double r2_need;   // refinement may skip k-mers with r2 in [r2_ref, r2_need), see may_refine; 0: none
  double thr2_ynorm2;  // corr_thr^2 * ynorm^2 (division-free Pearson gate)
  double gate_unit;    // the limbs' rounding moves x.(y - mean) by at most popcount(x) times this
  double a[KMAX];
  double g[KMAX];
  ScreenParams S;
};

// Column map of the int8 limb contraction (prep.hpp LimbCols).
struct LimbMap {
  int N, count_col;
  int first[KMAX + 1];
  int nl[KMAX + 1];
  double scale[KMAX + 1];
  // Epilogue constants of the kernels whose accumulators hold -128 * digit
  // sums (set_limb_consts): for the recombined integer V, biased to the
  // double 1.5 * 2^52 + V, e = fma(biased, esc, eoff) = V * (-scale / 128)
  // exactly (both factors are powers of two times integers).
  double esc[KMAX + 1];   // -scale / 128
  double eoff[KMAX + 1];  // 1.5 * 2^52 * scale / 128
};

inline void set_limb_consts(LimbMap& L) {
  for (int j = 0; j <= KMAX; ++j) {
    L.esc[j] = -L.scale[j] / 128.0;
    L.eoff[j] = 6755399441055744.0 * L.scale[j] / 128.0;
  }
}

// Smallest share of c (n - c) / n at which xxM is used to place a k-mer below a
// cut, and how far below the cut it has to be.
constexpr double XXM_FLOOR = 0.02, CUT_ROOM = 0.9;

// Whether r2 = xyM^2 / (xxM yyM) below CUT_ROOM of a cut means that the exact r2
// is below the cut, where xxM is at least XXM_FLOOR of xcn = c (n - c) / n.  u and
// y: errors of (s_1 ..) and of xyM over sqrt(yyM cut), in units of sqrt(xcn).
// xxM = xcn - |s|^2 with |s|^2 <= xcn is then off by at most (2 u + u^2) xcn.
inline bool cut_room_covers(double u, double y) {
  const double rho = (2.0 * u + u * u) / XXM_FLOOR, root = std::sqrt(CUT_ROOM) + y / std::sqrt(XXM_FLOOR);
  return rho < 1.0 && root * root <= 0.999 * (1.0 - rho);
}

// The part of the refinement range that a launch without per-k-mer outputs
// leaves out: a k-mer whose r2 in the split form is below CUT_ROOM of the emit cut
// is not emitted whatever the refinement gives, as long as the split form's
// xxM is at least XXM_FLOOR of c (n - c) / n (may_refine) and the limbs are good
// enough for that.  They are not where many values of a column are rounded the
// same way (columns that mark single samples, n above about 10,000): there
// every k-mer from r2_ref up is refined.
inline void set_refine_need(EpiParams& P, const LimbLoss& B) {
  P.r2_need = cut_room_covers(B.u, B.y / std::sqrt(P.yyM * P.r2_cand)) ? CUT_ROOM * P.r2_cand : 0.0;
}

// EpiParams::gate_unit: half a unit of the last limb of every column, U columns
// weighted as the gate sums them.
inline void set_gate_unit(EpiParams& P, const LimbMap& L, bool drop0) {
  P.gate_unit = 0.5 * L.scale[P.k];
  for (int j = drop0 ? 1 : 0; j < P.k; ++j) P.gate_unit += 0.5 * std::fabs(P.g[j]) * L.scale[j];
}

// Screen constants of a phenotype whose intercept carries no limbs (drop0)
// and whose limb columns are those of L: 3 per U column and 5 for y', of which
// the lowest is not read, or with f64 the FP64 form's 7 and 8, of which the four
// highest are read.  No screen where its margins (screen_verdict) do not cover
// its rounding: the limb sums, shifted into 32 bits, and the digits that are not
// read are off by at most two units S.su (S.sy) each, single precision by a few
// 2^-24 of every term, and 1 / sqrt(xcn) is at most 1.5.
inline void set_screen(EpiParams& P, const LimbMap& L, bool drop0, const LimbLoss& B, bool f64 = false) {
  ScreenParams& S = P.S;
  S = ScreenParams();
  // a cut from r2_need stands for the exact r2, the others for the limb sums' own
  double cut = P.r2_cand, lost_u = 0.0, lost_y = 0.0;
  if (P.refine && P.r2_ref < cut) {
    cut = P.r2_ref;
    if (P.r2_need > cut) {
      cut = P.r2_need;
      lost_u = B.u;
      lost_y = B.y / P.ynorm;
    }
  }
  const double yv = P.yyM / (P.ynorm * P.ynorm);
  // c - s_0^2 = c (n - c) / n, which the screen uses, holds for a unit intercept
  if (!(drop0 && std::fabs(P.a[0] * P.a[0] * P.n - 1.0) <= 1e-6) || !(P.ynorm >= 1e-12) || !(P.ynorm < 1e150) || !(cut > 0) || !(yv > 1e-6) || P.n >= 65536) return;
  while ((4 << S.shift) < P.n) ++S.shift;
  S.inv_n = (float)(1.0 / P.n);
  S.b = (float)(P.b / P.ynorm);
  S.kappa = (float)(P.kappa / P.ynorm);
  S.cut = (float)(CUT_ROOM * cut * yv);
  const double eps = 1e-4 * (P.n > 1024 ? P.n / 1024.0 : 1.0);
  const double lo = P.corr_thr > eps ? P.corr_thr - eps : 0.0, hi = P.corr_thr + eps;
  S.gate_lo = (float)(lo * lo);
  S.gate_hi = (float)(hi * hi);
  S.gate = P.corr_thr > 0.0;
  // accumulators hold -128 x the digit sums
  const double unit = -(double)(1 << S.shift) / 128.0, low3 = f64 ? 4294967296.0 : 1.0;  // 2^8 of the shift, 256^3
  S.sy = (float)(unit * (f64 ? low3 * 256.0 : 65536.0) * L.scale[P.k] / P.ynorm);
  double units2 = 0.0, gate = 0.0;
  const double round = (P.k + 16) * 5.97e-8;  // of every term of a sum
  for (int j = 1; j < P.k; ++j) {
    S.su[j - 1] = (float)(unit * low3 * L.scale[j]);
    S.g[j - 1] = (float)(P.g[j] / P.ynorm);
    const double e = 2.0 * std::fabs((double)S.su[j - 1]);
    units2 += e * e;
    gate += std::fabs((double)S.g[j - 1]) * (1.5 * e + round * B.norm[j]);
  }
  const double ey = 3.0 * std::fabs((double)S.sy) + round * B.norm[P.k] / P.ynorm;
  const double u = lost_u + 1.5 * std::sqrt(units2) + round;
  const double y = lost_y + ey + round * std::fabs((double)S.b) * P.n;
  gate += ey + round * std::fabs((double)S.kappa) * P.n;
  S.on = cut_room_covers(u, y / std::sqrt(cut * yv)) && (!S.gate || gate <= 0.5 * eps);
}

// Constants of one phenotype for the 4-bit screen (kernel_fs.cu); everything
// about y is relative to ynorm.
struct alignas(16) FsPheno {
  float n, inv_n;         // samples
  float cut, pad;         // lowest r2 of an emitted row x yyM / ynorm^2
  float b, kappa, thr;    // b / ynorm, kappa / ynorm, the correlation threshold
  float bu, mu;           // bounds of what the limbs leave out (fs_verdict): U columns,
  float by, my, bg;       // y' and
  float sy[3];            // limb sums of y' -> e_y
  float mg;               // y - mean(y)
  float sg[4];            // limb sums of y - mean(y)
  float su[2 * KMAX];     // limb sums of the U columns, one or two limbs each
};

// Refinement candidates: marks of entries whose correlation gate is not decided.
constexpr unsigned long long CAND_OPEN = 1ull << 63, CAND_OPEN_MP = 1ull << 47;

// Counters of a launch (device): [0] tested, [1] hits, [2] error bits, [3]
// refinement candidates, and those of the 4-bit screen: the tests that it has
// decided, its undecided ones (candidates in the place of [3]'s), whether it has
// given up in this launch and in any launch of the call.
constexpr int CNT_FS_TESTED = 4, CNT_FS_OPEN = 5, CNT_FS_OVER = 6, CNT_FS_EVER = 7, NCOUNT = 8;

// Undecided tests at which the screen gives up, and a kernel that evaluates every
// test runs in its place.  A row near the span of U (a marker of a lineage) is
// undecided whatever its statistic, and refining one costs as much as screening a
// hundred (3 ns and 0.03 ns on the whole device at n = 1000, r = 16+1).  While an
// eighth of the tests are done the limit is one in 128 of those, so that rows of one
// kind are found out early, later one in 64 of all; calls of up to `base` tests never
// give up.  1e7 rows at n = 1000, r = 16+1, of which 0, 1, 3, 10 and 100 % are lineage
// markers, about half of them undecided: 0.30, 0.46, 0.79, 1.9 and 16 ms with all
// of those refined; now 0.30, 0.47, 0.49, 0.50 and 0.49; 0.47 without the screen.
constexpr unsigned long long FS_OPEN_BASE = 4096;
__host__ __device__ inline unsigned long long fs_open_limit(unsigned long long base, unsigned long long done,
                                                            unsigned long long total, unsigned long long cap) {
  const unsigned long long v = total > base && 8 * done <= total ? base / 4 + done / 128 : base + total / 64;
  return v < cap ? v : cap;
}
// Candidates that a launch of so many tests may have to list (at most 128 MB).
inline unsigned long long fs_cand_room(unsigned long long base, unsigned long long total) {
  const unsigned long long v = fs_open_limit(base, total, total, 1ull << 24);
  return v > (1ull << 20) ? v : 1ull << 20;
}

// Device outputs of one launch.
struct DevOut {
  unsigned long long* counters;
  kg_hit* hits;
  unsigned long long hit_cap;
  unsigned long long kmer_offset;  // added to the launch-local k-mer index
  // optional per-k-mer arrays, indexed by kmer_offset + local index
  uint8_t* tested;
  double *chisq, *pval, *effect, *mlog10p, *xxM, *xyM, *cor;
  // FP64 refinement list (global k-mer indices), used when EpiParams::refine
  unsigned long long* cand;
  unsigned long long cand_cap;
  // optional: a tested k-mer counts weight[kmer_offset + local] times in
  // counters[0] (a row that stands for a run of equal rows)
  const uint32_t* weight;
  // pipeline wait limit in ns (0: WAIT_LIMIT_NS)
  unsigned long long wait_ns;
  // test hook of the bounded waits: when non-zero, the row producer of each
  // CTA issues this many row loads and then stops, so that the consumers'
  // waits run out (0: off)
  unsigned long long stall_loads;
  // fs_kernel: the base of fs_open_limit; no undecided k-mer is counted as tested
  // (the kernel that takes them counts them)
  unsigned long long open_base;
  int count_sure;
  // tb_kernel, FP64 form: the rows are the gathered rows of the k-mers
  // index[0 .. *rows), at most m
  const unsigned long long* index;
  const unsigned long long* rows;
  // a launch behind the screen: its counter CNT_FS_OVER.  The kernels run only
  // where the screen has given up, the refinement and what reads `rows` take its
  // candidates where it has not
  const unsigned long long* over;
  __host__ __device__ unsigned long long kmer(unsigned long long local) const {
    return index ? index[local] : kmer_offset + local;
  }
};

enum : unsigned { ERR_TIMEOUT_FULL = 1u, ERR_TIMEOUT_MMA = 2u, ERR_HIT_OVERFLOW = 4u, ERR_CAND_OVERFLOW = 8u };

// Chi-square above which the split form hands a k-mer to the FP64
// refinement kernel: there -log10 p ~ T / (2 ln 10) grows with T, so an
// absolute 1e-6 bound needs FP64 accuracy; below it 24-bit U limbs suffice.
constexpr double REFINE_CHISQ = 12.0;

// One phenotype of a multi-phenotype launch (device memory).
struct MPheno {
  EpiParams P;
  LimbMap LM;       // limb columns relative to the phenotype's slot in its group
  int drop0;        // U column 0 carries no limbs (intercept handled in FP64)
  int pad;
};

// Outputs of a multi-phenotype launch.
struct DevOutMP {
  unsigned long long* counters;
  unsigned long long* tested;        // [shard * n_pheno + pheno]
  kg_phit* hits;
  unsigned long long hit_cap;
  unsigned long long* cand;          // kmer | pheno << 48
  unsigned long long cand_cap;
  const unsigned long long* shard_start;  // ascending, global k-mer indices
  int n_shards;
  int n_pheno;
  unsigned long long kmer_offset;
  // optional: a tested (k-mer, phenotype) counts weight[global k-mer] times
  // (a row that stands for a run of equal rows)
  const uint32_t* weight;
  // pipeline wait limit in ns (0: WAIT_LIMIT_NS)
  unsigned long long wait_ns;
  // test hook of the bounded waits, as DevOut::stall_loads (0: off)
  unsigned long long stall_loads;
  // behind the screen, as DevOut::over; its counts, which the refinement adds to
  // `tested` where it has not given up, and clears
  const unsigned long long* over;
  unsigned long long* fs_tested;
  unsigned long long open_base;      // of fs_open_limit
};

// Outputs of the 2-D pair test (kernel_pairs.cu).
struct DevOutPairs {
  unsigned long long* counters;  // [0]: evaluated pairs
  kg_pair* hits;
  unsigned long long hit_cap;
  unsigned long long* cand;      // i << 32 | j
  unsigned long long cand_cap;
  unsigned long long wait_ns;    // pipeline wait limit in ns (0: WAIT_LIMIT_NS)
  const unsigned long long* over;  // behind the screen, as DevOut::over
  unsigned long long open_base;    // of fs_open_limit
};

// Pair schedule: pairs (i, j), i < j, row_start <= i < row_end, j < n_kmers.
// Unit u covers j-block jb (j in [128 jb, 128 jb + 128)) and up to `ic`
// consecutive i; units of j-block jb are unit_off[jb] .. unit_off[jb+1]-1.
struct PairSched {
  const unsigned long long* unit_off;  // njb + 1 entries (device)
  int njb;
  unsigned long long n_units, n_kmers, row_start, row_end, ic;
};

}  // namespace kg
