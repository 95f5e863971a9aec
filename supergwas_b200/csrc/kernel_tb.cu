// kernel_tb.cu -- the association test against a limb image that does not fit
// shared memory: tiles in pairs, the image streamed.
//
// One phenotype of a large cohort (n = 5000 at r = 32+1: 560 KB of limbs), or
// many (src/kgwas.cpp:44-56, 132-218 once per k-mer and phenotype).  A CTA
// takes T = 2 tiles of 128 k-mers at a time (one when there are too few tiles
// for every SM) and runs every phenotype group over them; the group's image
// streams from L2 in chunks of 256 samples, each chunk used by both tiles.
// The work of a pair of tiles and a group is an item; its super-stages (512
// samples of one tile) alternate between the tiles.
//
// Warps (16, 128 registers a thread):
//   0-3    epilogue: the accumulators of an item's tiles in turn (screen, and
//          the FP64 statistic near a cut, as in the other kernels); items are
//          long (2 x 9000 MMA cycles at n = 5000), so one group and one
//          accumulator per tile do;
//   4-11   unpack, two groups, one TMEM A slot each: packed rows -> int8;
//   12     row producer: 2-D TMA loads of 128 rows x 128 bytes (no multicast);
//   13     image producer: one bulk copy per chunk into a ring;
//   14-15  MMA, one warp per tile of the pair: tcgen05.mma kind::i8, A from
//          TMEM, B from the ring.
//
// Per SM the image takes 256 N bytes per 16 N/2 MMA cycles, 32 bytes per cycle
// (L2 delivered over 100 per cycle and SM to bulk copies of 56 KB, measured).
// The kernel that this replaces streamed 128 samples at a time for one tile,
// with two waits and two commits per four MMAs: 1200 cycles per 224 cycles of
// MMAs.  8 phenotypes x 1e6 k-mers at n = 5000, r = 32+1: 10.9 -> 3.28 ms; one
// phenotype x 2e6, which ran on the smem-A kernel: 3.74 -> 0.96 ms.  At 1.63 ms
// per 8 x 5e5 the MMAs take 61 % of the time; the unpack feeds them.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "device.cuh"
#include "kernels.hpp"

namespace kg {

constexpr int TB_TM = 128;
constexpr int TB_KS = 128;     // samples per sub-stage (4 MMAs)
constexpr int TB_SUPER = 4;    // sub-stages per super-stage
// Sub-stages per image chunk: one for the widest images of the FP64 form, whose
// ring of three chunks of two would not fit.
__host__ __device__ constexpr int tb_chunk(int N) { return N > 192 ? 1 : 2; }
constexpr int TB_UG = 2;       // unpack groups = A slots of 128 TMEM columns
constexpr int TB_XST_MAX = 6, TB_XST_MIN = 4, TB_NB_MAX = 8, TB_NB_MIN = 3;
constexpr int TB_WUNP = 4, TB_WXP = TB_WUNP + 4 * TB_UG, TB_WBP = TB_WXP + 1, TB_WMMA = TB_WBP + 1;
constexpr int TB_THREADS = 32 * (TB_WMMA + 2);
constexpr int TB_A0 = 512 - TB_UG * 128;

struct TbSmem {
  uint32_t x, b, bars, tmem, abort, total;
};
__host__ __device__ inline TbSmem tb_smem(int N, int xst, int nb, int rb) {
  TbSmem L;
  L.x = 0;
  L.b = (uint32_t)xst * TB_TM * rb;
  L.bars = L.b + (uint32_t)nb * tb_chunk(N) * TB_KS * N;
  L.tmem = L.bars + 8 * (2 * TB_XST_MAX + 2 * TB_NB_MAX + 2 * TB_UG + 4 + 2);
  L.abort = L.tmem + 8;
  L.total = L.abort + 8;
  return L;
}

// One phenotype, outputs of kernel_ts.cu (DevOut).
template <int N>
__device__ __forceinline__ void tb_single(const DevOut& O, const MPheno* ME, uint32_t taddr, unsigned long long local,
                                          bool valid, uint32_t& tested_local) {
  const EpiParams& P = ME->P;
  if (!O.tested) {
    const int v = mp_screen<N>(P, taddr, valid);
    if (!__any_sync(0xffffffffu, v == 2)) {
      if (v) tested_local += O.weight ? O.weight[O.kmer_offset + local] : 1u;
      return;
    }
  }
  int c = 0;
  double cd = 0, ey = 0, ss = 0, gs = 0;
  mp_exact_chunk<N, 0>(ME, taddr, c, cd, ey, ss, gs);
  if (N > MP_CH) mp_exact_chunk<N, 1>(ME, taddr, c, cd, ey, ss, gs);
  if (N > 2 * MP_CH) mp_exact_chunk<N, 2>(ME, taddr, c, cd, ey, ss, gs);
  if (O.tested) finish_kmer(P, O, local, valid, c, ss, gs, ey);
  else finish_kmer_lean(P, O, local, valid, c, cd, ss, gs, ey, tested_local);
}

// ---------------------------------------------------- FP64 form in limbs
// Columns: the count, 8 limbs of y', one for the centred part of U column 0 where
// that is rounding noise of U itself (drop0), 7 of every other U column (62 and 54
// bits below the column's largest value, so at least what a double holds of
// it).  The sums are exact and rounded once, where fp64_kernel rounds after
// every sample: the error against 64 bits is that of fp64_kernel or below it
// (8.2e-14 and 3.1e-13 in p-values at n = 1000 were the same on both).
// fp64_kernel does n (k + 2) FP64 multiply-adds per k-mer, half of whose time
// goes to broadcasting the columns from shared memory; here they are int8 MMAs
// of 9 + 7 k columns.  5e6 k-mers, r = 10+1, n = 1000: 9.70 -> 0.37 ms; 3e5 at
// n = 5000, r = 32+1: 6.79 -> 0.22 ms; 5e6 at n = 200, r = 5+1: 1.25 -> 0.16 ms.
constexpr int F64_LY = 8, F64_LU = 7;
constexpr int F64_E0 = 1 + F64_LY, F64_U = F64_E0 + 1;  // the noise column, the first U column with 7 limbs

__device__ __forceinline__ long long limb4(const uint32_t* d) {
  return mad_wide<(1 << 24)>(d[0], limb3(d[1], d[2], d[3]));
}

// Reads the N accumulator columns at taddr, 32 at a time, and hands over the
// count and y' (first(d)) and then the 7 limbs of each of the ku U columns
// (column(j, d)) as they arrive.
template <int N, class F, class G>
__device__ __forceinline__ void f64_columns(uint32_t taddr, int ku, F first, G column) {
  constexpr int KU = (N - F64_U) / F64_LU;
  uint32_t d[N];
#pragma unroll
  for (int q = 0; q < N; q += 32) {
#pragma unroll
    for (int c16 = q; c16 < q + 32 && c16 < N; c16 += 16) tc_ld16p(taddr + c16, d + c16);
    tc_wait_ld();
#pragma unroll
    for (int c16 = q; c16 < q + 32 && c16 < N; c16 += 16) reg_fence16(d + c16);
    if (q == 0) first(d);
#pragma unroll
    for (int j = 0; j < KU; ++j) {
      const int o = F64_U + F64_LU * j;
      // N is rounded up to 16: at most two groups past the last column
      if (o + F64_LU - 1 >= q && o + F64_LU - 1 < q + 32 && (j < KU - 2 || j < ku)) column(j, d + o);
    }
  }
}

template <int N, bool GATE>
__device__ __forceinline__ int f64_screen(const EpiParams& P, uint32_t taddr, int ku, bool valid) {
  const ScreenParams& S = P.S;
  int c = 0;
  float ey = 0.0f, ss = 0.0f, gs = 0.0f;
  f64_columns<N>(
      taddr, ku,
      [&](const uint32_t* d) {
        c = (-(int)d[0]) >> 7;
        ey = shifted_float(limb4(d + 1), S.shift + 8) * S.sy;
      },
      [&](int j, const uint32_t* d) {
        const float e = shifted_float(limb4(d), S.shift + 8) * __ldg(S.su + j);
        ss = fmaf(e, e, ss);
        if (GATE) gs = fmaf(__ldg(S.g + j), e, gs);
      });
  return screen_verdict<GATE, false>(S, P.n, c, ey, ss, gs, valid);
}

// One phenotype in the FP64 form: the sums of fp64_kernel (kernels.cu), each
// rounded once, then its statistic.  Without per-k-mer outputs the screen
// decides most k-mers first.
template <int N>
__device__ __forceinline__ void tb_single64(const DevOut& O, const MPheno* ME, uint32_t taddr,
                                            unsigned long long local, bool valid, uint32_t& tested_local) {
  const EpiParams& P = ME->P;
  const int drop0 = ME->drop0, ku = P.k - drop0;
  if (!O.tested && P.S.on) {
    const int v = P.S.gate ? f64_screen<N, true>(P, taddr, ku, valid) : f64_screen<N, false>(P, taddr, ku, valid);
    if (!__any_sync(0xffffffffu, v == 2)) {
      if (v) tested_local += O.weight ? O.weight[O.kmer(local)] : 1u;
      return;
    }
  }
  int c = 0;
  double cd = 0, ey = 0, ss = 0, gs = 0;
  f64_columns<N>(
      taddr, ku,
      [&](const uint32_t* d) {
        c = (-(int)d[0]) >> 7;
        cd = i2d_exact(c);
        const double sy = ME->LM.esc[P.k];
        ey = fma(i2d_exact(limb4(d + 1)), sy * 4294967296.0, i2d_exact(limb4(d + 5)) * sy);
        if (drop0) {
          const double e0 = i2d_exact((int)d[F64_E0]) * ME->LM.esc[0], s0 = fma(P.a[0], cd, e0);
          ss = s0 * s0;
          gs = P.g[0] * e0;
        }
      },
      [&](int jj, const uint32_t* d) {
        const int j = jj + drop0;
        const double su = ME->LM.esc[j];
        const double e = fma(i2d_exact(limb4(d)), su * 16777216.0, i2d_exact(limb3(d[4], d[5], d[6])) * su);
        const double sj = fma(P.a[j], cd, e);
        ss = fma(sj, sj, ss);
        gs = fma(P.g[j], e, gs);
      });
  finish_kmer(P, O, local, valid, c, ss, gs, ey);
}

// The image of the FP64 form from the FP64 columns V (row = sample position:
// count, d_0 .. d_{k-1}, d_y, cm apart), in the layout and with the digits
// (of v, or of -2 v where a sample enters as 64 x) of put_b_image_ts.  One
// thread per sample position and logical column (0: count, 1: y', 2 + j: U
// column j + drop0).
struct F64Scales {
  double up[KMAX + 1];  // 2^s of U column j; [k]: y'
};
__global__ void __launch_bounds__(128) f64_image_kernel(const double* __restrict__ V, int vrows, int cm, int k,
                                                        int drop0, int kpad, int N,
                                                        const __grid_constant__ F64Scales S,
                                                        int8_t* __restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, col = blockIdx.y;
  if (i >= kpad) return;
  const int a = i >> 7, q = (i >> 5) & 3, t = (i >> 3) & 3, jj = 7 - (i & 7);
  const int kap = 128 * a + 4 * (8 * q + jj) + t;
  if (col == 2 && !drop0) return;
  const int j = col < 2 ? k : col == 2 ? 0 : col - 3 + drop0;  // U column (k: y')
  const int vc = col == 0 ? 0 : 1 + j;
  const int L = col == 0 || col == 2 ? 1 : col == 1 ? F64_LY : F64_LU;
  const int first = col == 0 ? 0 : col == 1 ? 1 : col == 2 ? F64_E0 : F64_U + F64_LU * (col - 3);
  long long v = 0;
  if (i < vrows) v = __double2ll_rn(V[(size_t)i * cm + vc] * (col == 0 ? 1.0 : S.up[j]));
  if (jj & 1) v *= -2;
  for (int l = L - 1; l >= 0; --l) {
    const int8_t digit = (int8_t)(v & 255);  // balanced: [-128, 127]
    v = (v - digit) >> 8;
    const int cc = first + l;
    img[(size_t)(kap >> 4) * (N * 16) + (size_t)(cc >> 3) * 128 + (size_t)(cc & 7) * 16 + (kap & 15)] = digit;
  }
}

// FORM: TB_MANY phenotypes to O; TB_ONE phenotype (G = 1) to O1; TB_ONE64 the
// same in the FP64 form.
enum { TB_MANY, TB_ONE, TB_ONE64 };
template <int NP, int PPG, int FORM>
__global__ void __launch_bounds__(TB_THREADS, 1)
    tb_kernel(const __grid_constant__ CUtensorMap tmap, unsigned long long m, int nbox, int nsub, int G, int T,
              int xst, int nb, int rb, const int8_t* __restrict__ Bimg, unsigned long long img_bytes,
              const MPheno* __restrict__ ph, const DevOutMP O, const DevOut O1) {
  constexpr int N = NP * PPG;
  static_assert(N <= (FORM == TB_ONE64 ? 256 : 128) && N % 16 == 0, "group width");  // T * N <= 256
  constexpr bool SINGLE = FORM != TB_MANY;
  constexpr uint32_t IDESC = idesc_i8(TB_TM, N);
  constexpr uint32_t BSTEP = (2 * N * 16) >> 4;             // descriptor step of one K = 32 MMA
  constexpr int TB_CHUNK = tb_chunk(N);
  constexpr uint32_t BCH = (uint32_t)TB_CHUNK * TB_KS * N;  // bytes of one image chunk
  constexpr int NK = TB_CHUNK * (TB_KS / 32);               // MMAs per chunk
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  const uint32_t xbytes = TB_TM * (uint32_t)rb, swz = rb == 128 ? 7u : 0u;  // boxes as in kernel_ts.cu
  const TbSmem L = tb_smem(N, xst, nb, rb);
  const uint32_t sx = base + L.x, sb = base + L.b;
  const uint32_t x_full = base + L.bars, x_empty = x_full + 8 * TB_XST_MAX;
  const uint32_t b_full = x_empty + 8 * TB_XST_MAX, b_empty = b_full + 8 * TB_NB_MAX;
  const uint32_t a_full = b_empty + 8 * TB_NB_MAX, a_empty = a_full + 8 * TB_UG;
  const uint32_t acc_full = a_empty + 8 * TB_UG, acc_empty = acc_full + 16, drain = acc_empty + 16;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(gbase + L.tmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(gbase + L.abort);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned long long* const counters = SINGLE ? O1.counters : O.counters;
  const unsigned long long lim = wait_limit(SINGLE ? O1.wait_ns : O.wait_ns);
  // behind the screen: the rows that it has left (FP64 form), or every row where it
  // has given up
  const unsigned long long* const over = SINGLE ? O1.over : O.over;
  const bool left = FORM == TB_ONE64 && O1.rows;
  if (over) {
    wait_for_previous();
    if ((*over != 0) == left) return;
  }
  if (left) {
    m = *O1.rows;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(O1.counters, O1.counters[CNT_FS_TESTED]);
  }
  const int nsp = (nsub + TB_SUPER - 1) / TB_SUPER;     // super-stages of a tile
  const int nchunk = (nsub + TB_CHUNK - 1) / TB_CHUNK;  // image chunks
  const uint32_t ntg = (uint32_t)((m + (unsigned)(TB_TM * T) - 1) / (unsigned)(TB_TM * T));  // tile groups

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int s = 0; s < xst; ++s) {
      mbar_init(x_full + 8 * s, 1);
      mbar_init(x_empty + 8 * s, 8);  // four warps, twice
    }
    for (int s = 0; s < nb; ++s) {
      mbar_init(b_full + 8 * s, 1);
      mbar_init(b_empty + 8 * s, (uint32_t)T);  // the commits of T MMA warps
    }
    for (int t = 0; t < TB_UG; ++t) {
      mbar_init(a_full + 8 * t, 4);
      mbar_init(a_empty + 8 * t, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 4);
      mbar_init(drain + 8 * b, 1);
    }
    *s_abort = 0;
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);

  if (warp == TB_WXP) {
    // -------------------------------------------------------- row producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
      RingN xr(xst);
      uint32_t last_phase[TB_XST_MAX];
      bool issued[TB_XST_MAX];
      for (int s = 0; s < TB_XST_MAX; ++s) issued[s] = false, last_phase[s] = 0;
      bool ok = true;
      unsigned long long loads = 0;
      for (uint32_t tg = blockIdx.x; tg < ntg && ok; tg += gridDim.x)
        for (int g = 0; g < G && ok; ++g)
          for (int bx = 0; bx < nbox && ok; ++bx)
            for (int t = 0; t < T; ++t, xr.next()) {
              if (xr.used && !wait_or_abort(x_empty + 8 * xr.slot, xr.phase ^ 1u, s_abort, counters, ERR_TIMEOUT_FULL,
                                            lim)) {
                ok = false;
                break;
              }
              if (SINGLE && O1.stall_loads && loads++ == O1.stall_loads) {  // test hook: stop feeding the pipeline
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(x_full + 8 * xr.slot, xbytes);
              // rows past the last k-mer (an odd tile's partner) read as zero
              tma_load_2d(sx + xr.slot * xbytes, &tmap, bx * 128, (int)((tg * (uint32_t)T + t) * TB_TM),
                          x_full + 8 * xr.slot);
              issued[xr.slot] = true;
              last_phase[xr.slot] = xr.phase;
            }
      // no copy may still be landing when the block exits
      for (int s = 0; s < xst; ++s)
        if (issued[s]) mbar_wait(x_full + 8 * s, last_phase[s], counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp == TB_WBP) {
    // ------------------------------------------------------ image producer
    if (lane == 0) {
      RingN br(nb);
      uint32_t last_phase[TB_NB_MAX];
      bool issued[TB_NB_MAX];
      for (int s = 0; s < TB_NB_MAX; ++s) issued[s] = false, last_phase[s] = 0;
      bool ok = true;
      for (uint32_t tg = blockIdx.x; tg < ntg && ok; tg += gridDim.x)
        for (int g = 0; g < G && ok; ++g) {
          const int8_t* src = Bimg + (size_t)g * img_bytes;
          for (int c = 0; c < nchunk; ++c, br.next()) {
            if (br.used && !wait_or_abort(b_empty + 8 * br.slot, br.phase ^ 1u, s_abort, counters, ERR_TIMEOUT_FULL,
                                          lim)) {
              ok = false;
              break;
            }
            const int subs = nsub - c * TB_CHUNK < TB_CHUNK ? nsub - c * TB_CHUNK : TB_CHUNK;
            const uint32_t bytes = (uint32_t)subs * TB_KS * N;
            mbar_arrive_expect_tx(b_full + 8 * br.slot, bytes);
            bulk_g2s(sb + br.slot * BCH, src + (size_t)c * BCH, bytes, b_full + 8 * br.slot);
            issued[br.slot] = true;
            last_phase[br.slot] = br.phase;
          }
        }
      for (int s = 0; s < nb; ++s)
        if (issued[s]) mbar_wait(b_full + 8 * s, last_phase[s], counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp >= TB_WMMA) {
    // ----------------------------------------------------------------- MMA
    // Warp w issues the MMAs of tile w of every item: with two tiles from slot
    // w alone, with one from both slots in turn.
    const bool leader = elect_one();
    const uint32_t w = (uint32_t)(warp - TB_WMMA);
    bool ok = w < (uint32_t)T;
    const uint32_t d_t = tmem + w * N;
    RingN br(nb);
    uint32_t aslot = T == 2 ? w : 0u, aphase = 0;  // slots alternate over the CTA's super-stages
    uint32_t item = 0;
    for (uint32_t tg = blockIdx.x; tg < ntg && ok; tg += gridDim.x)
      for (int g = 0; g < G && ok; ++g, ++item) {
        if (item >= 1 && !__all_sync(0xffffffffu, wait_or_abort(acc_empty + 8 * w, (item - 1) & 1u, s_abort, counters,
                                                                ERR_TIMEOUT_MMA, lim))) {
          ok = false;
          break;
        }
        for (int sp = 0; sp < nsp; ++sp) {
          if (!__all_sync(0xffffffffu, wait_or_abort(a_full + 8 * aslot, aphase, s_abort, counters, ERR_TIMEOUT_MMA,
                                                     lim))) {
            ok = false;
            break;
          }
          const int here = nsub - sp * TB_SUPER < TB_SUPER ? nsub - sp * TB_SUPER : TB_SUPER;
          const uint32_t a_t = tmem + TB_A0 + aslot * 128;
#pragma unroll
          for (int h = 0; h < TB_SUPER / TB_CHUNK; ++h) {
            if (h * TB_CHUNK < here) {
              if (!__all_sync(0xffffffffu, wait_or_abort(b_full + 8 * br.slot, br.phase, s_abort, counters,
                                                         ERR_TIMEOUT_MMA, lim))) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint64_t bd = sdesc_noswz(sb + br.slot * BCH, N * 16, 128);
              const bool last = (h + 1) * TB_CHUNK >= here;
              if (leader) {
                if (here - h * TB_CHUNK >= TB_CHUNK) {
#pragma unroll
                  for (int k = 0; k < NK; ++k)
                    tc_mma_i8_ts(d_t, a_t + h * TB_CHUNK * 32 + k * 8, bd + (uint64_t)(k * BSTEP), IDESC,
                                 (sp | h | k) ? 1u : 0u);
                } else {
#pragma unroll
                  for (int k = 0; k < NK / 2; ++k)
                    tc_mma_i8_ts(d_t, a_t + h * TB_CHUNK * 32 + k * 8, bd + (uint64_t)(k * BSTEP), IDESC,
                                 (sp | h | k) ? 1u : 0u);
                }
                tc_commit(b_empty + 8 * br.slot);
                if (last) tc_commit(a_empty + 8 * aslot);
              }
              __syncwarp();
              br.next();
            }
          }
          if (!ok) break;
          if (T == 2) {
            aphase ^= 1u;  // the same slot again, a lap later
          } else if (++aslot == (uint32_t)TB_UG) {
            aslot = 0;
            aphase ^= 1u;
          }
        }
        if (!ok) break;
        if (leader) tc_commit(acc_full + 8 * w);
        __syncwarp();
      }
    // drain: wait (bounded) until every issued MMA has completed
    if (leader) {
      tc_commit(drain + 8 * w);
      mbar_wait(drain + 8 * w, 0, counters, ERR_TIMEOUT_MMA);
    }
    __syncwarp();
  } else if (warp >= TB_WUNP) {
    // -------------------------------------------------------------- unpack
    // Group grp fills every second super-stage of the CTA's sequence into its
    // own slot: with two tiles those of tile grp.  A parity wait must not be a
    // lap of its ring ahead.  Two tiles: the ring's size is even, so a tile's
    // boxes keep to their own slots and the group visits each lap of them.  One
    // tile: the MMA warp takes super-stages in order, so when this group's slot
    // is released all boxes up to four super-stages back have landed, and four
    // super-stages span at most the four boxes of the smallest ring.
    const int grp = (warp - TB_WUNP) >> 2;
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t rx = r & swz;
    const uint32_t row0 = sx + r * rb;
    const uint32_t a_t = tmem + ((uint32_t)(q * 32) << 16) + TB_A0 + grp * 128;
    uint32_t off[TB_SUPER];
#pragma unroll
    for (int c = 0; c < TB_SUPER; ++c) off[c] = (c ^ rx) << 4;
    uint32_t xslot = 0, xphase = 0, aphase = 0;
    bool used = false;
    const int nst = nsp * T, nbx = nbox * T;  // super-stages and boxes of an item
    // items of this CTA
    unsigned long long left =
        ntg > blockIdx.x ? (unsigned long long)((ntg - blockIdx.x + gridDim.x - 1) / gridDim.x) * (unsigned)G : 0ull;
    int s = 0, box = 0;
    for (int step = grp;; step = TB_UG) {
      int b1 = -box;
      for (s += step; s >= nst; s -= nst) {
        if (left) --left;
        b1 += nbx;
      }
      if (!left) break;
      const int sp = T == 2 ? s >> 1 : s, t = T == 2 ? s & 1 : 0;
      box = (sp >> 1) * T + t;
      xslot += (uint32_t)(b1 + box);
      while (xslot >= (uint32_t)xst) {
        xslot -= (uint32_t)xst;
        xphase ^= 1u;
      }
      if (!__all_sync(0xffffffffu, wait_or_abort(x_full + 8 * xslot, xphase, s_abort, counters, ERR_TIMEOUT_FULL, lim)))
        break;
      const uint32_t xrow = row0 + xslot * xbytes;
      const uint32_t half = (uint32_t)(sp & 1) << 6;
      auto slot_free = [&] {
        return !used || __all_sync(0xffffffffu, wait_or_abort(a_empty + 8 * grp, aphase ^ 1u, s_abort, counters,
                                                              ERR_TIMEOUT_MMA, lim));
      };
      const int here = nsub - sp * TB_SUPER;
      bool ok = true;
      if (here >= TB_SUPER) {
        uint32_t wd[TB_SUPER][4];
#pragma unroll
        for (int sub = 0; sub < TB_SUPER; ++sub)
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(wd[sub][0]), "=r"(wd[sub][1]), "=r"(wd[sub][2]), "=r"(wd[sub][3])
                       : "r"(xrow + (off[sub] ^ half)));
#pragma unroll
        for (int sub = 0; sub < TB_SUPER; ++sub) {
          uint32_t o[32];
          unpack_stage(wd[sub], o);
          if (sub == 0 && !slot_free()) {
            ok = false;
            break;
          }
          tc_st32(a_t + sub * 32, o);
        }
      } else {
        for (int sub = 0; sub < here; ++sub) {
          uint4 v;
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(xrow + ((uint32_t)(sub ^ rx) << 4 ^ half)));
          const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
          uint32_t o[32];
          unpack_stage(w4, o);
          if (sub == 0 && !slot_free()) {
            ok = false;
            break;
          }
          tc_st32(a_t + sub * 32, o);
        }
      }
      if (!ok) break;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(a_full + 8 * grp, lane == 0);
      // each warp arrives twice per box: once per super-stage, or twice for
      // a single one
      mbar_arrive_if(x_empty + 8 * xslot, lane == 0, (sp & 1) == 0 && sp + 1 == nsp ? 2u : 1u);
      aphase ^= 1u;
      used = true;
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    uint32_t item = 0, tested_local = 0;
    bool ok = true;
    for (uint32_t tg = blockIdx.x; tg < ntg && ok; tg += gridDim.x)
      for (int g = 0; g < G && ok; ++g, ++item)
        for (int t = 0; t < T; ++t) {
          if (!__all_sync(0xffffffffu, wait_or_abort(acc_full + 8 * t, item & 1u, s_abort, counters, ERR_TIMEOUT_MMA,
                                                     lim))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const unsigned long long local = (unsigned long long)(tg * (uint32_t)T + t) * TB_TM + r;
          const bool valid = local < m;
          const uint32_t acc = tmem + lane_base + t * N;
          if constexpr (FORM == TB_ONE64) {
            tb_single64<N>(O1, ph, acc, local, valid, tested_local);
          } else if constexpr (FORM == TB_ONE) {
            tb_single<N>(O1, ph, acc, local, valid, tested_local);
          } else {
            const unsigned long long gk = O.kmer_offset + local;
            const int shard = mp_shard(O, valid ? gk : O.kmer_offset);
            const uint32_t wt = O.weight && valid ? O.weight[gk] : 1u;  // rows this row stands for
#pragma unroll
            for (int pp = 0; pp < PPG; ++pp) {
              const int p = g * PPG + pp;
              if (p < O.n_pheno)  // warp-uniform
                tb_count(O, p, shard, mp_test<NP>(O, ph + p, acc + pp * NP, p, gk, shard, valid) ? wt : 0u);
            }
          }
          tc_fence_before();
          __syncwarp();
          mbar_arrive_if(acc_empty + 8 * t, lane == 0);
        }
    if (SINGLE) flush_tested(O1, tested_local);
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ------------------------------------------------------------------- host

// Ring sizes: as many image chunks as fit beside TB_XST_MIN row boxes, then two
// more boxes where they still fit.  False where even the smallest rings do not fit.
static bool tb_rings(int N, int rb, int& xst, int& nb) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return false;
  auto fits = [&](int x, int n) { return tb_smem(N, x, n, rb).total + 1024 <= (uint32_t)optin; };
  xst = TB_XST_MIN;
  nb = TB_NB_MAX;
  while (nb >= TB_NB_MIN && !fits(xst, nb)) --nb;
  if (nb < TB_NB_MIN) return false;
  while (xst < TB_XST_MAX && fits(xst + 2, nb)) xst += 2;  // even: see the unpack warps
  return true;
}

static int tb_box_bytes(int wpk) { return wpk * 8 < 128 ? wpk * 8 : 128; }

bool tb_supported(int N, int wpk) {
  int xst, nb;
  return N >= 16 && N <= 128 && N % 16 == 0 && wpk * 8 >= 128 && tb_rings(N, 128, xst, nb);
}

int tb_tiles(unsigned long long m, int num_sms) { return (m + TB_TM - 1) / TB_TM > (unsigned)num_sms ? 2 : 1; }

int tb_ring(int N) {
  int xst, nb;
  return tb_rings(N, 128, xst, nb) ? nb : 0;
}

int f64_limb_cols(int k, bool drop0) {
  const int used = F64_U + F64_LU * (k - (drop0 ? 1 : 0));
  return (used + 15) / 16 * 16;
}

// Samples up to which the sum of four limbs is an exact double: digits of
// magnitude 128 enter every second sample as 128 x and the others as 64 x, and
// i2d_exact takes integers below 2^51.
constexpr int F64_NMAX = 10880;
static_assert((long long)F64_NMAX / 2 * 128 * (128 + 64) * ((1ll << 24) + (1ll << 16) + (1ll << 8) + 1) < (1ll << 51),
              "limb4 sums");

bool f64_limbs_supported(int N, int n_row, int wpk) {
  int xst, nb;
  return N <= 256 && n_row <= F64_NMAX && tb_rings(N, tb_box_bytes(wpk), xst, nb);
}

cudaError_t launch_f64_image(const LaunchF64Image& L, cudaStream_t st) {
  F64Scales S{};
  for (int j = 0; j <= L.k; ++j) S.up[j] = L.up[j];
  cudaError_t e = cudaMemsetAsync(L.img, 0, (size_t)L.kpad * L.N, st);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((L.kpad + 127) / 128), (unsigned)(3 + L.k - (L.drop0 ? 1 : 0)));
  f64_image_kernel<<<grid, 128, 0, st>>>(L.V, L.vrows, L.cm, L.k, L.drop0 ? 1 : 0, L.kpad, L.N, S, L.img);
  return cudaGetLastError();
}

template <int NP, int PPG, int FORM>
static cudaError_t launch_tb_t(const LaunchTb& L, const CUtensorMap& tm, cudaStream_t st) {
  constexpr int N = NP * PPG;
  const int rb = tb_box_bytes(L.wpk);
  int xst, nb;
  if (!tb_rings(N, rb, xst, nb)) return cudaErrorInvalidValue;
  const size_t smem = tb_smem(N, xst, nb, rb).total + 1024;
  cudaError_t e =
      cudaFuncSetAttribute(tb_kernel<NP, PPG, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int T = N <= 128 ? tb_tiles(L.m, L.num_sms) : 1;
  const unsigned long long groups = (L.m + (unsigned long long)TB_TM * T - 1) / ((unsigned long long)TB_TM * T);
  const unsigned grid = (unsigned)std::min<unsigned long long>(groups, (unsigned long long)L.num_sms);
  // the 128-sample sub-stages of the image that a row reaches
  const int nsub = std::min(L.kpad / TB_KS, L.wpk / 2), nbox = (nsub * 16 + 127) / 128;
  DevOutMP O{};
  DevOut O1{};
  if (FORM == TB_MANY) O = *L.O;
  else O1 = *L.O1;
  return launch_behind((FORM == TB_MANY ? O.over : O1.over) != nullptr, tb_kernel<NP, PPG, FORM>, grid, TB_THREADS,
                       smem, st, tm, L.m, nbox, nsub, L.G, T, xst, nb, rb, L.Bimg, (unsigned long long)L.kpad * N,
                       L.ph, O, O1);
}

cudaError_t launch_tb(const LaunchTb& L, cudaStream_t st) {
  if (L.m == 0) return cudaSuccess;
  CUtensorMap tm;
  if (!mp_tmap(L.x, L.m, L.wpk, &tm)) return cudaErrorInvalidValue;
  if (L.fp64) {
#define KG_TB_CASE(NN) \
  if (L.NP == NN) return launch_tb_t<NN, 1, TB_ONE64>(L, tm, st);
    KG_TB_CASE(16)
    KG_TB_CASE(32)
    KG_TB_CASE(48)
    KG_TB_CASE(64)
    KG_TB_CASE(80)
    KG_TB_CASE(96)
    KG_TB_CASE(112)
    KG_TB_CASE(128)
    KG_TB_CASE(144)
    KG_TB_CASE(160)
    KG_TB_CASE(176)
    KG_TB_CASE(192)
    KG_TB_CASE(208)
    KG_TB_CASE(224)
    KG_TB_CASE(240)
    KG_TB_CASE(256)
#undef KG_TB_CASE
    return cudaErrorInvalidValue;
  }
  if (L.O1) {
#define KG_TB_CASE(NN) \
  if (L.NP == NN) return launch_tb_t<NN, 1, TB_ONE>(L, tm, st);
    KG_TB_CASE(16)
    KG_TB_CASE(32)
    KG_TB_CASE(48)
    KG_TB_CASE(64)
    KG_TB_CASE(80)
    KG_TB_CASE(96)
    KG_TB_CASE(112)
    KG_TB_CASE(128)
#undef KG_TB_CASE
    return cudaErrorInvalidValue;
  }
#define KG_TB_CASE(NP_, PPG_) \
  if (L.NP == NP_ && L.PPG == PPG_) return launch_tb_t<NP_, PPG_, TB_MANY>(L, tm, st);
  KG_MP_GROUPS(KG_TB_CASE)
#undef KG_TB_CASE
  return cudaErrorInvalidValue;
}

}  // namespace kg
