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
constexpr int TB_CHUNK = 2;    // sub-stages per image chunk
constexpr int TB_UG = 2;       // unpack groups = A slots of 128 TMEM columns
constexpr uint32_t TB_XBYTES = TB_TM * 128;
constexpr int TB_XST_MAX = 6, TB_XST_MIN = 4, TB_NB_MAX = 8, TB_NB_MIN = 3;
constexpr int TB_WUNP = 4, TB_WXP = TB_WUNP + 4 * TB_UG, TB_WBP = TB_WXP + 1, TB_WMMA = TB_WBP + 1;
constexpr int TB_THREADS = 32 * (TB_WMMA + 2);
constexpr int TB_A0 = 512 - TB_UG * 128;

struct TbSmem {
  uint32_t x, b, bars, tmem, abort, total;
};
__host__ __device__ inline TbSmem tb_smem(int N, int xst, int nb) {
  TbSmem L;
  L.x = 0;
  L.b = (uint32_t)xst * TB_XBYTES;
  L.bars = L.b + (uint32_t)nb * TB_CHUNK * TB_KS * N;
  L.tmem = L.bars + 8 * (2 * TB_XST_MAX + 2 * TB_NB_MAX + 2 * TB_UG + 4 + 2);
  L.abort = L.tmem + 8;
  L.total = L.abort + 8;
  return L;
}

// Adds the lanes' counts of phenotype p to their (shard, phenotype) counters:
// one atomic per distinct shard in the warp.
__device__ __forceinline__ void tb_count(const DevOutMP& O, int p, int shard, uint32_t cnt) {
  const unsigned match = __match_any_sync(0xffffffffu, shard);
  const unsigned tot = __reduce_add_sync(match, cnt);
  if ((int)(threadIdx.x & 31u) == __ffs(match) - 1 && tot)
    atomicAdd(O.tested + (size_t)shard * O.n_pheno + p, (unsigned long long)tot);
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

// SINGLE: one phenotype (G = 1), results to O1; otherwise to O.
template <int NP, int PPG, bool SINGLE>
__global__ void __launch_bounds__(TB_THREADS, 1)
    tb_kernel(const __grid_constant__ CUtensorMap tmap, unsigned long long m, int nbox, int nsub, int G, int T,
              int xst, int nb, const int8_t* __restrict__ Bimg, unsigned long long img_bytes,
              const MPheno* __restrict__ ph, const DevOutMP O, const DevOut O1) {
  constexpr int N = NP * PPG;
  static_assert(N <= 128 && N % 16 == 0, "group width");
  constexpr uint32_t IDESC = idesc_i8(TB_TM, N);
  constexpr uint32_t BSTEP = (2 * N * 16) >> 4;             // descriptor step of one K = 32 MMA
  constexpr uint32_t BCH = (uint32_t)TB_CHUNK * TB_KS * N;  // bytes of one image chunk
  constexpr int NK = TB_CHUNK * (TB_KS / 32);               // MMAs per chunk
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  const TbSmem L = tb_smem(N, xst, nb);
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
              mbar_arrive_expect_tx(x_full + 8 * xr.slot, TB_XBYTES);
              // rows past the last k-mer (an odd tile's partner) read as zero
              tma_load_2d(sx + xr.slot * TB_XBYTES, &tmap, bx * 128, (int)((tg * (uint32_t)T + t) * TB_TM),
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
    const uint32_t rx = r & 7;
    const uint32_t row0 = sx + r * 128;
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
      const uint32_t xrow = row0 + xslot * TB_XBYTES;
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
          if (SINGLE) {
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
static bool tb_rings(int N, int& xst, int& nb) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return false;
  auto fits = [&](int x, int n) { return tb_smem(N, x, n).total + 1024 <= (uint32_t)optin; };
  xst = TB_XST_MIN;
  nb = TB_NB_MAX;
  while (nb >= TB_NB_MIN && !fits(xst, nb)) --nb;
  if (nb < TB_NB_MIN) return false;
  while (xst < TB_XST_MAX && fits(xst + 2, nb)) xst += 2;  // even: see the unpack warps
  return true;
}

bool tb_supported(int N, int wpk) {
  int xst, nb;
  return N >= 16 && N <= 128 && N % 16 == 0 && wpk * 8 >= 128 && tb_rings(N, xst, nb);
}

int tb_tiles(unsigned long long m, int num_sms) { return (m + TB_TM - 1) / TB_TM > (unsigned)num_sms ? 2 : 1; }

int tb_ring(int N) {
  int xst, nb;
  return tb_rings(N, xst, nb) ? nb : 0;
}

template <int NP, int PPG, bool SINGLE>
static cudaError_t launch_tb_t(const LaunchTb& L, const CUtensorMap& tm, cudaStream_t st) {
  constexpr int N = NP * PPG;
  int xst, nb;
  if (!tb_rings(N, xst, nb)) return cudaErrorInvalidValue;
  const size_t smem = tb_smem(N, xst, nb).total + 1024;
  cudaError_t e =
      cudaFuncSetAttribute(tb_kernel<NP, PPG, SINGLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int T = tb_tiles(L.m, L.num_sms);
  const unsigned long long groups = (L.m + (unsigned long long)TB_TM * T - 1) / ((unsigned long long)TB_TM * T);
  const unsigned grid = (unsigned)std::min<unsigned long long>(groups, (unsigned long long)L.num_sms);
  // the 128-sample sub-stages of the image that a row reaches
  const int nsub = std::min(L.kpad / TB_KS, L.wpk / 2), nbox = (nsub * 16 + 127) / 128;
  DevOutMP O{};
  DevOut O1{};
  if (SINGLE) O1 = *L.O1;
  else O = *L.O;
  tb_kernel<NP, PPG, SINGLE><<<grid, TB_THREADS, smem, st>>>(tm, L.m, nbox, nsub, L.G, T, xst, nb, L.Bimg,
                                                             (unsigned long long)L.kpad * N, L.ph, O, O1);
  return cudaGetLastError();
}

cudaError_t launch_tb(const LaunchTb& L, cudaStream_t st) {
  if (L.m == 0) return cudaSuccess;
  CUtensorMap tm;
  if (!mp_tmap(L.x, L.m, L.wpk, &tm)) return cudaErrorInvalidValue;
  if (L.O1) {
#define KG_TB_CASE(NN) \
  if (L.NP == NN) return launch_tb_t<NN, 1, true>(L, tm, st);
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
  if (L.NP == NP_ && L.PPG == PPG_) return launch_tb_t<NP_, PPG_, false>(L, tm, st);
  KG_MP_GROUPS(KG_TB_CASE)
#undef KG_TB_CASE
  return cudaErrorInvalidValue;
}

}  // namespace kg
