// kernel_fs.cu -- 4-bit screen of the association test.
//
// Nearly every k-mer of a batch is one whose row is not emitted, and telling
// that takes few digits of its sums.  This kernel computes them against the
// structure and phenotype columns in a few e2m1 (4-bit) limbs, with a bound on
// what the limbs leave out (FsPheno, prep.cpp), and decides for every k-mer:
// not tested; tested and certainly below the emit cut (only counted); or
// undecided, which goes to the FP64 refinement list.  The refinement kernel
// evaluates the statistic (src/kgwas.cpp:44-56, 182-218) in FP64 and emits:
// every value that leaves the device is FP64, and no decision rests on a sum
// whose bound does not carry it.  Where too many tests stay undecided
// (fs_open_limit) the screen gives up: its CTAs leave by the path of a wait that
// ran out, without an error, and another kernel evaluates every test: launched
// behind it, where it ends at once otherwise, or by a second call where the rows are
// in a buffer of the context.
//
// Operands: A = the packed bits spread over 4-bit floats, 8 per 32-bit word,
// in tensor memory: of a word w, w & 0x11111111 holds its samples 4i as 0.5,
// w & 0x22222222 the samples 4i + 1 as 1, w & 0x44444444 the samples 4i + 2 as
// 2 and (w >> 1) & 0x44444444 the samples 4i + 3 as 2.  One MMA (kind::mxf4,
// K = 64) takes one of the four of 8 words, and its B scale (2, 1 or 1/2, the
// same for every column) undoes the weight: the products are x times e2m1
// values, multiples of 1/2 of at most 6, and the FP32 sums are exact.
// Five bit operations spread 32 samples, against 12 for int8, and they fill
// half the tensor memory columns; the MMA rate is twice that of kind::i8.
//
// Roles (one persistent CTA per SM): as kernel_ts.cu -- 8 epilogue warps (a
// group per accumulator), one unpack group of 4 warps per A slot, a row
// producer (2-D TMA, 128 rows x 128 bytes = 1024 samples, no multicast), two
// MMA warps taking alternate items -- and an image producer.  An item is a tile
// of 128 k-mers against one group of PPG phenotypes, whose image is resident in
// shared memory; with several groups each runs over `bt` tiles of the CTA
// before the next one's image replaces it, 1024 samples at a time.
//
// What bounds it: one phenotype, the rows' bytes (1e8 k-mers at n = 1000,
// r = 16+1: 12.8 GB at 6.5 TB/s are 1.96 ms; the kernel takes 2.2 ms); many,
// the MMAs (64 phenotypes x 4e6 at n = 2000, r = 20+1: 3.7 of 4.6 ms at 24
// columns a phenotype).  Whole calls, before (int8 limbs, kernel_ts.cu,
// kernel_tb.cu, kernel_mpb2.cu) and now: 1e8 at n = 1000 4.80 -> 2.7 ms; 1e7
// at n = 2000 1.12 -> 0.56; 2e6 at n = 5000, r = 32+1 0.99 -> 0.37; 64
// phenotypes x 4e6 at n = 2000 22.9 -> 5.4; 8 x 1e6 at n = 5000 3.38 -> 1.06.
// One limb per U column: with two (48 columns instead of 24 at n = 1000) the MMAs
// bound it (2.6 ms); the few more undecided k-mers cost 0.01 ms.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "fs.cuh"
#include "kernels.hpp"

namespace kg {

struct FsSmem {
  uint32_t x, b, bars, tmem, abort, total;
};
__host__ __device__ inline FsSmem fs_smem(int b_bytes, int xst, int rb) {
  FsSmem L;
  L.x = 0;
  L.b = (uint32_t)xst * FS_TM * rb;
  L.bars = L.b + (uint32_t)((b_bytes + 127) / 128) * 128;
  L.tmem = L.bars + 8 * (2 * FS_XST_MAX + 2 * FS_CH_MAX + 2 * FS_MAXSLOT + 4 + 4);
  L.abort = L.tmem + 8;
  L.total = L.abort + 8;
  return L;
}

// MANY: PPG phenotypes per group, G groups, outputs O; otherwise one
// phenotype, outputs O1.
template <int NP, int PPG, int LU, bool GATE, bool MANY>
__global__ void __launch_bounds__(fs_threads(NP * PPG), 1)
    fs_kernel(const __grid_constant__ CUtensorMap tmap, unsigned long long m, int nunit, int G, int bt, int xst, int rb,
              const uint8_t* __restrict__ Bimg, int b_bytes, const __grid_constant__ FsPheno F1,
              const FsPheno* __restrict__ ph, const DevOutMP O, const DevOut O1) {
  constexpr int N = NP * PPG;
  constexpr int NSLOT = fs_nslot(N);
  constexpr int SF0 = 512 - FS_SF, A0 = SF0 - NSLOT * 128;
  static_assert(A0 >= 2 * N && NP % 8 == 0, "TMEM budget");
  constexpr int W_UNP = 8, W_XP = W_UNP + 4 * NSLOT, W_BP = W_XP + 1, W_MMA = W_BP + 1;
  constexpr uint32_t BSTEP = (2 * N * 16) >> 4;                   // descriptor step of one MMA
  constexpr uint32_t BCH = (uint32_t)FS_SUPER * FS_UNIT * N / 2;  // bytes of one image chunk
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  const uint32_t xbytes = FS_TM * (uint32_t)rb, swz = rb == 128 ? 7u : 0u;  // boxes as in kernel_ts.cu
  const FsSmem L = fs_smem(b_bytes, xst, rb);
  const uint32_t sx = base + L.x, sb = base + L.b;
  const uint32_t x_full = base + L.bars, x_empty = x_full + 8 * FS_XST_MAX;
  const uint32_t b_full = x_empty + 8 * FS_XST_MAX, b_empty = b_full + 8 * FS_CH_MAX;
  const uint32_t a_full = b_empty + 8 * FS_CH_MAX, a_empty = a_full + 8 * FS_MAXSLOT;
  const uint32_t acc_full = a_empty + 8 * FS_MAXSLOT, acc_empty = acc_full + 16;
  const uint32_t drain = acc_empty + 16, turn = drain + 16;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(gbase + L.tmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(gbase + L.abort);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned long long* const counters = MANY ? O.counters : O1.counters;
  const unsigned long long lim = wait_limit(MANY ? O.wait_ns : O1.wait_ns);
  const unsigned long long stall = MANY ? O.stall_loads : O1.stall_loads;
  const int nsp = (nunit + FS_SUPER - 1) / FS_SUPER;  // super-stages of a tile
  const uint32_t ntiles = (uint32_t)((m + FS_TM - 1) / FS_TM);
  const uint32_t mine = ntiles > blockIdx.x ? (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;  // tiles of this CTA

  next_may_start();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int s = 0; s < xst; ++s) {
      mbar_init(x_full + 8 * s, 1);
      mbar_init(x_empty + 8 * s, 4);  // the warps of one unpack group
    }
    for (int s = 0; s < nsp; ++s) {
      mbar_init(b_full + 8 * s, 1);
      mbar_init(b_empty + 8 * s, 2);  // the commits of the MMA warps
    }
    for (int t = 0; t < NSLOT; ++t) {
      mbar_init(a_full + 8 * t, 4);
      mbar_init(a_empty + 8 * t, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 4);
      mbar_init(drain + 8 * b, 1);
      mbar_init(turn + 8 * b, 1);
    }
    *s_abort = 0;
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);
  if (warp < 4) {
    fs_scales(tmem + ((uint32_t)(warp * 32) << 16) + SF0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == W_XP) {
    // -------------------------------------------------------- row producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
      RingN xr(xst);
      uint32_t last_phase[FS_XST_MAX];
      bool issued[FS_XST_MAX];
      for (int s = 0; s < FS_XST_MAX; ++s) issued[s] = false, last_phase[s] = 0;
      bool ok = true;
      unsigned long long loads = 0;
      for (uint32_t i0 = 0; i0 < mine && ok; i0 += bt)
        for (int g = 0; g < G && ok; ++g)
          for (uint32_t i = i0; i < mine && i < i0 + bt && ok; ++i)
            for (int bx = 0; bx < nsp; ++bx, xr.next()) {
              if (xr.used && !fs_wait(x_empty + 8 * xr.slot, xr.phase ^ 1u, s_abort, counters, ERR_TIMEOUT_FULL,
                                            lim)) {
                ok = false;
                break;
              }
              if (stall && loads++ == stall) {  // test hook: stop feeding the pipeline
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(x_full + 8 * xr.slot, xbytes);
              tma_load_2d(sx + xr.slot * xbytes, &tmap, bx * 128, (int)((blockIdx.x + i * gridDim.x) * FS_TM),
                          x_full + 8 * xr.slot);
              issued[xr.slot] = true;
              last_phase[xr.slot] = xr.phase;
            }
      // no copy may still be landing when the block exits
      for (int s = 0; s < xst; ++s)
        if (issued[s]) mbar_wait(x_full + 8 * s, last_phase[s], counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp == W_BP) {
    // ------------------------------------------------------ image producer
    if (lane == 0) {
      uint32_t pass = 0;
      uint32_t issued = 0, last_phase = 0;  // a bit per chunk
      bool ok = true;
      for (uint32_t i0 = 0; i0 < mine && ok; i0 += bt)
        for (int g = 0; g < G && ok; ++g, ++pass) {
          const uint8_t* src = Bimg + (size_t)g * (uint32_t)b_bytes;
          for (int c = 0; c < nsp; ++c) {
            if (pass && !fs_wait(b_empty + 8 * c, (pass - 1) & 1u, s_abort, counters, ERR_TIMEOUT_FULL, lim)) {
              ok = false;
              break;
            }
            const int units = nunit - c * FS_SUPER < FS_SUPER ? nunit - c * FS_SUPER : FS_SUPER;
            const uint32_t bytes = (uint32_t)units * FS_UNIT * N / 2;
            mbar_arrive_expect_tx(b_full + 8 * c, bytes);
            bulk_g2s(sb + c * BCH, src + (size_t)c * BCH, bytes, b_full + 8 * c);
            issued |= 1u << c;
            last_phase = (last_phase & ~(1u << c)) | (pass & 1u) << c;
          }
        }
      // no copy may still be landing when the block exits
      for (int c = 0; c < nsp; ++c)
        if (issued >> c & 1u) mbar_wait(b_full + 8 * c, last_phase >> c & 1u, counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp >= W_MMA) {
    // ----------------------------------------------------------------- MMA
    // Two warps take alternate items, warp w accumulator w; see kernel_ts.cu
    // for `turn`, which keeps both in step with the ring of A slots.
    const bool leader = elect_one();
    const uint32_t b = (uint32_t)(warp - W_MMA);
    const uint64_t bdesc0 = sdesc_noswz(sb, N * 16, 128);
    const uint32_t d_t = tmem + b * N, sf = tmem + SF0;
    bool ok = true;
    Ring<NSLOT> ar;
    uint32_t item = 0, i2 = 0, pass = 0;  // items of the CTA, of this warp; passes
    for (uint32_t i0 = 0; i0 < mine && ok; i0 += bt)
      for (int g = 0; g < G && ok; ++g, ++pass) {
        const uint32_t cnt = mine - i0 < (uint32_t)bt ? mine - i0 : (uint32_t)bt;
        const uint32_t bpar = G == 1 ? 0u : pass & 1u;
        bool first = true;
        for (uint32_t i = 0; i < cnt && ok; ++i, ++item) {
          if ((item & 1u) != b) {
            for (int sp = 0; sp < nsp; ++sp) ar.next();
            continue;
          }
          const bool lastone = G > 1 && i + 2 >= cnt;  // this warp's last item of the pass
          if (i2 >= 1 && !__all_sync(0xffffffffu, fs_wait(acc_empty + 8 * b, (i2 - 1) & 1u, s_abort, counters,
                                                                ERR_TIMEOUT_MMA, lim))) {
            ok = false;
            break;
          }
          if ((b || i2 >= 1) && !__all_sync(0xffffffffu, fs_wait(turn + 8 * b, b ? i2 & 1u : (i2 - 1) & 1u,
                                                                       s_abort, counters, ERR_TIMEOUT_MMA, lim))) {
            ok = false;
            break;
          }
          uint64_t bd = bdesc0;
          for (int sp = 0; sp < nsp; ++sp, ar.next()) {
            if (first && !__all_sync(0xffffffffu, fs_wait(b_full + 8 * sp, bpar, s_abort, counters,
                                                                ERR_TIMEOUT_FULL, lim))) {
              ok = false;
              break;
            }
            if (!__all_sync(0xffffffffu, fs_wait(a_full + 8 * ar.slot, ar.phase, s_abort, counters,
                                                       ERR_TIMEOUT_MMA, lim))) {
              ok = false;
              break;
            }
            mbar_arrive_if(turn + 8 * (b ^ 1u), leader && sp + 1 == nsp);
            tc_fence_after();
            const int here = nunit - sp * FS_SUPER < FS_SUPER ? nunit - sp * FS_SUPER : FS_SUPER;
            const uint32_t a_t = tmem + A0 + ar.slot * 128;
            if (leader) {
              fs_mmas<N>(d_t, a_t, bd, sf, here, sp == 0);
              tc_commit(a_empty + 8 * ar.slot);
              if (lastone) tc_commit(b_empty + 8 * sp);
            }
            __syncwarp();
            bd += (uint64_t)(FS_SUPER * 4 * BSTEP);
          }
          if (!ok) break;
          first = false;
          if (leader) tc_commit(acc_full + 8 * b);
          __syncwarp();
          ++i2;
        }
        // a pass of one item: the other warp releases the image too
        if (ok && first && G > 1 && leader)
          for (int c = 0; c < nsp; ++c) tc_commit(b_empty + 8 * c);
        __syncwarp();
      }
    // drain: wait (bounded) until every issued MMA has completed
    if (leader) {
      tc_commit(drain + 8 * b);
      mbar_wait(drain + 8 * b, 0, counters, ERR_TIMEOUT_MMA);
    }
    __syncwarp();
  } else if (warp >= W_UNP) {
    // -------------------------------------------------------------- unpack
    // Group grp fills every NSLOT-th super-stage of the CTA's sequence into
    // its own slot.  The ring's size is a multiple of NSLOT, so that a box slot
    // belongs to one group, which sees each of its laps.
    const int grp = (warp - W_UNP) >> 2;
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t rx = r & swz;
    const uint32_t row0 = sx + r * rb;
    const uint32_t a_t = tmem + ((uint32_t)(q * 32) << 16) + A0 + grp * 128;
    const int chunks = rb >> 4;
    uint32_t xslot = (uint32_t)grp, xphase = 0, aphase = 0;
    bool used = false;
    unsigned long long left = (unsigned long long)mine * (unsigned)G;  // items from the current one on
    int sp = 0;
    for (int step = grp;; step = NSLOT) {
      for (sp += step; sp >= nsp; sp -= nsp)
        if (left) --left;
      if (!left) break;
      if (!__all_sync(0xffffffffu, fs_wait(x_full + 8 * xslot, xphase, s_abort, counters, ERR_TIMEOUT_FULL, lim)))
        break;
      const uint32_t xrow = row0 + xslot * xbytes;
      const int here = nunit - sp * FS_SUPER;
      bool ok = true;
#pragma unroll
      for (int u = 0; u < FS_SUPER; ++u) {
        if (u < here) {
          uint32_t w[8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int ch = 2 * u + h;
            if (ch < chunks)  // a short row may end in the middle of a unit
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(w[4 * h]), "=r"(w[4 * h + 1]), "=r"(w[4 * h + 2]), "=r"(w[4 * h + 3])
                           : "r"(xrow + (((uint32_t)ch ^ rx) << 4)));
            else
              w[4 * h] = w[4 * h + 1] = w[4 * h + 2] = w[4 * h + 3] = 0u;
          }
          uint32_t o[32];
          unpack_unit(w, o);
          if (u == 0 && used &&
              !__all_sync(0xffffffffu,
                          fs_wait(a_empty + 8 * grp, aphase ^ 1u, s_abort, counters, ERR_TIMEOUT_MMA, lim))) {
            ok = false;
            break;
          }
          tc_st32(a_t + u * 32, o);
        }
      }
      if (!ok) break;
      mbar_arrive_if(x_empty + 8 * xslot, lane == 0);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(a_full + 8 * grp, lane == 0);
      aphase ^= 1u;
      used = true;
      if ((xslot += NSLOT) >= (uint32_t)xst) {
        xslot -= (uint32_t)xst;
        xphase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const uint32_t e = (uint32_t)(warp >> 2);
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + e * N;
    uint32_t item = 0, jt = 0, tested_local = 0;
    bool ok = true;
    // MANY: tested counts of the group's phenotypes in the shard of k-mers
    // [s_lo, s_hi) (one atomic per item and phenotype, after a match of the
    // lanes' shards, took a quarter of the kernel's time)
    uint32_t cnt[PPG] = {};
    int shard = 0;
    unsigned long long s_lo = 1, s_hi = 0;
    auto flush = [&](int g) {
#pragma unroll
      for (int pp = 0; pp < PPG; ++pp) {
        const unsigned tot = __reduce_add_sync(0xffffffffu, cnt[pp]);
        const int p = g * PPG + pp;
        if (lane == 0 && tot && p < O.n_pheno)
          atomicAdd(O.tested + (size_t)shard * O.n_pheno + p, (unsigned long long)tot);
        cnt[pp] = 0;
      }
    };
    for (uint32_t i0 = 0; i0 < mine && ok; i0 += bt)
      for (int g = 0; g < G && ok; ++g) {
        for (uint32_t i = i0; i < mine && i < i0 + bt; ++i, ++item) {
          if ((item & 1u) != e) continue;
          if (!__all_sync(0xffffffffu, fs_wait(acc_full + 8 * e, jt & 1u, s_abort, counters, ERR_TIMEOUT_MMA,
                                                     lim))) {
            ok = false;
            break;
          }
          ++jt;
          tc_fence_after();
          const unsigned long long local = (unsigned long long)(blockIdx.x + i * gridDim.x) * FS_TM + r;
          const bool valid = local < m;
          uint32_t wt = 1u;
          uint32_t open = 0;  // two bits a phenotype: undecided, its gate included
          bool same = true;  // the warp's rows lie in one shard, whose counts stay in registers
          if (MANY) {
            const unsigned long long w0 = O.kmer_offset + local - lane, end = O.kmer_offset + m;
            if (w0 < end && !(w0 >= s_lo && w0 < s_hi)) {
              flush(g);
              shard = mp_shard(O, w0);
              s_lo = w0;
              s_hi = shard + 1 < O.n_shards ? O.shard_start[shard + 1] : ~0ull;
            }
            same = w0 + 32 <= s_hi || end <= s_hi;
            if (O.weight && valid) wt = O.weight[O.kmer_offset + local];
          }
#pragma unroll
          for (int pp = 0; pp < PPG; ++pp) {
            uint32_t d[NP];
            fs_load<NP>(acc + pp * NP, d);
            if (pp + 1 == PPG) {
              tc_fence_before();
              __syncwarp();
              mbar_arrive_if(acc_empty + 8 * e, lane == 0);
            }
            const int p = g * PPG + pp;
            if (MANY && p >= O.n_pheno) continue;  // warp-uniform
            if constexpr (MANY) {
              FsPheno F;
              fs_constants<NP, LU, GATE>(ph + p, F);
              const int v = fs_verdict<NP, LU, GATE>(F, d, valid);
              const uint32_t t = v == 1 || v == 2 ? wt : 0u;
              if (same) cnt[pp] += t;
              else tb_count(O, p, mp_shard(O, valid ? O.kmer_offset + local : O.kmer_offset), t);
              open |= v >= 2 ? (unsigned)(v - 1) << (2 * pp) : 0u;
            } else {
              const int v = fs_verdict<NP, LU, GATE>(F1, d, valid);
              if (v == 1 || (v == 2 && !O1.count_sure))
                tested_local += O1.weight ? O1.weight[O1.kmer_offset + local] : 1u;
              if (__any_sync(0xffffffffu, v >= 2))
                fs_push_call(counters, s_abort, O1.cand, O1.cand_cap, O1.open_base,
                             (item + 1ull) * gridDim.x * FS_TM, m, v >= 2,
                             (O1.kmer_offset + local) | (v == 3 && !O1.count_sure ? CAND_OPEN : 0ull));
            }
          }
          // one copy of the push behind the PPG verdicts, not one in each (64 phenotypes
          // at n = 2000: 4.67 -> 4.55 ms)
          if (MANY && __any_sync(0xffffffffu, open != 0u)) {
#pragma unroll 1
            for (int pp = 0; pp < PPG; ++pp) {
              const uint32_t v = open >> (2 * pp) & 3u;
              if (__any_sync(0xffffffffu, v != 0u))
                fs_push(counters, s_abort, O.cand, O.cand_cap, O.open_base, (item + 1ull) * gridDim.x * (FS_TM * PPG),
                        m * (unsigned)O.n_pheno, v != 0u,
                        (O.kmer_offset + local) | ((unsigned long long)(g * PPG + pp) << 48) |
                            (v == 2u ? CAND_OPEN_MP : 0ull));
            }
          }
        }
        if (MANY) flush(g);
      }
    if (!MANY) fs_flush(counters, tested_local);
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Copies the rows of the screen's candidates to dst, 16 bytes a
// thread; none where it has given up.
__global__ void __launch_bounds__(256) fs_gather_kernel(const uint4* __restrict__ x, int chunks,
                                                        const unsigned long long* __restrict__ cand,
                                                        const unsigned long long* __restrict__ counters,
                                                        unsigned long long offset, uint4* __restrict__ dst) {
  if (counters[CNT_FS_OVER]) return;
  const unsigned long long rows = counters[CNT_FS_OPEN];
  const unsigned long long total = rows * (unsigned)chunks;
  for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = t / (unsigned)chunks;
    dst[t] = x[(cand[r] - offset) * (unsigned)chunks + (t - r * (unsigned)chunks)];
  }
}

// ------------------------------------------------------------------- host

cudaError_t launch_fs_gather(const uint64_t* x, int wpk, const unsigned long long* cand,
                             const unsigned long long* counters, unsigned long long offset, uint64_t* dst, int num_sms,
                             cudaStream_t st) {
  fs_gather_kernel<<<2 * num_sms, 256, 0, st>>>(reinterpret_cast<const uint4*>(x), wpk / 2, cand, counters, offset,
                                                reinterpret_cast<uint4*>(dst));
  return cudaGetLastError();
}

static int fs_box_bytes(int wpk) { return wpk * 8 < 128 ? wpk * 8 : 128; }

// Row boxes that fit beside the image: a multiple of the A slots (see the
// unpack warps); 0 where fewer than two per slot fit.
static int fs_ring(int N, int kpad, int rb) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  const int ns = fs_nslot(N);
  int x = FS_XST_MAX / ns * ns;
  while (x > 0 && fs_smem(kpad * N / 2, x, rb).total + 1024 > (uint32_t)optin) x -= ns;
  return x >= 2 * ns ? x : 0;
}

bool fs_supported(int N, int kpad, int wpk) {
  return N >= 8 && N <= 112 && N % 8 == 0 && kpad <= FS_CH_MAX * FS_SUPER * FS_UNIT &&
         fs_ring(N, kpad, fs_box_bytes(wpk)) > 0;
}

template <int NP, int PPG, int LU, bool GATE, bool MANY>
static cudaError_t launch_fs_t(const LaunchFs& L, const CUtensorMap& tm, cudaStream_t st) {
  constexpr int N = NP * PPG;
  const int rb = fs_box_bytes(L.wpk);
  const int xst = fs_ring(N, L.kpad, rb);
  if (!xst) return cudaErrorInvalidValue;
  const int b_bytes = L.kpad * N / 2;
  const size_t smem = fs_smem(b_bytes, xst, rb).total + 1024;
  cudaError_t e = cudaFuncSetAttribute(fs_kernel<NP, PPG, LU, GATE, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned long long tiles = (L.m + FS_TM - 1) / FS_TM;
  const unsigned grid = (unsigned)std::min<unsigned long long>(tiles, (unsigned long long)L.num_sms);
  DevOutMP O{};
  DevOut O1{};
  if (MANY) O = *L.O;
  else O1 = *L.O1;
  const int bt = L.G == 1 ? 1 << 30 : L.bt;
  fs_kernel<NP, PPG, LU, GATE, MANY><<<grid, fs_threads(N), smem, st>>>(tm, L.m, L.kpad / FS_UNIT, L.G, bt, xst, rb,
                                                                      L.Bimg, b_bytes, MANY ? FsPheno() : *L.F1, L.ph, O, O1);
  return cudaGetLastError();
}

cudaError_t launch_fs(const LaunchFs& L, cudaStream_t st) {
  if (L.m == 0) return cudaSuccess;
  CUtensorMap tm;
  if (!mp_tmap(L.x, L.m, L.wpk, &tm)) return cudaErrorInvalidValue;
  if (L.O1) {
#define KG_FS_CASE(NN, LL)     \
  if (L.NP == NN && L.lu == LL) \
    return L.gate ? launch_fs_t<NN, 1, LL, true, false>(L, tm, st) : launch_fs_t<NN, 1, LL, false, false>(L, tm, st);
    KG_FS_SINGLE(KG_FS_CASE)
#undef KG_FS_CASE
    return cudaErrorInvalidValue;
  }
#define KG_FS_CASE(NP_, PPG_)                                                              \
  if (L.NP == NP_ && L.PPG == PPG_ && L.lu == 1)                                           \
    return L.gate ? launch_fs_t<NP_, PPG_, 1, true, true>(L, tm, st) : launch_fs_t<NP_, PPG_, 1, false, true>(L, tm, st);
  KG_FS_GROUPS(KG_FS_CASE)
#undef KG_FS_CASE
  return cudaErrorInvalidValue;
}

}  // namespace kg
