// kernel_fsp.cu -- the 2-D pair test (src/kgwas_2d.cpp:237-331) with the 4-bit
// screen of kernel_fs.cu: A = the AND of two packed rows, spread over 4-bit
// floats, against the phenotype's screen image.  Pairs that the screen cannot
// place below the emit cut go to the FP64 refinement list, which
// pr_refine_kernel recomputes, counts and emits; with too many of them
// (fs_open_limit) pairs_kernel evaluates every pair instead.
//
// Schedule and roles are those of kernel_pairs.cu: a tile is 128 pairs (i, j)
// sharing i, j in one 128-row j-block; the unit's boxes (its j-block and up to
// FSP_IC rows i, 1024 samples each, TMA without multicast) stay in shared memory
// for all its tiles; two MMA warps take alternate tiles.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "fs.cuh"
#include "kernels.hpp"

namespace kg {

constexpr int FSP_IC = 32;
constexpr uint32_t FSP_XBYTES = FS_TM * 128, FSP_SLOT = FSP_XBYTES + FSP_IC * 128;

__host__ __device__ constexpr int fsp_threads(int N) { return 32 * (8 + 4 * fs_nslot(N) + 3); }

struct FspSmem {
  uint32_t x, b, bars, tmem, abort, total;
};
__host__ __device__ inline FspSmem fsp_smem(int b_bytes, int xst) {
  FspSmem L;
  L.x = 0;
  L.b = (uint32_t)xst * FSP_SLOT;
  L.bars = L.b + (uint32_t)((b_bytes + 127) / 128) * 128;
  L.tmem = L.bars + 8 * (2 * FS_XST_MAX + 2 * FS_MAXSLOT + 4 + 5);
  L.abort = L.tmem + 8;
  L.total = L.abort + 8;
  return L;
}

template <int N, int LU, bool GATE>
__global__ void __launch_bounds__(fsp_threads(N), 1)
    fsp_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap itmap, int nunit, int xst,
               const __grid_constant__ PairSched S, const uint8_t* __restrict__ Bimg, int b_bytes,
               const __grid_constant__ FsPheno F, const DevOutPairs O) {
  constexpr int NSLOT = fs_nslot(N);
  constexpr int SF0 = 512 - FS_SF, A0 = SF0 - NSLOT * 128;
  static_assert(A0 >= 2 * N, "TMEM budget");
  constexpr int W_UNP = 8, W_PROD = W_UNP + 4 * NSLOT, W_MMA = W_PROD + 1;
  constexpr uint32_t BSUPER = (uint32_t)(FS_SUPER * 4 * 2 * N * 16) >> 4;  // descriptor step of a super-stage
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  const FspSmem L = fsp_smem(b_bytes, xst);
  const uint32_t sx = base + L.x, sb = base + L.b;
  const uint32_t x_full = base + L.bars, x_empty = x_full + 8 * FS_XST_MAX;
  const uint32_t a_full = x_empty + 8 * FS_XST_MAX, a_empty = a_full + 8 * FS_MAXSLOT;
  const uint32_t acc_full = a_empty + 8 * FS_MAXSLOT, acc_empty = acc_full + 16, b_full = acc_empty + 16;
  const uint32_t drain = b_full + 8, turn = drain + 16;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(gbase + L.tmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(gbase + L.abort);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int nsp = (nunit + FS_SUPER - 1) / FS_SUPER;  // super-stages of a tile = boxes of a unit

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int s = 0; s < xst; ++s) {
      mbar_init(x_full + 8 * s, 1);
      mbar_init(x_empty + 8 * s, 4 * NSLOT);  // every unpack warp, once per unit
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
    mbar_init(b_full, 1);
    *s_abort = 0;
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);
  const unsigned long long lim = wait_limit(O.wait_ns);
  if (warp < 4) fs_scales(tmem + ((uint32_t)(warp * 32) << 16) + SF0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == W_PROD) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
      mbar_arrive_expect_tx(b_full, (uint32_t)b_bytes);
      for (int off = 0; off < b_bytes; off += 32768) {
        const int len = b_bytes - off < 32768 ? b_bytes - off : 32768;
        bulk_g2s(sb + off, Bimg + off, (uint32_t)len, b_full);
      }
      RingN xr(xst);
      uint32_t last_phase[FS_XST_MAX];
      bool issued[FS_XST_MAX];
      for (int s = 0; s < FS_XST_MAX; ++s) issued[s] = false, last_phase[s] = 0;
      bool ok = true;
      for (unsigned long long u = blockIdx.x; u < S.n_units && ok; u += gridDim.x) {
        const PairUnit U = pr_unit(S, u);
        for (int bx = 0; bx < nsp; ++bx, xr.next()) {
          if (xr.used && !fs_wait(x_empty + 8 * xr.slot, xr.phase ^ 1u, s_abort, O.counters, ERR_TIMEOUT_FULL,
                                        lim)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(x_full + 8 * xr.slot, FSP_SLOT);
          tma_load_2d(sx + xr.slot * FSP_SLOT, &tmap, bx * 128, (int)(U.jb * FS_TM), x_full + 8 * xr.slot);
          tma_load_2d(sx + xr.slot * FSP_SLOT + FSP_XBYTES, &itmap, bx * 128, (int)U.i0, x_full + 8 * xr.slot);
          issued[xr.slot] = true;
          last_phase[xr.slot] = xr.phase;
        }
      }
      // no copy may still be landing when the block exits
      mbar_wait(b_full, 0, O.counters, ERR_TIMEOUT_FULL);
      for (int s = 0; s < xst; ++s)
        if (issued[s]) mbar_wait(x_full + 8 * s, last_phase[s], O.counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp >= W_MMA) {
    // ----------------------------------------------------------------- MMA
    // two warps taking alternate tiles, in the order of kernel_ts.cu
    const bool leader = elect_one();
    const uint32_t b = (uint32_t)(warp - W_MMA);
    bool ok = __all_sync(0xffffffffu, fs_wait(b_full, 0, s_abort, O.counters, ERR_TIMEOUT_FULL, lim));
    const uint64_t bdesc0 = sdesc_noswz(sb, N * 16, 128);
    const uint32_t d_t = tmem + b * N, sf = tmem + SF0;
    Ring<NSLOT> ar;
    uint32_t v = 0, t = 0;  // tiles of the CTA, of this warp
    for (unsigned long long u = blockIdx.x; u < S.n_units && ok; u += gridDim.x) {
      const PairUnit U = pr_unit(S, u);
      const uint32_t cnt = (uint32_t)(U.i1 - U.i0);
      for (uint32_t i = 0; i < cnt; ++i, ++v) {
        if ((v & 1u) != b) {  // the other warp's tile
          for (int sp = 0; sp < nsp; ++sp) ar.next();
          continue;
        }
        if (t >= 1 && !__all_sync(0xffffffffu, fs_wait(acc_empty + 8 * b, (t - 1) & 1u, s_abort, O.counters,
                                                             ERR_TIMEOUT_MMA, lim))) {
          ok = false;
          break;
        }
        if ((b || t >= 1) && !__all_sync(0xffffffffu, fs_wait(turn + 8 * b, b ? t & 1u : (t - 1) & 1u, s_abort,
                                                                    O.counters, ERR_TIMEOUT_MMA, lim))) {
          ok = false;
          break;
        }
        ++t;
        uint64_t bd = bdesc0;
        for (int sp = 0; sp < nsp; ++sp, ar.next()) {
          if (!__all_sync(0xffffffffu,
                          fs_wait(a_full + 8 * ar.slot, ar.phase, s_abort, O.counters, ERR_TIMEOUT_MMA, lim))) {
            ok = false;
            break;
          }
          mbar_arrive_if(turn + 8 * (b ^ 1u), leader && sp + 1 == nsp);
          tc_fence_after();
          const int here = nunit - sp * FS_SUPER < FS_SUPER ? nunit - sp * FS_SUPER : FS_SUPER;
          if (leader) {
            fs_mmas<N>(d_t, tmem + A0 + ar.slot * 128, bd, sf, here, sp == 0);
            tc_commit(a_empty + 8 * ar.slot);
          }
          __syncwarp();
          bd += BSUPER;
        }
        if (!ok) break;
        if (leader) tc_commit(acc_full + 8 * b);
        __syncwarp();
      }
    }
    // drain: wait (bounded) until every issued MMA has completed
    if (leader) {
      tc_commit(drain + 8 * b);
      mbar_wait(drain + 8 * b, 0, O.counters, ERR_TIMEOUT_MMA);
    }
    __syncwarp();
  } else if (warp >= W_UNP) {
    // -------------------------------------------------------------- unpack
    // group grp fills super-stages grp, grp + NSLOT, ... of the CTA's tiles
    // into its own slot
    const int grp = (warp - W_UNP) >> 2;
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t a_t = tmem + ((uint32_t)(q * 32) << 16) + A0 + grp * 128;
    RingN xr(xst);
    uint32_t aphase = 0;
    bool used = false, ok = true;
    int skip = grp;  // super-stages from here to this group's next one
    for (unsigned long long u = blockIdx.x; u < S.n_units && ok; u += gridDim.x) {
      const PairUnit U = pr_unit(S, u);
      const int cnt = (int)(U.i1 - U.i0);
      // box bx of the unit is slot slot0 + bx of the ring
      const uint32_t slot0 = xr.slot;
      for (int bx = 0; bx < nsp; ++bx, xr.next())
        if (ok && !__all_sync(0xffffffffu, fs_wait(x_full + 8 * xr.slot, xr.phase, s_abort, O.counters,
                                                         ERR_TIMEOUT_FULL, lim)))
          ok = false;
      int ii = 0, sp = skip;  // tile of the unit, super-stage of the tile
      for (; sp >= nsp; sp -= nsp) ++ii;
      while (ok && ii < cnt) {
        uint32_t slot = slot0 + (uint32_t)sp;
        if (slot >= (uint32_t)xst) slot -= (uint32_t)xst;
        const uint32_t rj = sx + slot * FSP_SLOT + r * 128, ri = sx + slot * FSP_SLOT + FSP_XBYTES + ii * 128;
        const int here = nunit - sp * FS_SUPER;
#pragma unroll
        for (int un = 0; un < FS_SUPER; ++un) {
          if (un < here) {
            uint32_t w[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              // 16 bytes of row j and, at one address for the warp, of row i
              // (a box is zero past the row's end)
              const uint32_t ch = 2 * un + h;
              uint32_t wi[4];
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(w[4 * h]), "=r"(w[4 * h + 1]), "=r"(w[4 * h + 2]), "=r"(w[4 * h + 3])
                           : "r"(rj + ((ch ^ (r & 7)) << 4)));
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(wi[0]), "=r"(wi[1]), "=r"(wi[2]), "=r"(wi[3])
                           : "r"(ri + ((ch ^ (ii & 7)) << 4)));
#pragma unroll
              for (int t = 0; t < 4; ++t) w[4 * h + t] &= wi[t];
            }
            uint32_t o[32];
            unpack_unit(w, o);
            if (un == 0 && used &&
                !__all_sync(0xffffffffu, fs_wait(a_empty + 8 * grp, aphase ^ 1u, s_abort, O.counters,
                                                       ERR_TIMEOUT_MMA, lim))) {
              ok = false;
              break;
            }
            tc_st32(a_t + un * 32, o);
          }
        }
        if (!ok) break;
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(a_full + 8 * grp, lane == 0);
        aphase ^= 1u;
        used = true;
        for (sp += NSLOT; sp >= nsp; sp -= nsp) ++ii;
      }
      if (!ok) break;
      skip = (ii - cnt) * nsp + sp;
      __syncwarp();
      if (lane == 0)
        for (int bx = 0; bx < nsp; ++bx) {
          const uint32_t slot = slot0 + bx < (uint32_t)xst ? slot0 + bx : slot0 + bx - (uint32_t)xst;
          mbar_arrive(x_empty + 8 * slot);
        }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const uint32_t e = (uint32_t)(warp >> 2);
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + e * N;
    uint32_t v = 0, jt = 0, evaluated = 0;
    bool ok = true;
    for (unsigned long long u = blockIdx.x; u < S.n_units && ok; u += gridDim.x) {
      const PairUnit U = pr_unit(S, u);
      const unsigned long long j = U.jb * FS_TM + r;
      for (unsigned long long i = U.i0; i < U.i1; ++i, ++v) {
        if ((v & 1u) != e) continue;
        if (!__all_sync(0xffffffffu, fs_wait(acc_full + 8 * e, jt & 1u, s_abort, O.counters, ERR_TIMEOUT_MMA,
                                                   lim))) {
          ok = false;
          break;
        }
        ++jt;
        tc_fence_after();
        uint32_t d[N];
        fs_load<N>(acc, d);
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(acc_empty + 8 * e, lane == 0);
        const int vd = fs_verdict<N, LU, GATE, true>(F, d, j < S.n_kmers && j > i);
        evaluated += vd == 1 ? 1u : 0u;
        if (__any_sync(0xffffffffu, vd >= 2))
          fs_push_call(O.counters, s_abort, O.cand, O.cand_cap, O.open_base, (v + 1ull) * gridDim.x * FS_TM,
                  S.n_units * S.ic * FS_TM, vd >= 2, (i << 32) | j);
      }
    }
    fs_flush(O.counters, evaluated);
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ------------------------------------------------------------------- host

// Boxes in the ring: as many as fit beside the image, at least two units'; 0
// where those do not fit.
static int fsp_ring(int N, int kpad) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  const int nsp = (kpad / FS_UNIT + FS_SUPER - 1) / FS_SUPER;
  int x = FS_XST_MAX;
  while (x > 0 && fsp_smem(kpad * N / 2, x).total + 1024 > (uint32_t)optin) --x;
  return x >= 2 * nsp ? x : 0;
}

bool fsp_supported(int N, int lu, int kpad, int wpk, unsigned long long ic) {
  return N >= 8 && N <= 112 && N % 8 == 0 && (lu == 1 || lu == 2) && ic <= FSP_IC && wpk * 8 >= 128 &&
         fsp_ring(N, kpad) > 0;
}

template <int N, int LU, bool GATE>
static cudaError_t launch_fsp_t(const LaunchFsPairs& L, const CUtensorMap& tm, const CUtensorMap& itm,
                                cudaStream_t st) {
  const int xst = fsp_ring(N, L.kpad);
  if (!xst) return cudaErrorInvalidValue;
  const int b_bytes = L.kpad * N / 2;
  const size_t smem = fsp_smem(b_bytes, xst).total + 1024;
  cudaError_t e =
      cudaFuncSetAttribute(fsp_kernel<N, LU, GATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)std::min<unsigned long long>(L.S.n_units, (unsigned long long)L.num_sms);
  fsp_kernel<N, LU, GATE><<<grid, fsp_threads(N), smem, st>>>(tm, itm, L.kpad / FS_UNIT, xst, L.S, L.Bimg, b_bytes, *L.F,
                                                              *L.O);
  return cudaGetLastError();
}

cudaError_t launch_fs_pairs(const LaunchFsPairs& L, cudaStream_t st) {
  if (L.S.n_units == 0) return cudaSuccess;
  CUtensorMap tm, itm;
  if (!mp_tmap(L.x, L.S.n_kmers, L.wpk, &tm) || !mp_tmap(L.x, L.S.n_kmers, L.wpk, &itm, FSP_IC))
    return cudaErrorInvalidValue;
#define KG_FSP_CASE(NN, LL)                                                                          \
  if (L.N == NN && L.lu == LL)                                                                       \
    return L.gate ? launch_fsp_t<NN, LL, true>(L, tm, itm, st) : launch_fsp_t<NN, LL, false>(L, tm, itm, st);
  KG_FS_SINGLE(KG_FSP_CASE)
#undef KG_FSP_CASE
  return cudaErrorInvalidValue;
}

}  // namespace kg
