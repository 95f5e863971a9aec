// kernel_ts.cu -- split-precision association kernel with the unpacked x
// operand held in tensor memory.
//
// One persistent CTA per SM, warp-specialised (736 threads; 608 for N = 80,
// 480 above):
//   epilogue  8 warps, two groups of four (one warp per TMEM lane quarter),
//             group e owning accumulator buffer e, i.e. every other tile:
//             tcgen05.ld of the int32 accumulators (one TMEM lane = one
//             k-mer), then the single-precision screen (screen_kmer), and for
//             warps holding a k-mer that it cannot decide the exact limb
//             recombination and FP64 statistic; warp-aggregated hits;
//   unpack    groups of four warps, one per TMEM A slot (one group for
//             N > 80, so that the epilogue keeps its registers), taking
//             super-stages in turn: read 128 samples of a packed row from the
//             TMA-filled shared tile and write them as int8 (0 / -128, or
//             0 / 64 against -2x the B digits) straight into the slot with
//             tcgen05.st -- the unpacked operand never touches shared memory;
//   producer  one warp: one 2-D TMA load (128 rows x 128 bytes, 128-byte
//             swizzle, no multicast; whole rows where they are shorter) per
//             1024 samples of a 128-k-mer tile;
//   MMA       two warps taking alternate tiles: tcgen05.mma kind::i8, A from
//             TMEM, B (the int8 limbs of the centred structure and phenotype
//             columns, resident in shared memory for the whole launch) from a
//             smem descriptor.
// Tile = 128 k-mers (M), N = 16..128 limb columns.
//
// A kind::i8 M=128 N=64 K=32 MMA occupies the tensor pipe 32 cycles (16384
// int8 ops per SM cycle), and every barrier test, commit or runtime division
// between MMAs adds its latency on top.  So the A operand moves in
// super-stages of 512 samples (4 sub-stages of 128 samples = 128 TMEM columns
// = 16 MMAs) with one barrier wait and one commit each.
// TMEM (512 columns): two accumulators of N columns, then NSLOT super-slots.
//
// What bounds it (n = 1000, r = 16+1, N = 64; ncu and copies with a role's work
// left out): 11.8 SM-cycles per k-mer against 8 of MMAs; the tensor pipe is
// 74 % active, the ALU pipe of the unpack's masks (2 cycles per warp
// instruction) 60 %, instruction issue 67 %; 11.0 without the epilogue's
// arithmetic, 8.3 with the unpack alone.  4e7 k-mers take 1.62 ms.  Before
// (2.19 ms): the FP64 statistic of every k-mer in the epilogue, whose FP64
// instructions share a pipe with the MMAs (3100 cycles per tile; with the
// screen 2.06 ms); one MMA warp, 400 of its 1850 cycles per tile in barrier
// tests that the pipe's queue of six MMAs does not cover (two: 1.93 ms); every
// k-mer of chi-square 12 and up refined (1.67 ms); unpack groups that visited
// every box and took super-stages in a 64-bit loop (1.62 ms).
//
// The accumulators hold -128 * sum_i x_i * digit_l(i) for every limb l; the
// epilogue recombines the limbs exactly in int64, scales by 2^-s / 128, and
// evaluates the reference's statistic (src/kgwas.cpp:44-56, 182-218) in FP64,
// for the k-mers that the screen leaves.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "device.cuh"
#include "kernels.hpp"

namespace kg {

constexpr int TS_TM = 128;
constexpr int TS_KS = 128;         // samples per sub-stage (32 TMEM columns, 4 MMAs)
constexpr int TS_SUPER = 4;        // sub-stages per super-stage (one barrier, one commit)
constexpr int TS_BOX = 1024;       // samples per TMA box (128 bytes)
// Packed boxes in flight: as many as the shared memory left by the B image
// holds, up to TS_XST_MAX (chosen at launch).  HBM latency under this load is
// ~2 us, so 4 boxes (64 KB per SM) cap the row stream near 4.3 TB/s.
constexpr int TS_XST_MAX = 12;
constexpr int TS_MAXSLOT = 3;
// Super-slots of 128 TMEM columns left after the two N-column accumulators.
__host__ __device__ constexpr int ts_nslot(int N) {
  return (512 - 2 * N) / 128 > TS_MAXSLOT ? TS_MAXSLOT : (512 - 2 * N) / 128;
}
// Unpack groups, taking super-stages in turn: one per slot, so that a group
// always fills the same slot and waits for every release of it; one for wide
// N, so that the epilogue keeps its registers.
__host__ __device__ constexpr int ts_ug(int N) { return N <= 80 ? ts_nslot(N) : 1; }
__host__ __device__ constexpr int ts_threads(int N) { return 32 * (8 + 4 * ts_ug(N) + 3); }
constexpr int TS_LU = 3, TS_LY = 5;
constexpr int TS_WARP_UNPACK0 = 8;  // then the unpack groups, the producer, two MMA warps

struct TsSmem {  // offsets from the 1024-aligned base
  uint32_t x, b, bars, tmem, abort, total;
};
__host__ __device__ inline TsSmem ts_smem(int b_bytes, int xst, int rb) {
  TsSmem L;
  L.x = 0;
  L.b = xst * TS_TM * rb;
  L.bars = L.b + ((b_bytes + 127) / 128) * 128;
  L.tmem = L.bars + 8 * (2 * TS_XST_MAX + 2 * TS_MAXSLOT + 4 + 5);
  L.abort = L.tmem + 8;
  L.total = L.abort + 8;
  return L;
}

template <int N, bool DROP0, bool GATE, bool WIDE>
__global__ void __launch_bounds__(ts_threads(N), 1)
    ts_kernel(const __grid_constant__ CUtensorMap tmap, unsigned long long m, int nbox, int nsub, int xst,
              int ug, int row_bytes, const int8_t* __restrict__ Bimg, int b_bytes, const __grid_constant__ EpiParams P,
              const __grid_constant__ LimbMap LM, const DevOut O) {
  constexpr int UG = ts_ug(N);
  constexpr int TS_WARP_PROD = TS_WARP_UNPACK0 + 4 * UG, TS_WARP_MMA = TS_WARP_PROD + 1;
  constexpr int NSLOT = ts_nslot(N);
  constexpr int A0 = 512 - NSLOT * 128;  // first A column (>= 2N)
  static_assert(NSLOT >= 2 && A0 >= 2 * N, "TMEM budget");
  constexpr uint32_t IDESC = idesc_i8(TS_TM, N);
  constexpr int KU_MAX = (N - 1 - TS_LY) / TS_LU;  // U columns that fit in N
  constexpr uint32_t BSTEP = (2 * N * 16) >> 4;    // descriptor step of one K=32 MMA
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  // WIDE: boxes of 128 swizzled bytes per row; otherwise a box holds whole
  // rows of row_bytes < 128 (a run-time width would cost the wide case 1 %)
  const int rb = WIDE ? 128 : row_bytes;
  constexpr uint32_t swz = WIDE ? 7u : 0u;
  const uint32_t xbytes = TS_TM * (uint32_t)rb;  // one box: 128 rows
  const TsSmem L = ts_smem(b_bytes, xst, rb);
  const uint32_t sx = base + L.x, sb = base + L.b;
  const uint32_t x_full = base + L.bars, x_empty = x_full + 8 * TS_XST_MAX;
  const uint32_t a_full = x_empty + 8 * TS_XST_MAX, a_empty = a_full + 8 * TS_MAXSLOT;
  const uint32_t acc_full = a_empty + 8 * TS_MAXSLOT, acc_empty = acc_full + 16, b_full = acc_empty + 16;
  const uint32_t drain = b_full + 8, turn = drain + 16;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(gbase + L.tmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(gbase + L.abort);
  // warp-uniform values as such: the roles' loops then run on the uniform datapath
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int nsp = (nsub + TS_SUPER - 1) / TS_SUPER;  // super-stages per tile

  if (O.over) {
    wait_for_previous();
    if (!*O.over) return;  // the screen has decided
  }
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
    for (int t = 0; t < NSLOT; ++t) {
      mbar_init(a_full + 8 * t, 4);   // the four warps of one unpack group
      mbar_init(a_empty + 8 * t, 1);  // tcgen05.commit
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 4);  // the four warps of epilogue group b
    }
    mbar_init(b_full, 1);
    for (int b = 0; b < 2; ++b) {
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
  const unsigned long long ntiles = (m + TS_TM - 1) / TS_TM;
  const unsigned long long lim = wait_limit(O.wait_ns);

  if (warp == TS_WARP_PROD) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
      mbar_arrive_expect_tx(b_full, (uint32_t)b_bytes);
      for (int off = 0; off < b_bytes; off += 32768) {
        const int len = b_bytes - off < 32768 ? b_bytes - off : 32768;
        bulk_g2s(sb + off, Bimg + off, (uint32_t)len, b_full);
      }
      RingN xr(xst);
      uint32_t last_phase[TS_XST_MAX];
      bool issued[TS_XST_MAX];
      for (int s = 0; s < TS_XST_MAX; ++s) issued[s] = false, last_phase[s] = 0;
      bool ok = true;
      unsigned long long loads = 0;
      for (unsigned long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        for (int bx = 0; bx < nbox; ++bx, xr.next()) {
          if (xr.used && !wait_or_abort(x_empty + 8 * xr.slot, xr.phase ^ 1u, s_abort, O.counters, ERR_TIMEOUT_FULL, lim)) {
            ok = false;
            break;
          }
          if (O.stall_loads && loads++ == O.stall_loads) {  // test hook: stop feeding the pipeline
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(x_full + 8 * xr.slot, xbytes);
          tma_load_2d(sx + xr.slot * xbytes, &tmap, bx * 128, (int)(tile * TS_TM), x_full + 8 * xr.slot);
          issued[xr.slot] = true;
          last_phase[xr.slot] = xr.phase;
        }
      }
      // no copy may still be landing when the block exits
      mbar_wait(b_full, 0, O.counters, ERR_TIMEOUT_FULL);
      for (int s = 0; s < xst; ++s)
        if (issued[s]) mbar_wait(x_full + 8 * s, last_phase[s], O.counters, ERR_TIMEOUT_FULL);
    }
  } else if (warp >= TS_WARP_MMA) {
    // ----------------------------------------------------------------- MMA
    // Two warps take alternate tiles, warp w accumulator w: an issuing thread
    // spends 20-30 cycles per MMA and ~100 per barrier test, which the other
    // warp's MMAs cover.  Each whole warp runs its loop (warp-uniform control
    // flow and operands); one elected lane issues the MMAs and the commits
    // that track them.  The super-stages' barriers are waited for in order
    // across both warps (a warp passes `turn` on once it has seen its tile's
    // last super-stage full): a parity wait is only sound for a waiter that
    // is less than a lap of the ring ahead.
    const bool leader = elect_one();
    const uint32_t b = (uint32_t)(warp - TS_WARP_MMA);
    bool ok = __all_sync(0xffffffffu, wait_or_abort(b_full, 0, s_abort, O.counters, ERR_TIMEOUT_FULL, lim));
    const uint64_t bdesc0 = sdesc_noswz(sb, N * 16, 128);
    const uint32_t d_t = tmem + b * N;
    Ring<NSLOT> ar;
    if (b)
      for (int sp = 0; sp < nsp; ++sp) ar.next();  // the first tile is the other warp's
    uint32_t i = 0;  // tiles of this warp
    for (unsigned long long tile = blockIdx.x + (unsigned long long)b * gridDim.x; tile < ntiles && ok;
         tile += 2ull * gridDim.x, ++i) {
      if (i >= 1 && !__all_sync(0xffffffffu, wait_or_abort(acc_empty + 8 * b, (i - 1) & 1u, s_abort, O.counters,
                                                           ERR_TIMEOUT_MMA, lim))) {
        ok = false;
        break;
      }
      if ((b || i >= 1) && !__all_sync(0xffffffffu, wait_or_abort(turn + 8 * b, b ? i & 1u : (i - 1) & 1u, s_abort,
                                                                  O.counters, ERR_TIMEOUT_MMA, lim))) {
        ok = false;
        break;
      }
      uint64_t bd = bdesc0;
      for (int sp = 0; sp < nsp; ++sp, ar.next()) {
        if (!__all_sync(0xffffffffu, wait_or_abort(a_full + 8 * ar.slot, ar.phase, s_abort, O.counters, ERR_TIMEOUT_MMA, lim))) {
          ok = false;
          break;
        }
        mbar_arrive_if(turn + 8 * (b ^ 1u), leader && sp + 1 == nsp);
        tc_fence_after();
        const int nsub_here = nsub - sp * TS_SUPER < TS_SUPER ? nsub - sp * TS_SUPER : TS_SUPER;
        const uint32_t a_t = tmem + A0 + ar.slot * 128;
        if (leader) {
          if (nsub_here == TS_SUPER) {
            // full super-stage: 16 MMAs with compile-time operand offsets
#pragma unroll
            for (int k = 0; k < TS_SUPER * (TS_KS / 32); ++k)
              tc_mma_i8_ts(d_t, a_t + k * 8, bd + (uint64_t)(k * BSTEP), IDESC, (sp | k) ? 1u : 0u);
          } else {
            uint64_t bk = bd;
            for (int sub = 0; sub < nsub_here; ++sub) {
#pragma unroll
              for (int ks = 0; ks < TS_KS / 32; ++ks) {
                tc_mma_i8_ts(d_t, a_t + sub * 32 + ks * 8, bk, IDESC, (sp | sub | ks) ? 1u : 0u);
                bk += BSTEP;
              }
            }
          }
          tc_commit(a_empty + 8 * ar.slot);
        }
        __syncwarp();
        bd += (uint64_t)(TS_SUPER * (TS_KS / 32) * BSTEP);
      }
      if (!ok) break;
      if (leader) tc_commit(acc_full + 8 * b);
      __syncwarp();
      for (int sp = 0; sp < nsp; ++sp) ar.next();  // the other warp's tile
    }
    // drain: wait (bounded) until every issued MMA has completed
    if (leader) {
      tc_commit(drain + 8 * b);
      mbar_wait(drain + 8 * b, 0, O.counters, ERR_TIMEOUT_MMA);
    }
    __syncwarp();
  } else if (warp >= TS_WARP_UNPACK0) {
    // -------------------------------------------------------------- unpack
    // Group grp fills super-stages grp, grp + ug, ... of the CTA's stream of
    // tiles (ug: ts_groups).  A box holds two super-stages (the last of a tile
    // may hold one).
    const int grp = (warp - TS_WARP_UNPACK0) >> 2;
    const int q = warp & 3;      // TMEM lane quarter
    const int r = q * 32 + lane;  // row of the tile = TMEM lane
    const uint32_t rx = r & swz;
    const uint32_t row0 = sx + r * rb;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const uint32_t xst_u = (uint32_t)xst;
    uint32_t xslot = 0, xphase = 0;  // the box of this group's super-stage
    Ring<NSLOT> ar;
    for (int g = 0; g < grp; ++g) ar.next();
    uint32_t off[TS_SUPER];  // 16-byte chunks 0-3 of the row, swizzled
#pragma unroll
    for (int c = 0; c < TS_SUPER; ++c) off[c] = (c ^ rx) << 4;
    const uint32_t nt32 = (uint32_t)ntiles;  // row indices fit 31 bits (TMA coordinates)
    uint32_t tile = blockIdx.x;
    int sp = 0;  // super-stage of the tile
    for (int step = grp; grp < ug; step = ug) {
      // on to this group's next super-stage, `step` further
      int nb = -(sp >> 1);  // boxes passed over
      for (sp += step; sp >= nsp; sp -= nsp) {
        tile += gridDim.x;
        nb += nbox;
      }
      if (tile >= nt32) break;
      xslot += (uint32_t)(nb + (sp >> 1));
      if (xslot >= xst_u) {
        xslot -= xst_u;
        xphase ^= 1u;
      }
      if (!__all_sync(0xffffffffu, wait_or_abort(x_full + 8 * xslot, xphase, s_abort, O.counters, ERR_TIMEOUT_FULL,
                                                 lim)))
        break;
      const uint32_t xrow = row0 + xslot * xbytes;
      const uint32_t a_t = tmem + lane_base + A0 + ar.slot * 128;
      const uint32_t half = (uint32_t)(sp & 1) << 6;  // chunks 4-7 of the box: chunk ^ 4
      // 16 bytes (128 samples) of row r per sub-stage; 128-byte swizzle:
      // chunk c of row r sits at c ^ (r % 8).  Column 8qq+jj of a stage =
      // word qq shifted left by 2*(jj/2), masked to bit 7 (jj even: byte t
      // holds sample 8t+7-jj as 0 / -128) or bit 6 (jj odd: 0 / 64; the B
      // image holds -2 V there), so one shift serves two columns.  The
      // shift is a multiply so that it issues on the FMA pipe and the
      // masks on the ALU pipe.
      // The slot is waited for once the first sub-stage is unpacked.
      auto slot_free = [&] {
        return !ar.used || __all_sync(0xffffffffu, wait_or_abort(a_empty + 8 * ar.slot, ar.phase ^ 1u, s_abort,
                                                                 O.counters, ERR_TIMEOUT_MMA, lim));
      };
      const int nsub_here = nsub - sp * TS_SUPER;
      bool ok = true;
      if (nsub_here >= TS_SUPER) {
        uint32_t w[TS_SUPER][4];
#pragma unroll
        for (int sub = 0; sub < TS_SUPER; ++sub)
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(w[sub][0]), "=r"(w[sub][1]), "=r"(w[sub][2]), "=r"(w[sub][3])
                       : "r"(xrow + (WIDE ? off[sub] ^ half : off[sub] + half)));
#pragma unroll
        for (int sub = 0; sub < TS_SUPER; ++sub) {
          uint32_t o[32];
          unpack_stage(w[sub], o);
          if (sub == 0 && !slot_free()) {
            ok = false;
            break;
          }
          tc_st32(a_t + sub * 32, o);
        }
      } else {
        for (int sub = 0; sub < nsub_here; ++sub) {
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
      mbar_arrive_if(a_full + 8 * ar.slot, lane == 0);
      // each warp arrives twice per box: once per super-stage, or twice for
      // a single one
      mbar_arrive_if(x_empty + 8 * xslot, lane == 0, (sp & 1) == 0 && sp + 1 == nsp ? 2u : 1u);
      if (ug == NSLOT) {  // the same slot again, a lap later
        ar.phase ^= 1u;
        ar.used = 1;
      } else {
        ar.next();
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int e = warp >> 2;  // group = accumulator buffer
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const int ku = P.k - (DROP0 ? 1 : 0);  // U columns with limbs
    uint32_t jt = 0;            // tiles taken by this group
    uint32_t tested_local = 0;  // k-mers this thread tested (lean path)
    for (unsigned long long tile = blockIdx.x + (unsigned long long)e * gridDim.x; tile < ntiles;
         tile += 2ull * gridDim.x, ++jt) {
      if (!__all_sync(0xffffffffu, wait_or_abort(acc_full + 8 * e, jt & 1u, s_abort, O.counters, ERR_TIMEOUT_MMA, lim))) break;
      tc_fence_after();
      // all N columns in flight at once, then one wait
      uint32_t d[N];
#pragma unroll
      for (int c16 = 0; c16 < N / 16; ++c16) tc_ld16p(tmem + lane_base + e * N + c16 * 16, d + c16 * 16);
      tc_wait_ld();
#pragma unroll
      for (int c16 = 0; c16 < N / 16; ++c16) reg_fence16(d + c16 * 16);
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(acc_empty + 8 * e, lane == 0);
      const unsigned long long local = tile * TS_TM + r;
      const bool valid = local < m;
      if (DROP0 && P.S.on && !O.tested) {
        const int v = screen_kmer<KU_MAX, 5, GATE, false>(P.S, P.n, d, ku, valid);
        if (!__any_sync(0xffffffffu, v == 2)) {
          if (v) tested_local += O.weight ? O.weight[O.kmer_offset + local] : 1u;
          continue;
        }
      }
      // accumulators hold -128 * (integer limb sums).  The limbs are
      // recombined exactly in int64 and turned into doubles with the
      // bias trick (integer add + one FMA, no conversion instructions):
      //   U column: V = sum_l 256^(L-1-l) d_l = -128 v, |V| < 2^41, and
      //   e = V * (-scale/128) = v * scale, exact (LimbMap esc/eoff);
      //   y':       |V| < 2^57, so v = -V >> 7 (exact) first.
      // The values equal those of the smem-A kernel bit for bit.
      // Each partial sum below is one 32 x 32 -> 64-bit multiply-add (the
      // limb sums are int32, |d| <= 2^24).
      const int c = (-(int)d[0]) >> 7;
      const double cd = i2d_exact(c);
      long long Vy = (long long)(int)d[1 + TS_LY - 1];
#pragma unroll
      for (int l = 1; l < TS_LY; ++l) Vy += (long long)(int)d[TS_LY - l] * (1ll << (8 * l));
      const double sy = LM.scale[P.k];
      const double ey = fma(magic_raw((-Vy) >> 7), sy, -MAGIC_BIAS * sy);
      double ss = 0, gs = 0;
      if (DROP0) {
        const double s0 = P.a[0] * cd;
        ss = s0 * s0;
      }
      // the ku column slots in use: at least KU_MAX - 5, as N is the limb
      // columns rounded up to 16.  e_j = V * esc exactly; every operation has
      // one constant operand, which it reads from the parameter bank.
#pragma unroll
      for (int jj = 0; jj < KU_MAX; ++jj) {
        if (jj >= KU_MAX - 5 && jj >= ku) break;
        const int j = jj + (DROP0 ? 1 : 0);
        const int o = 1 + TS_LY + TS_LU * jj;
        const double e = i2d_exact(limb3(d[o], d[o + 1], d[o + 2])) * LM.esc[j];
        const double sj = fma(P.a[j], cd, e);
        ss = fma(sj, sj, ss);
        if (GATE) gs = fma(P.g[j], e, gs);  // only the Pearson gate reads gs
      }
      if (O.tested) finish_kmer(P, O, local, valid, c, ss, gs, ey);
      else finish_kmer_lean(P, O, local, valid, c, cd, ss, gs, ey, tested_local);
    }
    flush_tested(O, tested_local);
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ------------------------------------------------------------------- host

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
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

// Bytes of a packed row in one TMA box: 128 (1024 samples), or the whole row
// where it is shorter.  A short row's box is not swizzled: its rows lie
// wpk * 8 bytes apart in shared memory, where a warp's 16-byte reads take up
// to 4 times as long (64-byte rows), a few cycles per 128-sample stage.
// Against the smem-A kernel, which those rows took before (one 128-thread
// block per SM, load, unpack, MMA and epilogue one after another): 1e7 k-mers
// at n = 700, r = 8+1 in 0.56 ms instead of 3.38 ms, 1e6 at n = 200, r = 5+1
// in 0.10 instead of 0.25 ms (whole calls).
static int ts_box_bytes(int wpk) { return wpk * 8 < 128 ? wpk * 8 : 128; }

bool ts_supported(int N, int limbs_u, int limbs_y, int kpad, int wpk) {
  if (limbs_u != TS_LU || limbs_y != TS_LY) return false;
  if (N < 16 || N > 128 || N % 16) return false;
  if (ts_nslot(N) < 2) return false;
  // the whole image stays in shared memory, beside two boxes at least: up to
  // 195 KB, with the ring as deep as the rest allows (1e7 k-mers at n = 2000,
  // r = 20+1, 160 KB and 4 boxes: 1.24 ms; the smem-A kernel takes 8.3 ms)
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return false;
  if (ts_smem(kpad * N, 2, ts_box_bytes(wpk)).total + 1024 > (uint32_t)optin) return false;
  return encode_fn() != nullptr;
}

// Boxes of the packed-row ring that fit next to the B image (at least 2).
static int ts_ring_depth(int b_bytes, int rb) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) optin = 0;
  int x = TS_XST_MAX;
  while (x > 2 && ts_smem(b_bytes, x, rb).total + 1024 > (uint32_t)optin) --x;
  if (const char* v = std::getenv("KG_TS_XST")) {
    const int want = std::atoi(v);
    if (want >= 2 && want < x) x = want;
  }
  return x;
}

// Unpack groups that take part.  A parity wait is only sound for a waiter less
// than a lap of its ring ahead.  A group that waits for the box of super-stage
// s has filled s - ug, so the MMAs of s - 2 ug have completed, and those were
// issued after every earlier super-stage was full: all boxes up to that one's
// have landed.  With ug groups the ring must therefore hold at least the boxes
// from s - 2 ug to s; where it does not (an image that leaves two or three
// boxes), one group takes every super-stage and visits every box.
static int ts_groups(int ug, int nsub, int xst) {
  const int nsp = (nsub + TS_SUPER - 1) / TS_SUPER, nbox = (nsp + 1) / 2;
  int need = 0;
  for (int s = 0; s < nsp; ++s) {
    const int e = s + 2 * ug;
    need = std::max(need, e / nsp * nbox + (e % nsp) / 2 - s / 2);
  }
  return xst >= need ? ug : 1;
}

template <int N, bool D0, bool GATE, bool WIDE>
static cudaError_t launch_ts_w(const LaunchTs& L, const CUtensorMap& tm, cudaStream_t st) {
  const int b_bytes = L.kpad * N;
  // 128-sample sub-stages: those of the image that a row reaches (kpad is
  // rounded up further; the image is zero past the row's samples)
  const int nsub = L.kpad / TS_KS < L.wpk / 2 ? L.kpad / TS_KS : L.wpk / 2;
  const int rb = ts_box_bytes(L.wpk);
  const int xst = ts_ring_depth(b_bytes, rb);
  const size_t smem = ts_smem(b_bytes, xst, rb).total + 1024;
  const int ug = ts_groups(ts_ug(N), nsub, xst);
  cudaError_t e =
      cudaFuncSetAttribute(ts_kernel<N, D0, GATE, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned long long tiles = (L.m + TS_TM - 1) / TS_TM;
  unsigned long long grid = (unsigned long long)L.num_sms;
  if (grid > tiles) grid = tiles;
  const int nbox = (nsub * 16 + 127) / 128;
  return launch_behind(L.O->over != nullptr, ts_kernel<N, D0, GATE, WIDE>, (unsigned)grid, ts_threads(N), smem, st, tm,
                       L.m, nbox, nsub, xst, ug, rb, L.Bimg, b_bytes, *L.P, *L.LM, *L.O);
}

template <int N, bool D0, bool GATE>
static cudaError_t launch_ts_t(const LaunchTs& L, const CUtensorMap& tm, cudaStream_t st) {
  return ts_box_bytes(L.wpk) == 128 ? launch_ts_w<N, D0, GATE, true>(L, tm, st)
                                    : launch_ts_w<N, D0, GATE, false>(L, tm, st);
}

cudaError_t launch_ts(const LaunchTs& L, cudaStream_t st) {
  auto enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  CUtensorMap tm;
  const cuuint64_t rowbytes = (cuuint64_t)L.wpk * 8;
  cuuint64_t gdim[2] = {rowbytes, (cuuint64_t)L.m};
  cuuint64_t gstride[1] = {rowbytes};
  const int rb = ts_box_bytes(L.wpk);
  cuuint32_t box[2] = {(cuuint32_t)rb, TS_TM};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)L.x, gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   rb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
  const bool d0 = L.drop0;
  // the per-k-mer statistics path (O.tested) evaluates the correlation too
  const bool gate = L.P->corr_thr > 0.0 || L.O->tested != nullptr;
  switch (L.LM->N) {
#define KG_TS_CASE(NN)                                                                       \
  case NN:                                                                                   \
    if (gate) return d0 ? launch_ts_t<NN, true, true>(L, tm, st) : launch_ts_t<NN, false, true>(L, tm, st); \
    return d0 ? launch_ts_t<NN, true, false>(L, tm, st) : launch_ts_t<NN, false, false>(L, tm, st);
    KG_TS_CASE(16)
    KG_TS_CASE(32)
    KG_TS_CASE(48)
    KG_TS_CASE(64)
    KG_TS_CASE(80)
    KG_TS_CASE(96)
    KG_TS_CASE(112)
    KG_TS_CASE(128)
#undef KG_TS_CASE
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kg
