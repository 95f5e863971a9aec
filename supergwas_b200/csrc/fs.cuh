// fs.cuh -- parts shared by the 4-bit screen kernels (kernel_fs.cu, kernel_fsp.cu).
#pragma once
#include <cstddef>

#include "device.cuh"

namespace kg {

constexpr int FS_TM = 128;
constexpr int FS_UNIT = 256;       // samples per unit (32 TMEM columns, 4 MMAs)
constexpr int FS_SUPER = 4;        // units per super-stage = row box = image chunk
constexpr int FS_SF = 24;          // TMEM columns of the three scale constants
constexpr int FS_XST_MAX = 12, FS_CH_MAX = 24, FS_MAXSLOT = 3;
__host__ __device__ constexpr int fs_nslot(int N) { return 2 * N + FS_SF <= 128 ? 3 : 2; }
__host__ __device__ constexpr int fs_threads(int N) { return 32 * (8 + 4 * fs_nslot(N) + 4); }

// As wait_or_abort, but looks at the abort flag before every suspension, and
// suspends for a few microseconds at most: the screen gives up through the flag (at
// 16 suspensions of 1 ms per look a launch that gave up took 13 ms).
__device__ __forceinline__ bool fs_wait(uint32_t bar, uint32_t parity, volatile int* abort,
                                        unsigned long long* counters, unsigned code, unsigned long long limit_ns) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = gtimer_ns();
  while (!*abort) {
    if (mbar_try_sleep<4000u>(bar, parity)) return true;
    if (gtimer_ns() - t0 > limit_ns) {
      atomicOr(counters + 2, (unsigned long long)code);
      *abort = 1;
    }
  }
  return false;
}

// D[tmem] (+)= A[tmem] * B[smem desc], e2m1 x e2m1 in blocks of 32 with ue8m0
// scales at sfa / sfb, FP32 accumulate.
__device__ __forceinline__ void tc_mma_mxf4_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                               uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], [%1], %2, %3, [%5], [%6], p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// Instruction descriptor: e2m1 x e2m1, ue8m0 scales, both K-major, M x N, K = 64.
__host__ __device__ constexpr uint32_t idesc_mxf4(int M, int N) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (1u << 23) | ((uint32_t)(M >> 4) << 24);
}

// 256 packed samples (eight 32-bit words) -> 32 TMEM columns.
__device__ __forceinline__ void unpack_unit(const uint32_t (&w)[8], uint32_t (&o)[32]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o[i] = w[i] & 0x11111111u;
    o[8 + i] = w[i] & 0x22222222u;
    o[16 + i] = w[i] & 0x44444444u;
    o[24 + i] = (w[i] >> 1) & 0x44444444u;
  }
}

// 32 lanes x 32 bits, 8 consecutive columns per thread (no wait).
__device__ __forceinline__ void tc_ld8p(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// The NP (a multiple of 8) accumulator columns of a slot.
template <int NP>
__device__ __forceinline__ void fs_load(uint32_t taddr, uint32_t* d) {
#pragma unroll
  for (int c = 0; c + 16 <= NP; c += 16) tc_ld16p(taddr + c, d + c);
  if (NP % 16) tc_ld8p(taddr + NP / 16 * 16, d + NP / 16 * 16);
  tc_wait_ld();
  // later uses stay behind the wait
#pragma unroll
  for (int c = 0; c + 16 <= NP; c += 16) reg_fence16(d + c);
  if (NP % 16) {
    uint32_t* r = d + NP / 16 * 16;
    asm volatile(""
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]));
  }
}

// Verdict on one k-mer from its limb sums d (count, 3 y' limbs, with GATE 4
// limbs of y - mean(y), then LU limbs per U column):
//   0  not tested; 1  tested, not emitted; 2  tested, the FP64 test decides;
//   3  the FP64 test decides, the correlation gate included.
// With xc = x - mean(x) and a residual column r that the limbs leave out,
// |r.x| <= ||r|| ||xc|| + c |sum r| / n; for the U columns together the norm
// is the largest singular value of their residuals.  bu, by, bg and mu, my, mg
// are those factors, with room for the rounding of this arithmetic.
// PAIRS: the columns of y - mean(y), if any, are not read; c = n is left open.
template <int NP, int LU, bool GATE, bool PAIRS = false>
__device__ __forceinline__ int fs_verdict(const FsPheno& F, const uint32_t* d, bool valid) {
  auto f = [&](int i) { return __uint_as_float(d[i]); };
  constexpr int U0 = 4 + (GATE ? 4 : 0), KU = (NP - U0) / LU;
  const float cf = f(0);
  float s2[2] = {0.0f, 0.0f};
#pragma unroll
  for (int j = 0; j < KU; ++j) {  // slots past the U columns hold zero limbs and zero scales
    const int o = U0 + LU * j;
    const float e = LU == 2 ? fmaf(f(o + LU - 1), F.su[LU * j + LU - 1], f(o) * F.su[LU * j]) : f(o) * F.su[j];
    s2[j & 1] = fmaf(e, e, s2[j & 1]);
  }
  const float xcn = cf * (F.n - cf) * F.inv_n;
  float nx, rs;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(nx) : "f"(xcn));
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(s2[0] + s2[1]));
  bool in = valid && cf > 0.0f && (PAIRS || cf < F.n), open = false;
  if (GATE && !PAIRS) {
    const float eg = fmaf(f(7), F.sg[3], fmaf(f(6), F.sg[2], fmaf(f(5), F.sg[1], f(4) * F.sg[0])));
    const float q = fabsf(fmaf(F.kappa, cf, eg)), err = fmaf(F.bg, nx, F.mg * cf), t = F.thr * nx;
    in = in && !(q + err < t);
    open = !(q - err > t);
  }
  const float root = rs + fmaf(F.bu, nx, F.mu * cf);
  const float low = fmaf(-root, root, xcn);  // xxM is at least this
  const float ey = fmaf(f(3), F.sy[2], fmaf(f(2), F.sy[1], f(1) * F.sy[0]));
  const float y = fabsf(fmaf(F.b, cf, ey)) + fmaf(F.by, nx, F.my * cf);
  const bool below = xcn > 0.0f && low >= 1e-3f * xcn && y * y < F.cut * low;
  return !in ? 0 : open ? 3 : below ? 1 : 2;
}
// The constants that fs_verdict<NP, LU, GATE> reads, in registers.
template <int NP, int LU, bool GATE>
__device__ __forceinline__ void fs_constants(const FsPheno* __restrict__ F, FsPheno& R) {
  constexpr int U0 = 4 + (GATE ? 4 : 0), HEAD = (int)(offsetof(FsPheno, su) / 16), NV = ((NP - U0) / LU * LU + 3) / 4;
#pragma unroll
  for (int i = 0; i < HEAD + NV; ++i) {
    if (!GATE && i == HEAD - 1) continue;  // sg
    reinterpret_cast<float4*>(&R)[i] = __ldg(reinterpret_cast<const float4*>(F) + i);
  }
}

// Appends the lanes with `take` to the candidate list (warp-aggregated).  Where that
// is too many for the tests done (fs_open_limit) the screen gives up: the counters
// say so and the CTA's waits end.
__device__ __forceinline__ void fs_push(unsigned long long* counters, volatile int* abort,
                                            unsigned long long* cand, unsigned long long cap,
                                            unsigned long long base_open, unsigned long long done,
                                            unsigned long long total, bool take, unsigned long long entry) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned mask = __ballot_sync(0xffffffffu, take);
  unsigned long long base = 0;
  const int leader = __ffs(mask) - 1;
  if ((int)lane == leader) base = atomicAdd(counters + CNT_FS_OPEN, (unsigned long long)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (base + __popc(mask) > fs_open_limit(base_open, done, total, cap)) {
    if ((int)lane == leader) {
      atomicExch(counters + CNT_FS_OVER, 1ull);
      atomicExch(counters + CNT_FS_EVER, 1ull);
      *abort = 1;
    }
  } else if (take) {
    cand[base + __popc(mask & ((1u << lane) - 1u))] = entry;
  }
}
// The same as a call: where a warp has one test per item, few warps come here, and
// inlined it cost the rest of the kernel 2 % (1e8 k-mers at n = 1000).
static __device__ __noinline__ void fs_push_call(unsigned long long* counters, volatile int* abort,
                                                 unsigned long long* cand, unsigned long long cap,
                                                 unsigned long long base_open, unsigned long long done,
                                                 unsigned long long total, bool take, unsigned long long entry) {
  fs_push(counters, abort, cand, cap, base_open, done, total, take, entry);
}
// Adds a warp's counts of decided tests (32 bits in all, as flush_tested).
__device__ __forceinline__ void fs_flush(unsigned long long* counters, uint32_t cnt) {
  const unsigned tot = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31u) == 0 && tot) atomicAdd(counters + CNT_FS_TESTED, (unsigned long long)tot);
}

// Scale constants in the FS_SF columns at t: every byte of a region of 8 columns is
// one ue8m0 value, so any arrangement of the scales reads the same: 2, 1, 1/2.
// Called by the warps of all four lane quarters.
__device__ __forceinline__ void fs_scales(uint32_t t) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t v = i == 0 ? 0x80808080u : i == 1 ? 0x7f7f7f7fu : 0x7e7e7e7eu;
    const uint32_t r8[8] = {v, v, v, v, v, v, v, v};
    tc_st8(t + 8 * i, r8);
  }
  tc_wait_st();
}
// The MMAs of one super-stage: `here` units of A at a_t against the image at bd.
template <int N>
__device__ __forceinline__ void fs_mmas(uint32_t d_t, uint32_t a_t, uint64_t bd, uint32_t sf, int here, bool first) {
  constexpr uint32_t IDESC = idesc_mxf4(FS_TM, N);
  constexpr uint32_t BSTEP = (2 * N * 16) >> 4;  // descriptor step of one MMA
#pragma unroll
  for (int u = 0; u < FS_SUPER; ++u) {
    if (u < here) {
#pragma unroll
      for (int cl = 0; cl < 4; ++cl)
        tc_mma_mxf4_ts(d_t, a_t + u * 32 + cl * 8, bd + (uint64_t)((4 * u + cl) * BSTEP), IDESC, sf + 8,
                       sf + 8 * (cl < 2 ? cl : 2), (u | cl) ? 1u : first ? 0u : 1u);
    }
  }
}

}  // namespace kg
