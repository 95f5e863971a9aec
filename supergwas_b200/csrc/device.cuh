// device.cuh -- parameters, PTX helpers and the shared FP64 epilogue of the
// association kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "params.hpp"

namespace kg {

// A bounded wait gives up after this long and reports KG_ERR_TIMEOUT.
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Exact int64 -> double for |v| < 2^51 without the conversion unit: the
// double 1.5 * 2^52 has unit spacing and a zero low 51-bit mantissa field, so
// adding v to its bit pattern yields the double 1.5 * 2^52 + v exactly
// ("magic number" conversion, Hacker's Delight ch. 17 style).  The caller
// subtracts the bias, usually folded into an FMA.
constexpr double MAGIC_BIAS = 6755399441055744.0;  // 1.5 * 2^52
__device__ __forceinline__ double magic_raw(long long v) {
  return __longlong_as_double(0x4338000000000000LL + v);
}
__device__ __forceinline__ double i2d_exact(long long v) { return magic_raw(v) - MAGIC_BIAS; }

// a * B + c, 32 x 32 -> 64 bits in one multiply-add.  B is an immediate: from
// a register each use cost a move on the uniform datapath.
template <int B>
__device__ __forceinline__ long long mad_wide(uint32_t a, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "n"(B), "l"(c));
  return d;
}
// The integer 65536 hi + 256 mid + lo of three int32 limb sums.
__device__ __forceinline__ long long limb3(uint32_t hi, uint32_t mid, uint32_t lo) {
  return mad_wide<65536>(hi, mad_wide<256>(mid, (long long)(int)lo));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// count arrivals by each lane with p set, without a branch.
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool p, uint32_t count = 1) {
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "setp.ne.u32 P1, %1, 0;\n\t"
      "@P1 mbarrier.arrive.shared::cta.b64 _, [%0], %2;\n\t}" ::"r"(bar),
      "r"((uint32_t)p), "r"(count)
      : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Non-blocking test of a phase (mbarrier.test_wait never suspends the thread).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// As mbar_try, letting the hardware suspend the thread until the phase
// completes (or NS, about 1 ms, passes) instead of returning at once, so that a
// waiting warp takes no issue slots from the warps doing the work.
template <uint32_t NS = 1000000u>
__device__ __forceinline__ bool mbar_try_sleep(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(NS)
      : "memory");
  return ok != 0;
}
// Bounded wait: false (and an error bit in counters[2]) after WAIT_LIMIT_NS.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          unsigned long long* counters, unsigned code) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = gtimer_ns();
  while (!mbar_try(bar, parity)) {
    if (gtimer_ns() - t0 > WAIT_LIMIT_NS) {
      atomicOr(counters + 2, (unsigned long long)code);
      return false;
    }
  }
  return true;
}

// ----------------------------------------------------------- bulk copies
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc], kind::i8, int32 accumulate.
__device__ __forceinline__ void tc_mma_i8_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc], kind::i8.
__device__ __forceinline__ void tc_mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
// One lane of a converged warp (the lowest active one), chosen by elect.sync.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32-bit, 16 consecutive columns per thread.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Orders later uses of 16 registers after the preceding tcgen05.wait::ld:
// the registers pass through an (empty) volatile asm that follows the wait.
__device__ __forceinline__ void reg_fence16(uint32_t* r) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]));
}
// 32 lanes x 32-bit, 16 consecutive columns per thread, into r[0..15] (no wait).
__device__ __forceinline__ void tc_ld16p(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 32 lanes x 32-bit, 8 consecutive columns per thread.
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle (core matrix = 8 rows
// x 16 bytes contiguous); lbo = byte distance of K-adjacent core matrices,
// sbo = byte distance of M/N-adjacent 8-row groups.
__device__ __forceinline__ uint64_t sdesc_noswz(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  return d;               // base offset 0, layout type 0 (no swizzle)
}

// Instruction descriptor: kind::i8, s8 x s8 -> s32, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_i8(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ------------------------------------------- TMEM-A kernels (shared parts)
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(tmap), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// 128 packed samples (four 32-bit words) -> 32 TMEM columns of int8 A
// operand: column 8q+jj holds, in byte t, sample 32q + 8t + 7 - jj as -128 x
// (jj even) or 64 x (jj odd).  make_b_image_ts lays B out to match.
__device__ __forceinline__ void unpack_stage(const uint32_t (&w)[4], uint32_t (&o)[32]) {
#pragma unroll
  for (int qq = 0; qq < 4; ++qq)
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const uint32_t u = w[qq] * (1u << (2 * h));
      o[qq * 8 + 2 * h] = u & 0x80808080u;
      o[qq * 8 + 2 * h + 1] = u & 0x40404040u;
    }
}

// Bounded wait that also gives up when another role has aborted: one test (the
// common case: the phase is already complete), then tests that let the hardware
// suspend the warp; the abort flag and the clock are read only every 16 of
// those.  limit_ns:
// how long to wait before giving up (a launch parameter, see wait_limit).
static __device__ __forceinline__ bool wait_more(uint32_t bar, uint32_t parity, volatile int* abort,
                                              unsigned long long* counters, unsigned code,
                                              unsigned long long limit_ns) {
  const unsigned long long t0 = gtimer_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_sleep(bar, parity)) return true;
    if ((it & 15u) == 0) {
      if (*abort) return false;
      if (gtimer_ns() - t0 > limit_ns) {
        atomicOr(counters + 2, (unsigned long long)code);
        *abort = 1;
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort,
                                        unsigned long long* counters, unsigned code,
                                        unsigned long long limit_ns = WAIT_LIMIT_NS) {
  return mbar_try(bar, parity) || wait_more(bar, parity, abort, counters, code, limit_ns);
}

// The pipeline wait limit of a launch: the caller's value, or WAIT_LIMIT_NS
// when it left it at 0.  Only the waits between the roles of a pipeline use
// it; the final waits for a CTA's own copies and MMAs always allow
// WAIT_LIMIT_NS, so that nothing is still landing when a CTA exits.
__device__ __forceinline__ unsigned long long wait_limit(unsigned long long ns) {
  return ns ? ns : WAIT_LIMIT_NS;
}

// A launch behind the 4-bit screen may start while the one before it still runs
// (launch_behind in kernels.hpp): waits until that one is done and its writes are
// seen.  next_may_start: a launch that follows in this way may be set up.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Ring position: slot index and phase parity, advanced without division.
template <int NS>
struct Ring {
  uint32_t slot = 0, phase = 0, used = 0;  // used: laps completed (0 = first)
  __device__ __forceinline__ void next() {
    if (++slot == (uint32_t)NS) {
      slot = 0;
      phase ^= 1u;
      used = 1;
    }
  }
};
// The same with a size chosen at launch.
struct RingN {
  uint32_t slot = 0, phase = 0, used = 0, size;
  __device__ __forceinline__ explicit RingN(uint32_t n) : size(n) {}
  __device__ __forceinline__ void next() {
    if (++slot == size) {
      slot = 0;
      phase ^= 1u;
      used = 1;
    }
  }
};

// ---------------------------------------------------------------- epilogue
// -log10 erfc(z) without underflow (log-domain tail through erfcx).
__device__ __forceinline__ double mlog10_sf(double T) {
  if (!(T > 0.0)) return 0.0;
  const double z = sqrt(0.5 * T);
  if (z < 5.0) return -log10(erfc(z));
  return (z * z - log(erfcx(z))) * 0.43429448190325182765;
}

// Warp-aggregated outputs of one k-mer: tested count, hit record, FP64
// refinement candidate, and (when requested) the per-k-mer arrays.  All 32
// lanes of the warp must call it.
// Warp-aggregated hit records and refinement candidates of one k-mer per
// lane.  All 32 lanes of the warp must call it.
__device__ __forceinline__ void emit_rare(const DevOut& O, unsigned long long local, bool hit, bool cand, double T,
                                          double p, double effect) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned hmask = __ballot_sync(0xffffffffu, hit);
  if (hmask) {
    unsigned long long base = 0;
    const int leader = __ffs(hmask) - 1;
    if ((int)lane == leader) base = atomicAdd(O.counters + 1, (unsigned long long)__popc(hmask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (hit) {
      const unsigned long long slot = base + __popc(hmask & ((1u << lane) - 1u));
      if (slot < O.hit_cap) {
        kg_hit h;
        h.kmer = O.kmer(local);
        h.effect = effect;
        h.pval = p;
        h.chisq = T;
        O.hits[slot] = h;
      } else {
        atomicOr(O.counters + 2, (unsigned long long)ERR_HIT_OVERFLOW);
      }
    }
  }
  const unsigned cmask = __ballot_sync(0xffffffffu, cand);
  if (cmask) {
    unsigned long long base = 0;
    const int leader = __ffs(cmask) - 1;
    if ((int)lane == leader) base = atomicAdd(O.counters + 3, (unsigned long long)__popc(cmask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (cand) {
      const unsigned long long slot = base + __popc(cmask & ((1u << lane) - 1u));
      if (slot < O.cand_cap) O.cand[slot] = O.kmer_offset + local;
      else atomicOr(O.counters + 2, (unsigned long long)ERR_CAND_OVERFLOW);
    }
  }
}

__device__ __forceinline__ void emit_kmer(const DevOut& O, unsigned long long local, bool valid, bool tested,
                                          bool hit, bool cand, double T, double p, double effect, double xxM,
                                          double xyM, double cor) {
  const unsigned lane = threadIdx.x & 31u;
  if (O.weight) {
    const unsigned tot = __reduce_add_sync(0xffffffffu, tested ? O.weight[O.kmer(local)] : 0u);
    if (lane == 0 && tot) atomicAdd(O.counters + 0, (unsigned long long)tot);
  } else {
    const unsigned tmask = __ballot_sync(0xffffffffu, tested);
    if (lane == 0 && tmask) atomicAdd(O.counters + 0, (unsigned long long)__popc(tmask));
  }
  emit_rare(O, local, hit, cand, T, p, effect);
  if (valid && O.tested) {
    const unsigned long long g = O.kmer_offset + local;
    O.tested[g] = tested ? 1 : 0;
    O.chisq[g] = T;
    O.pval[g] = p;
    O.effect[g] = effect;
    O.mlog10p[g] = tested ? mlog10_sf(T) : 0.0;
    O.xxM[g] = xxM;
    O.xyM[g] = xyM;
    O.cor[g] = cor;
  }
}

// Statistics and outputs of one k-mer, given c = popcount(x),
// ss = sum_j s_j^2, gs = sum_j g_j e_j, ey = d_y . x.  Must be called by
// all 32 lanes of a warp (warp-aggregated atomics).
__device__ __forceinline__ void finish_kmer(const EpiParams& P, const DevOut& O, unsigned long long local,
                                            bool valid, int c, double ss, double gs, double ey) {
  const int n = P.n;
  bool tested = valid && c > 0 && c < n && !(P.ynorm < 1e-12);
  double cor = 0.0;
  if (tested) {
    const double xcn2 = (double)c * (double)(n - c) / (double)n;  // ||x - mean x||^2
    const double xyc = ey + gs + P.kappa * (double)c;              // x . (y - mean y)
    cor = xyc / (sqrt(xcn2) * P.ynorm);
    tested = !(fabs(cor) < P.corr_thr);                             // src/kgwas.cpp:199,467
  }
  double xxM = 0, xyM = 0, effect = 0, T = 0, p = 1;
  bool cand = false;
  if (tested) {
    xxM = (double)c - ss;
    xyM = P.b * (double)c + ey;
    // compute_hit, src/kgwas.cpp:44-56
    const double eps = 1e-12;
    if (xxM > eps && P.yyM > eps) {
      double r2 = (xyM * xyM) / (xxM * P.yyM);
      if (r2 < 0) r2 = 0;
      if (r2 >= 1) r2 = 1 - 1e-15;
      if (P.refine && r2 >= P.r2_ref) {
        cand = true;  // recomputed in FP64 by refine_kernel, which emits its row
        p = 2.0;
      } else if (O.tested || r2 >= P.r2_cand) {
        T = (double)n * log(1.0 / (1.0 - r2));
        p = erfc(sqrt(0.5 * T));
        effect = xyM / (xxM * P.yyM);
      } else {
        p = 2.0;  // provably above p_thresh; the row is not emitted and no stats are kept
      }
    }
  }
  emit_kmer(O, local, valid, tested, tested && p <= P.p_thresh, cand, T, p, effect, xxM, xyM, cor);
}

// Whether a tested k-mer of the split form goes to the FP64 refinement in a
// launch that returns emitted rows only: r2 = q / den at least r2_ref, and not
// so far below the emit cut that refining cannot matter (set_refine_need).
// Refining every k-mer from chi-square 12 up took 0.1 ms per 4e7 k-mers at
// n = 1000 (5e-4 of them, 20 KB of byte tables each); from 0.9 of the cut at
// p = 1e-6 it is 4e-6 of them.
__device__ __forceinline__ bool may_refine(const EpiParams& P, double cd, double xxM, double q, double den) {
  return q >= P.r2_ref * den &&
         (q >= P.r2_need * den || !(xxM >= XXM_FLOOR * cd * ((double)P.n - cd) / (double)P.n));
}

// As finish_kmer, for launches without per-k-mer outputs: the Pearson gate
// and the emit / refinement screens compare squares instead of dividing
// (|cor| >= thr  <=>  xyc^2 >= thr^2 ||xc||^2 ||yc||^2;  r2 >= t  <=>
// xyM^2 >= t xxM yyM), and only k-mers that may reach the emit cut evaluate
// the reference formula (src/kgwas.cpp:47-53) exactly.  Tested k-mers are counted
// in a register (tested_local, flushed once per warp by the caller): in the common
// case (no hit, no refinement candidate in the warp) it costs one ballot.
__device__ __forceinline__ void finish_kmer_lean(const EpiParams& P, const DevOut& O, unsigned long long local,
                                                 bool valid, int c, double cd, double ss, double gs, double ey,
                                                 uint32_t& tested_local) {
  const int n = P.n;
  bool tested = valid && c > 0 && c < n && !(P.ynorm < 1e-12);
  if (P.corr_thr > 0.0) {
    const double xcn2 = cd * (double)(n - c) / (double)n;
    const double xyc = ey + gs + P.kappa * cd;
    tested = tested && xyc * xyc >= P.thr2_ynorm2 * xcn2;
  }
  if (tested) tested_local += O.weight ? O.weight[O.kmer_offset + local] : 1u;
  const double eps = 1e-12;
  const double xxM = cd - ss;
  const double xyM = P.b * cd + ey;
  const double q = xyM * xyM, den = xxM * P.yyM;
  const bool ok = tested && xxM > eps && P.yyM > eps;
  const bool cand = ok && P.refine && may_refine(P, cd, xxM, q, den);
  const bool maybe = ok && !cand && q >= P.r2_cand * den;
  if (__ballot_sync(0xffffffffu, cand || maybe) == 0u) return;
  double T = 0, p = 1, effect = 0;
  bool hit = false;
  if (maybe) {
    double r2 = q / den;
    if (r2 < 0) r2 = 0;
    if (r2 >= 1) r2 = 1 - 1e-15;
    T = (double)n * log(1.0 / (1.0 - r2));
    p = erfc(sqrt(0.5 * T));
    effect = xyM / den;
    hit = p <= P.p_thresh;
  }
  emit_rare(O, local, hit, cand, T, p, effect);
}

// A limb sum (int64) shifted right by s < 32 into 32 bits, as a float.
__device__ __forceinline__ float shifted_float(long long v, int s) {
  return (float)(int)__funnelshift_r((uint32_t)v, (uint32_t)((unsigned long long)v >> 32), s);
}

// Single-precision screen of one k-mer from its limb sums d (count, 5 y' limbs,
// then 3 limbs per U column 1 .. ku; the intercept in double only).  Returns
//   0  not tested;
//   1  tested, and certainly neither a row to emit nor a refinement candidate;
//   2  undecided: the FP64 statistic decides.
// FP64 instructions and the MMAs share one pipe (ncu: pipe_shared), so an FP64
// instruction waits for the MMA in the pipe, ~36 cycles beside N = 64: the
// FP64 statistic of 16 U columns took 3100 cycles per 128-k-mer tile.  The
// screen uses the integer, conversion and FP32 pipes only.  The r2 compared here
// is within a few percent of that of the limb sums where xxM is at least XXM_FLOOR
// of c (n - c) / n, and the cut it is compared with is 10 % low; the correlation is
// within half the room of gate_lo and gate_hi.  set_screen checks both for the
// phenotype (a limb sum shifted into 32 bits is good to 2^-20 of its column's
// largest value per 1024 samples).
// PAIRS: no correlation gate, and c = n is left to the FP64 form.
template <bool GATE, bool PAIRS>
__device__ __forceinline__ int screen_verdict(const ScreenParams& S, int n, int c, float ey, float ss, float gs,
                                              bool valid) {
  const float cf = (float)c;
  const float xcn = (float)(c * (n - c)) * S.inv_n;
  if (!(valid && c > 0 && (PAIRS || c < n))) return 0;
  if (GATE) {
    const float xyc = fmaf(S.kappa, cf, ey + gs);
    const float q = xyc * xyc;
    if (q < S.gate_lo * xcn) return 0;
    if (!(q > S.gate_hi * xcn)) return 2;
  }
  const float xxM = xcn - ss, xyM = fmaf(S.b, cf, ey);
  return xxM >= (float)XXM_FLOOR * xcn && xcn > 0.0f && xyM * xyM < S.cut * xxM ? 1 : 2;
}
// e_y / ynorm from the y' limb sums d[1..5], without the lowest limb.
__device__ __forceinline__ float screen_ey(const ScreenParams& S, const uint32_t* d) {
  return shifted_float(mad_wide<(1 << 24)>(d[1], limb3(d[2], d[3], d[4])), S.shift + 8) * S.sy;
}
template <int KU_MAX, int LAST, bool GATE, bool PAIRS>
__device__ __forceinline__ int screen_kmer(const ScreenParams& S, int n, const uint32_t* d, int ku, bool valid) {
  const int c = (-(int)d[0]) >> 7;
  const float ey = screen_ey(S, d);
  float ss = 0.0f, gs = 0.0f;
#pragma unroll
  for (int jj = 0; jj < KU_MAX; ++jj) {
    if (jj >= KU_MAX - LAST && jj >= ku) break;
    const int o = 6 + 3 * jj;
    const float e = shifted_float(limb3(d[o], d[o + 1], d[o + 2]), S.shift) * S.su[jj];
    ss = fmaf(e, e, ss);
    if (GATE) gs = fmaf(S.g[jj], e, gs);
  }
  return screen_verdict<GATE, PAIRS>(S, n, c, ey, ss, gs, valid);
}

// Adds the per-thread tested counts of a warp to counters[0].
__device__ __forceinline__ void flush_tested(const DevOut& O, uint32_t tested_local) {
  const unsigned tot = __reduce_add_sync(0xffffffffu, tested_local);
  if ((threadIdx.x & 31u) == 0 && tot) atomicAdd(O.counters + 0, (unsigned long long)tot);
}

// ------------------------------------------------- FP64 refinement sums
// Column sums x . v_j of one packed row from byte tables: T[(g*256 + b)*CM + j]
// is the sum of column j over the samples of 8-sample group g whose bit is set
// in b.  Lane l accumulates columns l, l+32, ... over the row's bytes in
// order, one coalesced table row per byte (instead of one V row per set bit).
// nwords: words of the row covered by the tables.  With row2, the column is
// the product of two rows (AND of their words: the 2-D pair test).  Called by
// a whole warp.
template <int CM>
__device__ __forceinline__ void table_row_sums(const uint64_t* __restrict__ row, int nwords,
                                               const double* __restrict__ T, int lane,
                                               double (&acc)[(CM + 31) / 32],
                                               const uint64_t* __restrict__ row2 = nullptr) {
  constexpr int JW = (CM + 31) / 32;
#pragma unroll
  for (int jj = 0; jj < JW; ++jj) acc[jj] = 0.0;
  // Four words (32 loads) at a time where a lane has one column: a candidate is a
  // chain of L2 latencies and a launch has few of them.  1e8 k-mers at n = 1000,
  // r = 16+1: 23 us with one word at a time, 14 us now.  Two columns per lane
  // (k > 30) gained nothing.  The sums are added in the same order.
  constexpr int TRW = JW == 1 ? 4 : 1;
  for (int w0 = 0; w0 < nwords; w0 += TRW) {
    uint64_t bits[TRW];
#pragma unroll
    for (int u = 0; u < TRW; ++u) {
      const int w = w0 + u < nwords ? w0 + u : nwords - 1;
      bits[u] = __ldg(row + w);  // one address for the whole warp
      if (row2) bits[u] &= __ldg(row2 + w);
      if (w0 + u >= nwords) bits[u] = 0;  // the entries of an empty byte are zero
    }
    double v[TRW][8][JW];
#pragma unroll
    for (int u = 0; u < TRW; ++u) {
      const double* Tw = T + (size_t)(w0 + u < nwords ? w0 + u : nwords - 1) * (8 * 256 * CM);
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const unsigned b = (unsigned)(bits[u] >> (8 * t)) & 255u;
        const double* e = Tw + (size_t)(t * 256 + b) * CM;
#pragma unroll
        for (int jj = 0; jj < JW; ++jj) {
          const int j = lane + 32 * jj;
          v[u][t][jj] = (j < CM) ? __ldg(e + j) : 0.0;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < TRW; ++u)
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int jj = 0; jj < JW; ++jj) acc[jj] += v[u][t][jj];
  }
}

// The column sums of a row (of a product of two, with row2) over the values that
// the int8 limbs hold: integers times the column's scale, so exact in any order
// and equal to the recombined limb sums.  V: the FP64 columns, nwords * 64 rows;
// scale[j]: limb scale of U column j, of y' at k.  For the candidates whose
// outcome turns on the roundings of the limbs.
template <int CM>
__device__ __noinline__ void split_columns(int k, const double* scale, const double* __restrict__ V,
                                           const uint64_t* __restrict__ row, const uint64_t* __restrict__ row2,
                                           int nwords, int lane, double (&e)[(CM + 31) / 32]) {
#pragma unroll
  for (int jj = 0; jj < (CM + 31) / 32; ++jj) {
    e[jj] = 0.0;
    const int col = lane + 32 * jj;  // the count, U column col - 1, y' at k + 1
    if (col < 2 || col > k + 1) continue;
    const double sc = scale[col - 1], up = 1.0 / sc;  // powers of two
    double sum = 0.0;
    for (int w = 0; w < nwords; ++w) {
      const uint64_t bits = row2 ? row[w] & row2[w] : row[w];
      const double* v = V + (size_t)(64 * w) * CM + col;
      for (int b = 0; b < 64; b += 16) {
        double t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = __ldg(v + (size_t)(b + i) * CM);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum += (bits >> (b + i)) & 1u ? round(t[i] * up) : 0.0;
      }
    }
    e[jj] = sum * sc;
  }
}

// Correlation gate of a refinement candidate, identical in every lane: from its
// FP64 column sums (refine_reduce), or, where those are so near the threshold
// that the roundings of the limbs decide (P.gate_unit), from the limb sums in the
// expressions of the int8 kernels.
template <int CM>
__device__ __forceinline__ bool refine_gate(const EpiParams& P, const LimbMap& LM, const double* __restrict__ V,
                                            const uint64_t* __restrict__ row, int nwords,
                                            const double (&acc)[(CM + 31) / 32], int lane, int c, double ey) {
  constexpr int JW = (CM + 31) / 32;
  double gs = 0.0;
#pragma unroll
  for (int jj = 0; jj < JW; ++jj) {
    const int j = lane + 32 * jj;
    if (j >= 1 && j <= P.k) gs += P.g[j - 1] * acc[jj];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, o);
  const double cd = (double)c;
  const double xcn2 = cd * (double)(P.n - c) / (double)P.n;
  double xyc = ey + gs + P.kappa * cd;
  const double t = sqrt(P.thr2_ynorm2 * xcn2);
  if (!(fabs(fabs(xyc) - t) > 1.01 * P.gate_unit * cd + 1e-11 * t)) {
    double e[JW];
    split_columns<CM>(P.k, LM.scale, V, row, nullptr, nwords, lane, e);
    gs = 0.0;
#pragma unroll
    for (int jj = 0; jj < JW; ++jj)
      for (int l = 0; l < 32; ++l) {
        const double ej = __shfl_sync(0xffffffffu, e[jj], l);
        const int col = l + 32 * jj;
        if (col >= 2 && col <= P.k) gs = fma(P.g[col - 1], ej, gs);
        if (col == P.k + 1) ey = ej;
      }
    xyc = ey + gs + P.kappa * cd;
  }
  return xyc * xyc >= P.thr2_ynorm2 * xcn2;
}

// From the lane-distributed column sums (column 0 = count, 1..k = U columns,
// k+1 = y'): c, ss = sum_j (a_j c + e_j)^2 and ey, identical in every lane.
template <int CM>
__device__ __forceinline__ void refine_reduce(const EpiParams& P, const double (&acc)[(CM + 31) / 32], int lane,
                                              int& c, double& ss, double& ey) {
  constexpr int JW = (CM + 31) / 32;
  c = (int)__shfl_sync(0xffffffffu, acc[0], 0);
  const double cd = (double)c;
  double s2 = 0.0, y = 0.0;
#pragma unroll
  for (int jj = 0; jj < JW; ++jj) {
    const int j = lane + 32 * jj;
    if (j >= 1 && j <= P.k) {
      const double sj = P.a[j - 1] * cd + acc[jj];
      s2 += sj * sj;
    } else if (j == P.k + 1) {
      y = acc[jj];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  ss = s2;
  ey = y;
}

// ------------------------------------------------ many-phenotype helpers
// Shard of a global k-mer index (shard_start ascending, shard_start[0] = 0).
__device__ __forceinline__ int mp_shard(const DevOutMP& O, unsigned long long gk) {
  int lo = 0, hi = O.n_shards - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (O.shard_start[mid] <= gk) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Adds the lanes' counts of phenotype p to their (shard, phenotype) counters:
// one atomic per distinct shard in the warp.
__device__ __forceinline__ void tb_count(const DevOutMP& O, int p, int shard, uint32_t cnt) {
  const unsigned match = __match_any_sync(0xffffffffu, shard);
  const unsigned tot = __reduce_add_sync(match, cnt);
  if ((int)(threadIdx.x & 31u) == __ffs(match) - 1 && tot)
    atomicAdd(O.tested + (size_t)shard * O.n_pheno + p, (unsigned long long)tot);
}

// Statistic of one (k-mer, phenotype) from the exact integer sums, as the
// division-free screen of finish_kmer_lean; writes the outcome flags.
__device__ __forceinline__ void mp_eval(const EpiParams& P, bool valid, int c, double ss, double gs, double ey,
                                        bool& tested, bool& hit, bool& cand, double& T, double& p, double& effect) {
  const int n = P.n;
  tested = valid && c > 0 && c < n && !(P.ynorm < 1e-12);
  if (tested && P.corr_thr > 0.0) {
    const double xcn2 = (double)c * (double)(n - c) / (double)n;
    const double xyc = ey + gs + P.kappa * (double)c;
    tested = xyc * xyc >= P.thr2_ynorm2 * xcn2;
  }
  hit = cand = false;
  T = 0;
  p = 1;
  effect = 0;
  if (!tested) return;
  const double xxM = (double)c - ss, xyM = P.b * (double)c + ey;
  const double eps = 1e-12;
  if (!(xxM > eps && P.yyM > eps)) {
    hit = p <= P.p_thresh;
    return;
  }
  const double q = xyM * xyM, den = xxM * P.yyM;
  if (P.refine && may_refine(P, (double)c, xxM, q, den)) {
    cand = true;
  } else if (q >= P.r2_cand * den) {
    double r2 = q / den;
    if (r2 < 0) r2 = 0;
    if (r2 >= 1) r2 = 1 - 1e-15;
    T = (double)n * log(1.0 / (1.0 - r2));
    p = erfc(sqrt(0.5 * T));
    effect = xyM / den;
    hit = p <= P.p_thresh;
  }
}

__device__ __forceinline__ void mp_emit_rare(const DevOutMP& O, int p, unsigned long long gk, int shard, bool hit,
                                             bool cand, double T, double pv, double effect);

// Accumulator columns of one phenotype slot, 48 at a time: column 0 is the
// count, 1-5 the y' limbs, then 3 limbs per U column, so that a chunk never
// splits a limb group.
constexpr int MP_CH = 48;
template <int NP, int CHUNK>
__device__ __forceinline__ void mp_load_chunk(uint32_t taddr, uint32_t (&d)[MP_CH]) {
#pragma unroll
  for (int c16 = 0; c16 < MP_CH / 16; ++c16)
    if (CHUNK * MP_CH + c16 * 16 < NP) tc_ld16p(taddr + CHUNK * MP_CH + c16 * 16, d + c16 * 16);
  tc_wait_ld();
#pragma unroll
  for (int c16 = 0; c16 < MP_CH / 16; ++c16)
    if (CHUNK * MP_CH + c16 * 16 < NP) reg_fence16(d + c16 * 16);
}

// screen_kmer for one phenotype slot of NP accumulator columns at tensor-memory
// address taddr; the phenotype's constants come from global memory.  Slots
// past its U columns hold zero limbs.
template <int NP, int CHUNK, bool GATE>
__device__ __forceinline__ void mp_screen_chunk(const ScreenParams& S, uint32_t taddr, int& c, float& ey, float& ss,
                                                float& gs) {
  uint32_t d[MP_CH];
  mp_load_chunk<NP, CHUNK>(taddr, d);
  if (CHUNK == 0) {
    c = (-(int)d[0]) >> 7;
    ey = screen_ey(S, d);
  }
  constexpr int J0 = CHUNK == 0 ? 0 : (CHUNK * MP_CH - 6) / 3;
  constexpr int JN = (NP - 6) / 3, JE = (CHUNK * MP_CH + MP_CH - 6) / 3 < JN ? (CHUNK * MP_CH + MP_CH - 6) / 3 : JN;
#pragma unroll
  for (int j = J0; j < JE; ++j) {
    const int o = 6 + 3 * j - CHUNK * MP_CH;
    const float e = shifted_float(limb3(d[o], d[o + 1], d[o + 2]), S.shift) * __ldg(S.su + j);
    ss = fmaf(e, e, ss);
    if (GATE) gs = fmaf(__ldg(S.g + j), e, gs);
  }
}
template <int NP, bool GATE>
__device__ __forceinline__ int mp_screen_t(const ScreenParams& S, int n, uint32_t taddr, bool valid) {
  int c = 0;
  float ey = 0.0f, ss = 0.0f, gs = 0.0f;
  mp_screen_chunk<NP, 0, GATE>(S, taddr, c, ey, ss, gs);
  if (NP > MP_CH) mp_screen_chunk<NP, 1, GATE>(S, taddr, c, ey, ss, gs);
  if (NP > 2 * MP_CH) mp_screen_chunk<NP, 2, GATE>(S, taddr, c, ey, ss, gs);
  return screen_verdict<GATE, false>(S, n, c, ey, ss, gs, valid);
}
// Returns 2 where the phenotype has no screen.
template <int NP>
__device__ __forceinline__ int mp_screen(const EpiParams& P, uint32_t taddr, bool valid) {
  if (!P.S.on) return 2;
  return P.S.gate ? mp_screen_t<NP, true>(P.S, P.n, taddr, valid) : mp_screen_t<NP, false>(P.S, P.n, taddr, valid);
}

// The exact limb recombination and FP64 sums of one phenotype slot.
template <int NP, int CHUNK>
__device__ __forceinline__ void mp_exact_chunk(const MPheno* ME, uint32_t taddr, int& c, double& cd, double& ey,
                                               double& ss, double& gs) {
  const EpiParams& P = ME->P;
  const int drop0 = ME->drop0;
  uint32_t d[MP_CH];
  mp_load_chunk<NP, CHUNK>(taddr, d);
  if (CHUNK == 0) {
    // limb sums hold -128 * integer sums (see kernel_ts.cu)
    c = (-(int)d[0]) >> 7;
    cd = i2d_exact(c);
    long long Vy = (long long)(int)d[5];
#pragma unroll
    for (int l = 1; l < 5; ++l) Vy += (long long)(int)d[5 - l] * (1ll << (8 * l));
    const double sy = ME->LM.scale[P.k];
    ey = fma(magic_raw((-Vy) >> 7), sy, -MAGIC_BIAS * sy);
    if (drop0) {
      const double s0 = P.a[0] * cd;
      ss = s0 * s0;
    }
  }
  constexpr int J0 = CHUNK == 0 ? 0 : (CHUNK * MP_CH - 6) / 3;
  constexpr int JN = (NP - 6) / 3, JE = (CHUNK * MP_CH + MP_CH - 6) / 3 < JN ? (CHUNK * MP_CH + MP_CH - 6) / 3 : JN;
  // slots past the phenotype's k columns have zero limbs and zero constants:
  // they add exact zeros
#pragma unroll
  for (int jj = J0; jj < JE; ++jj) {
    const int o = 6 + 3 * jj - CHUNK * MP_CH;
    const int j = jj + drop0;
    const double ej = i2d_exact(limb3(d[o], d[o + 1], d[o + 2])) * ME->LM.esc[j];
    const double sj = fma(P.a[j], cd, ej);
    ss = fma(sj, sj, ss);
    gs = fma(P.g[j], ej, gs);
  }
}
// Statistic of one (k-mer, phenotype) of a resident-image kernel: the screen,
// and the FP64 statistic for warps with a k-mer that it leaves.  Returns
// whether the k-mer counts as tested; emits rows and candidates.  Called by
// all 32 lanes.
template <int NP>
__device__ __forceinline__ bool mp_test(const DevOutMP& O, const MPheno* ME, uint32_t taddr, int p,
                                        unsigned long long gk, int shard, bool valid) {
  const int v = mp_screen<NP>(ME->P, taddr, valid);
  if (!__any_sync(0xffffffffu, v == 2)) return v != 0;
  int c = 0;
  double cd = 0, ey = 0, ss = 0, gs = 0;
  mp_exact_chunk<NP, 0>(ME, taddr, c, cd, ey, ss, gs);
  if (NP > MP_CH) mp_exact_chunk<NP, 1>(ME, taddr, c, cd, ey, ss, gs);
  if (NP > 2 * MP_CH) mp_exact_chunk<NP, 2>(ME, taddr, c, cd, ey, ss, gs);
  bool tested, hit, cand;
  double T, pv, effect;
  mp_eval(ME->P, valid, c, ss, gs, ey, tested, hit, cand, T, pv, effect);
  if (__any_sync(0xffffffffu, hit || cand)) mp_emit_rare(O, p, gk, shard, hit, cand, T, pv, effect);
  return tested;
}

// Warp-aggregated hit records and FP64 refinement candidates (k-mer |
// phenotype << 48) of one (k-mer, phenotype) per lane.  All 32 lanes of the warp
// must call it.
__device__ __forceinline__ void mp_emit_rare(const DevOutMP& O, int p, unsigned long long gk, int shard, bool hit,
                                             bool cand, double T, double pv, double effect) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned hm = __ballot_sync(0xffffffffu, hit);
  if (hm) {
    unsigned long long hb = 0;
    const int hl = __ffs(hm) - 1;
    if ((int)lane == hl) hb = atomicAdd(O.counters + 1, (unsigned long long)__popc(hm));
    hb = __shfl_sync(0xffffffffu, hb, hl);
    if (hit) {
      const unsigned long long slot = hb + __popc(hm & ((1u << lane) - 1u));
      if (slot < O.hit_cap) {
        kg_phit hrec;
        hrec.kmer = gk;
        hrec.pheno = p;
        hrec.shard = shard;
        hrec.effect = effect;
        hrec.pval = pv;
        hrec.chisq = T;
        O.hits[slot] = hrec;
      } else {
        atomicOr(O.counters + 2, (unsigned long long)ERR_HIT_OVERFLOW);
      }
    }
  }
  const unsigned cm = __ballot_sync(0xffffffffu, cand);
  if (cm) {
    unsigned long long cb = 0;
    const int cl = __ffs(cm) - 1;
    if ((int)lane == cl) cb = atomicAdd(O.counters + 3, (unsigned long long)__popc(cm));
    cb = __shfl_sync(0xffffffffu, cb, cl);
    if (cand) {
      const unsigned long long slot = cb + __popc(cm & ((1u << lane) - 1u));
      if (slot < O.cand_cap) O.cand[slot] = gk | ((unsigned long long)p << 48);
      else atomicOr(O.counters + 2, (unsigned long long)ERR_CAND_OVERFLOW);
    }
  }
}

// ------------------------------------------------------ pair schedule
struct PairUnit {
  unsigned long long jb, i0, i1;
};
// Unit u -> its j-block (the last block whose first unit is <= u) and i range.
__device__ __forceinline__ PairUnit pr_unit(const PairSched& S, unsigned long long u) {
  int lo = 0, hi = S.njb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (S.unit_off[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  PairUnit U;
  U.jb = (unsigned long long)lo;
  const unsigned long long jend = 128ull * (U.jb + 1) < S.n_kmers ? 128ull * (U.jb + 1) : S.n_kmers;
  const unsigned long long ihi = S.row_end < jend - 1 ? S.row_end : jend - 1;
  U.i0 = S.row_start + (u - S.unit_off[lo]) * S.ic;
  U.i1 = U.i0 + S.ic < ihi ? U.i0 + S.ic : ihi;
  return U;
}

}  // namespace kg
