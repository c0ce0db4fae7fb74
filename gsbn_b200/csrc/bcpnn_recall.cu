/*
 * bcpnn_recall.cu -- replicate recall engine (include/bcpnn_recall.h).
 *
 * Two launches per tick on two streams, side by side (or, of a small BF16
 * network, one launch of CTAs of both kinds): the population update
 * of tick t (recall_pop_kernel: support from epsc(t-1), softmax/WTA, Philox
 * spikes, writing dsup(t), the BF16 spike row S(t) and the recall counters)
 * and the contraction with its epilogue epsc(t) = epsc(t-1) * (1 - kepsc) +
 * S(t-3) . W.  The contraction comes in two forms, chosen at create time:
 *
 * BF16 (recall_tick_kernel), persistent, CTA tile = 128 replicates x 256
 * destination MCUs, the K loop over the N source MCUs in stages of 64:
 *   warp 0      TMA producer: S(t-3) tile [128 x 64] and W^T tile [256 x 64]
 *               (BF16, 128-byte swizzle) into a 4-stage shared-memory ring,
 *               one mbarrier per stage with the transaction byte count;
 *   warp 1      allocates 512 TMEM columns (two accumulators); one elected
 *               thread issues tcgen05.mma.cta_group::1.kind::f16 (M=128,
 *               N=256, K=16, FP32 accumulate) per 16-wide K step and
 *               tcgen05.commit to free each stage and, at the end, to signal
 *               the accumulator;
 *   warps 2..5  epilogue, one replicate row per thread (TMEM lane = row):
 *               tcgen05.ld of the accumulator and the epsc update.
 *
 * FP32: W kept in FP32, the spikes as bits.  recall_events_kernel adds the
 * weights of the sources that spiked, in ascending order; where most sources
 * can spike, or a weight is not finite, recall_fp32_kernel multiplies densely
 * (CTA tile 128 x 128, 8 x 8 outputs per thread, K stages of 16
 * double-buffered in shared memory), to the same bits.
 *
 * Every mbarrier wait is bounded (1 s of %globaltimer); a wait that runs out
 * sets an error bit and the CTA leaves its loops, waits (bounded) for its own
 * outstanding copies and MMAs, frees TMEM and returns.  No cluster multicast.
 */
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "bcpnn_numerics.h"
#include "bcpnn_recall.h"
#include "host_copy.h"

namespace bcpnn_recall_dev {

constexpr int kTileM = 128, kTileN = 256, kTileK = 64, kStages = 4, kUmmaK = 16;
constexpr int kThreads = 192;
constexpr int kMaxPartsLog = 3, kMaxParts = 1 << kMaxPartsLog; /* column parts of a tile, see Tiles */
constexpr uint32_t kBytesA = kTileM * kTileK * 2; /* 16 KB */
constexpr uint32_t kBytesB = kTileN * kTileK * 2; /* 32 KB */
constexpr uint32_t kStageBytes = kBytesA + kBytesB;
constexpr uint32_t kTmemCols = 512; /* two 128 x 256 FP32 accumulators */
constexpr int kEpiThreads = 128;
constexpr int kErrWait = 4;
constexpr int kErrAlign = 8; /* a self-check found a misaligned or out-of-range access (skipped) */
constexpr unsigned long long kWaitNs = 1000000000ull;
/* dynamic shared memory: ring (1024-aligned) + barriers + TMEM address */
constexpr size_t kSmemBytes = 1024 + kStages * kStageBytes + 256;

struct Params {
  const float* dsup_prev;
  float* dsup_cur;
  const float* epsc_prev;
  float* epsc_cur;
  uint16_t* s_out; /* BF16 [R][N] spikes of this tick (BF16 contraction) */
  uint32_t* s_bits; /* the same as bits [R][N/32] (FP32 contraction) */
  uint8_t* counts; /* [R][N] */
  int count_on;
  const float* bj;
  const int32_t* lgidx; /* [R][H] */
  const float* wmask;   /* [R][H] */
  float lg_hit, lg_miss;
  int N, H, R;
  float taumdt, maxfqdt, wtagain, igain, wgain, lgbias, snoise, one_m_kepsc, pr;
  uint32_t seed_base;
  int simstep;
  int poisson;
  float one; /* 1, see add2m */
  /* maxfqdt in units of 2^-32, rounded up by 2^-20, as the division by an HCU's sum takes it: the quotient maxfqdt / sum
     of a sum near the largest float is subnormal, and off by more than that margin once times an activity */
  float bound1;
  uint32_t pr_count; /* a 24-bit uniform k 2^-24 is below pr for k < pr_count */
  int* err;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

/* bounded wait; false when it ran out or another thread reported an error */
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = gtimer();
  while (!mbar_try_wait(bar, parity)) {
    if (*(volatile int*)err) return false;
    if (gtimer() - t0 > kWaitNs) {
      atomicOr(err, kErrWait);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

/* shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row
   core groups 1024 bytes apart, descriptor version 1 (sm_100) */
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                /* leading byte offset (unused for swizzled K-major) */
  d |= (uint64_t)(1024 >> 4) << 32;      /* stride byte offset */
  d |= (uint64_t)1 << 46;                /* version */
  d |= (uint64_t)2 << 61;                /* SWIZZLE_128B */
  return d;
}

/* instruction descriptor: D F32, A BF16, B BF16, both K-major, M=128, N columns */
__device__ __forceinline__ uint32_t umma_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                     uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

/* 32 consecutive FP32 accumulator columns of this thread's lane */
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

/* population update of tick `simstep` for MCU 0 of the population (the
   softmax max seed of every HCU, Pop.cpp:270) */
__device__ __forceinline__ float dsup_mcu0(const Params& p, int row, uint32_t seed) {
  const size_t base = (size_t)row * p.N;
  float wsup = 0.0f;
  wsup += p.bj[0] + p.epsc_prev[base];
  float noise = 0.0f;
  if (p.snoise != 0.0f) noise = p.snoise * bx_normal01(seed, 0u, (uint32_t)p.simstep, 0u);
  float lginp = (p.lgidx[(size_t)row * p.H] == 0) ? p.lg_hit : p.lg_miss;
  float sup = p.lgbias + p.igain * lginp + noise;
  sup += (p.wgain * p.wmask[(size_t)row * p.H]) * wsup;
  float d = p.dsup_prev[base];
  return d + (sup - d) * p.taumdt;
}

/* two IEEE operations in one instruction, as a 64-bit register pair.  A sum
   that may take a product is add2m, a multiply-add by a 1 that the compiler does
   not know: a product before an add.rn.f32x2 came out as one multiply-add with
   one rounding. */
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  return (f32x2)__float_as_uint(a) | ((f32x2)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(a, a); }

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 c;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 c;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}

/* a * unit + b, unit = 1: a + b; unit = -1: b - a */
__device__ __forceinline__ f32x2 add2m(f32x2 a, f32x2 b, f32x2 unit) {
  f32x2 c;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(c) : "l"(a), "l"(unit), "l"(b));
  return c;
}

/* bx_expf of two values in (kExpLow, 0], where its result is normal: the same
   operations on pairs, without its clamps and its two-step scaling (the result
   is the polynomial's bits plus the exponent).  Same bits. */
constexpr float kExpLow = -83.0f;

__device__ __forceinline__ f32x2 exp2_near(f32x2 x, f32x2 one, f32x2 neg) {
  const f32x2 shift = dup2(0x1.8p23f);
  const f32x2 t = add2m(mul2(x, dup2(0x1.715476p+0f)), shift, one);
  const f32x2 kf = add2m(shift, t, neg);
  const f32x2 r = add2m(mul2(kf, dup2(0x1.7f7d1cp-20f)), add2m(mul2(kf, dup2(0x1.62e4p-1f)), x, neg), neg);
  f32x2 p = dup2(0x1.a01a02p-16f);
  p = add2m(mul2(p, r), dup2(0x1.a01a02p-13f), one);
  p = add2m(mul2(p, r), dup2(0x1.6c16c2p-10f), one);
  p = add2m(mul2(p, r), dup2(0x1.111112p-7f), one);
  p = add2m(mul2(p, r), dup2(0x1.555556p-5f), one);
  p = add2m(mul2(p, r), dup2(0x1.555556p-3f), one);
  p = add2m(mul2(p, r), dup2(0.5f), one);
  p = add2m(mul2(p, r), dup2(1.0f), one);
  p = add2m(mul2(p, r), dup2(1.0f), one);
  /* t's low bits are k + 2^22 (mod 2^9 all that shifts in): k << 23 */
  const uint32_t a = (uint32_t)p + ((uint32_t)t << 23), b = (uint32_t)(p >> 32) + ((uint32_t)(t >> 32) << 23);
  return (f32x2)a | ((f32x2)b << 32);
}

/* Population update of tick `simstep` (Pop.cpp:229-323) for a quarter of one
   HCU of one replicate: thread tid = (replicate * H + HCU) * 4 + q holds the
   groups of four MCUs q, q + 4, ... of the HCU (M/16 of them), so four
   consecutive lanes hold an HCU and read and write 64 contiguous bytes of every
   array at a time.  The HCU maximum is a shuffle max (exact); the activity sum
   keeps gsbn's serial MCU order by passing the running sum from lane to lane,
   group by group; one Philox call per four MCUs and stream.  Its own kernel,
   run beside the contraction on a second stream: a CTA of the BF16 contraction
   leaves room on its SM for three of its CTAs.

   Bound by instruction issue: two Philox4x32-10 calls of about 50 instructions
   per four MCUs, one exp per MCU.  Support and exp run on pairs of MCUs in one
   instruction.  The division of a spike's activity by the HCU's sum is done
   only where the uniform is below the activity times maxfq dt / sum, rounded up
   by 2^-20: about one group of four in 150 here; the comparison decides as if
   every MCU divided (the exact product is below that bound by more than its
   roundings, and a uniform of 0 always takes the exact path).  The recall counters are
   touched only where a group has a spike.  kBits: the spikes as bits, for the
   FP32 contraction.  64 x 64, 4096 replicates: 80 us alone; 100 as one exp and
   one division per MCU, with 16 contiguous MCUs per lane. */
template <int M, bool kBits>
__device__ __forceinline__ void recall_pop(const Params& p, int tid) {
  constexpr int G = M / 16; /* groups of four MCUs per lane */
  const int lane = threadIdx.x & 31;
  const int g = tid >> 2, q = tid & 3;
  const int h = g % p.H, r = g / p.H;
  const uint32_t seed = p.seed_base + (uint32_t)r;
  const size_t row = (size_t)r * p.N;
  const int c0 = h * M; /* group i of the lane: MCUs c0 + (4 i + q) * 4 .. + 3 */
  /* self-check: every vector access below is in bounds and aligned */
  {
    const size_t n = (size_t)p.R * p.N;
    const bool bad = r >= p.R || row + c0 + M > n || ((row + c0) & 15) != 0 || (c0 + M) > p.N ||
                     (reinterpret_cast<uintptr_t>(p.dsup_prev) & 15) || (reinterpret_cast<uintptr_t>(p.dsup_cur) & 15) ||
                     (reinterpret_cast<uintptr_t>(p.epsc_prev) & 15) || (reinterpret_cast<uintptr_t>(p.bj) & 15) ||
                     (kBits ? reinterpret_cast<uintptr_t>(p.s_bits) & 15 : reinterpret_cast<uintptr_t>(p.s_out) & 15) ||
                     (reinterpret_cast<uintptr_t>(p.counts) & 15);
    /* the warp leaves together: the shuffles below take all 32 lanes */
    if (__any_sync(0xffffffffu, bad)) {
      if (bad && atomicOr(p.err, kErrAlign) == 0) p.err[1] = tid;
      return;
    }
  }
  const float seed0 = dsup_mcu0(p, r, seed);
  const int lg = p.lgidx[(size_t)r * p.H + h];
  const float wm = p.wgain * p.wmask[(size_t)r * p.H + h];
  const float base_hit = p.lgbias + p.igain * p.lg_hit, base_miss = p.lgbias + p.igain * p.lg_miss;
  const f32x2 one = dup2(p.one), neg = dup2(-p.one);
  f32x2 d[2 * G];
#pragma unroll
  for (int i = 0; i < G; i++) {
    const int m = (4 * i + q) * 4;
    const float4 dp = *reinterpret_cast<const float4*>(p.dsup_prev + row + c0 + m);
    const float4 ep = *reinterpret_cast<const float4*>(p.epsc_prev + row + c0 + m);
    const float4 bb = *reinterpret_cast<const float4*>(p.bj + c0 + m);
    float sup[4];
#pragma unroll
    for (int k = 0; k < 4; k++) sup[k] = lg == m + k ? base_hit : base_miss;
    if (p.snoise != 0.0f) {
#pragma unroll
      for (int k = 0; k < 4; k++) sup[k] += p.snoise * bx_normal01(seed, 0u, (uint32_t)p.simstep, (uint32_t)(c0 + m + k));
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) sup[k] += 0.0f;
    }
    const f32x2 dv[2] = {pack2(dp.x, dp.y), pack2(dp.z, dp.w)};
    const f32x2 wsup[2] = {add2(dup2(0.0f), add2(pack2(bb.x, bb.y), pack2(ep.x, ep.y))),
                           add2(dup2(0.0f), add2(pack2(bb.z, bb.w), pack2(ep.z, ep.w)))};
#pragma unroll
    for (int v = 0; v < 2; v++) {
      const f32x2 s2 = add2m(mul2(dup2(wm), wsup[v]), pack2(sup[2 * v], sup[2 * v + 1]), one);
      d[2 * i + v] = add2m(mul2(add2m(dv[v], s2, neg), dup2(p.taumdt)), dv[v], one);
    }
  }
  float mx = seed0; /* the new dsup of population MCU 0 (also d[0] of HCU 0's first quarter) */
#pragma unroll
  for (int i = 0; i < 2 * G; i++) {
    mx = (lo2(d[i]) > mx) ? lo2(d[i]) : mx;
    mx = (hi2(d[i]) > mx) ? hi2(d[i]) : mx;
  }
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  const float maxact = bx_expf(p.wtagain * mx);
  f32x2 a[2 * G];
  bool near = true;
#pragma unroll
  for (int i = 0; i < 2 * G; i++) {
    a[i] = mul2(dup2(p.wtagain), add2m(dup2(mx), d[i], neg));
    near = near & (lo2(a[i]) > kExpLow) & (hi2(a[i]) > kExpLow) & (lo2(a[i]) <= 0.0f) & (hi2(a[i]) <= 0.0f);
  }
  if (near) {
#pragma unroll
    for (int i = 0; i < 2 * G; i++) a[i] = exp2_near(a[i], one, neg);
  } else {
#pragma unroll 1
    for (int i = 0; i < 2 * G; i++) {
      f32x2 v = 0;
#pragma unroll
      for (int j = 0; j < 2 * G; j++) v = i == j ? a[j] : v;
      v = pack2(bx_expf(lo2(v)), bx_expf(hi2(v)));
#pragma unroll
      for (int j = 0; j < 2 * G; j++) a[j] = i == j ? v : a[j];
    }
  }
  if (maxact < 1.0f) {
#pragma unroll
    for (int i = 0; i < 2 * G; i++) a[i] = mul2(a[i], dup2(maxact));
  }
  float vs = 0.0f;
#pragma unroll
  for (int i = 0; i < G; i++)
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const float v = (((vs + lo2(a[2 * i])) + hi2(a[2 * i])) + lo2(a[2 * i + 1])) + hi2(a[2 * i + 1]);
      vs = __shfl_sync(0xffffffffu, v, (lane & ~3) | s);
    }
  /* above every product (act / vs) * maxfqdt, in units of 2^-32 */
  const float bound = vs > 1.0f ? p.bound1 / vs : p.bound1;
#pragma unroll
  for (int i = 0; i < G; i++)
    *reinterpret_cast<float4*>(p.dsup_cur + row + c0 + (4 * i + q) * 4) =
        make_float4(lo2(d[2 * i]), hi2(d[2 * i]), lo2(d[2 * i + 1]), hi2(d[2 * i + 1]));
  uint32_t all = 0u; /* four bits per group */
#pragma unroll
  for (int i = 0; i < G; i++) {
    const int m = (4 * i + q) * 4;
    bx_u32x4 cu;
    cu.v[0] = (uint32_t)(c0 + m) >> 2;
    cu.v[1] = (uint32_t)p.simstep;
    cu.v[2] = 0u;
    cu.v[3] = 0u;
    uint32_t bits = 0u;
    if (p.poisson) {
      const bx_u32x4 op = bx_philox4x32_10(cu, seed, 0u * 16u + BX_STREAM_POISSON);
#pragma unroll
      for (int k = 0; k < 4; k++)
        if ((op.v[k] >> 8) < p.pr_count) bits |= 1u << k;
    }
    const bx_u32x4 ou = bx_philox4x32_10(cu, seed, 0u * 16u + BX_STREAM_UNIFORM);
    const float av[4] = {lo2(a[2 * i]), hi2(a[2 * i]), lo2(a[2 * i + 1]), hi2(a[2 * i + 1])};
    /* the uniform is x >> 8: x itself against the bound plus the low byte */
    bool near_spike = false;
#pragma unroll
    for (int k = 0; k < 4; k++) near_spike |= (float)ou.v[k] <= av[k] * bound + 257.0f;
    if (near_spike) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        float act = av[k];
        if (vs > 1.0f) act /= vs;
        if (bx_u01(ou.v[k]) < act * p.maxfqdt) bits |= 1u << k;
      }
    }
    if (!kBits) {
      /* BF16 1.0 = 0x3F80 */
      uint32_t w[2];
#pragma unroll
      for (int k = 0; k < 2; k++)
        w[k] = ((bits >> (2 * k)) & 1u) * 0x3F80u + ((bits >> (2 * k + 1)) & 1u) * 0x3F800000u;
      *reinterpret_cast<uint2*>(p.s_out + row + c0 + m) = make_uint2(w[0], w[1]);
    }
    if (p.count_on && bits) {
      uint32_t* c = reinterpret_cast<uint32_t*>(p.counts + row + c0 + m);
      uint32_t add = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) add |= ((bits >> k) & 1u) << (8 * k);
      *c = *c + add; /* no carry between bytes: at most 255 counted ticks between clears */
    }
    all |= bits << (4 * i);
  }
  if (kBits) {
    /* 16 spikes of the HCU per group index, the lane's four at 4 q */
#pragma unroll
    for (int i = 0; i < G; i++) {
      uint32_t v = ((all >> (4 * i)) & 15u) << (4 * q);
      v |= __shfl_xor_sync(0xffffffffu, v, 1);
      v |= __shfl_xor_sync(0xffffffffu, v, 2);
      if (q == 0) reinterpret_cast<uint16_t*>(p.s_bits)[(row + c0) / 16 + i] = (uint16_t)v;
    }
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int M, bool kBits>
__global__ void __launch_bounds__(256) recall_pop_kernel(Params p) {
  recall_pop<M, kBits>(p, blockIdx.x * 256 + threadIdx.x);
}

/* The output tiles of a launch: 128 x 256, or, where these are fewer than the
   SMs, column parts of 128, 64 or 32, as narrow as still gives every SM at most
   one.  A single tile (256 sources, 128 replicates) takes 8 CTAs of 32 columns
   instead of one: 24 -> 9.6 us, mostly its epilogue's loads; 32 tiles (N = R =
   1024) take 128 CTAs: 31 -> 17 us.  Cutting the last round of more tiles too
   makes the contraction shorter (512 tiles on 148 SMs: 158 -> 146 us in place),
   but not the tick (176, 178): the population update beside it is then what the
   tick waits for. */
struct Tiles {
  int n_n;   /* tiles across the columns */
  int whole; /* whole tiles, 0 .. whole - 1 */
  int parts; /* parts per tile from `whole` on */
  int total; /* whole tiles and parts */
  __host__ __device__ Tiles(int R, int N, int grid_max) {
    n_n = N / kTileN;
    const int n = n_n * (R / kTileM);
    whole = n / grid_max * grid_max;
    const int rest = n - whole;
    parts = 1;
    while (whole == 0 && parts < kMaxParts && 2 * parts * rest <= grid_max) parts *= 2;
    total = whole + rest * parts;
  }
  __device__ __forceinline__ void at(int t, int& m0, int& n0, int& cols) const {
    int tile = t, part = 0;
    cols = kTileN;
    if (t >= whole) {
      tile = whole + (t - whole) / parts;
      part = (t - whole) % parts;
      cols = kTileN / parts;
    }
    m0 = tile / n_n * kTileM;
    n0 = tile % n_n * kTileN + part * cols;
  }
};

/* W^T boxes of a tile's columns: whole, then halves, quarters and eighths */
struct WMaps {
  CUtensorMap of[kMaxPartsLog + 1];
};

/* Persistent contraction + epsc epilogue: one CTA per SM walks the tiles t =
   blockIdx.x, blockIdx.x + ctas, ... (Tiles).  The stage ring runs on
   across tiles; two TMEM accumulators of 256 columns alternate, so the epilogue
   of one tile overlaps the MMAs of the next (acc_full: MMA -> epilogue,
   acc_empty: epilogue -> MMA).  The epilogue loads the epsc of a tile's first 32
   columns before its accumulator is there.

   kPopM: the HCU size, and the CTAs from `ctas` on do the population update of
   the tick, which needs nothing of the contraction's; 0: recall_pop_kernel does
   it, on a stream of its own.  Where all of both find an SM each, one launch per
   tick costs less than two with the events between their streams, which the host
   takes longer to queue than the GPU to run, and a tick's launch, its barriers and
   its TMEM come beside the end of the tick before (programmatic launch; nothing
   that tick writes is touched before griddepcontrol.wait): 256 sources, 128
   replicates 9.5 -> 6.2 -> 4.2 us per tick. */
template <int kPopM>
__global__ void __launch_bounds__(kThreads, 1)
    recall_tick_kernel(const __grid_constant__ CUtensorMap map_s, const __grid_constant__ WMaps map_w, Params p,
                       int grid_max, int ctas) {
  if constexpr (kPopM > 0) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if ((int)blockIdx.x >= ctas) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const int tid = ((int)blockIdx.x - ctas) * kThreads + threadIdx.x;
      if (tid < p.R * p.H * 4) recall_pop<kPopM, false>(p, tid); /* whole warps: R is a multiple of 128 */
      return;
    }
  }
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;   /* [2] */
  uint64_t* acc_empty = acc_full + 2;     /* [2] */
  uint64_t* mma_done = acc_empty + 2;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(mma_done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Tiles tiles(p.R, p.N, grid_max);
  const int n_tiles = tiles.total;
  const int kIters = p.N / kTileK;
  const int part_log = tiles.parts == 1 ? 0 : tiles.parts == 2 ? 1 : tiles.parts == 4 ? 2 : 3;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int j = 0; j < 2; j++) {
      mbar_init(&acc_full[j], 1);
      mbar_init(&acc_empty[j], kEpiThreads);
    }
    mbar_init(mma_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  /* the set-up above ran beside the end of the tick before; all it wrote is there from here on */
  if constexpr (kPopM > 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tmem = *s_tmem;
  /* self-check of the set-up every access below relies on: ring and barrier
     alignment, the accumulators' TMEM columns, whole tiles */
  const bool setup_ok = (smem_u32(ring) & 1023u) == 0 && (smem_u32(full) & 7u) == 0 && (tmem >> 16) == 0 &&
                        (tmem & 0xFFFFu) + kTmemCols <= 512u && p.N % kTileN == 0 && p.R % kTileM == 0 &&
                        (reinterpret_cast<uintptr_t>(p.epsc_prev) & 15) == 0 &&
                        (reinterpret_cast<uintptr_t>(p.epsc_cur) & 15) == 0;
  if (!setup_ok && threadIdx.x == 0 && atomicOr(p.err, kErrAlign) == 0) p.err[1] = -1 - (int)blockIdx.x;

  if (setup_ok && warp == 0) {
    /* ---------------- TMA producer ---------------- */
    if (lane == 0) {
      long long it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += ctas) {
        int m0, n0, cols;
        tiles.at(t, m0, n0, cols);
        const CUtensorMap* w = &map_w.of[t < tiles.whole ? 0 : part_log];
        for (int k = 0; k < kIters; k++, it++) {
          const int s = (int)(it % kStages);
          if (!mbar_wait(&empty[s], (uint32_t)(((it / kStages) & 1) ^ 1), p.err)) {
            ok = false;
            break;
          }
          uint8_t* a = ring + s * kStageBytes;
          mbar_expect_tx(&full[s], kBytesA + (uint32_t)cols * kTileK * 2);
          tma_load_2d(a, &map_s, &full[s], k * kTileK, m0);
          tma_load_2d(a + kBytesA, w, &full[s], k * kTileK, n0);
        }
      }
      /* leave no copy in flight: the last use of every slot completes */
      for (long long j = (it > kStages ? it - kStages : 0); j < it; j++) {
        unsigned long long t0 = gtimer();
        while (!mbar_try_wait(&full[j % kStages], (uint32_t)((j / kStages) & 1)) && gtimer() - t0 < kWaitNs) {
        }
      }
    }
  } else if (setup_ok && warp == 1) {
    /* ---------------- MMA issuer ---------------- */
    if (lane == 0) {
      long long it = 0;
      bool ok = true;
      int li = 0;
      for (int t = blockIdx.x; t < n_tiles && ok; t += ctas, li++) {
        const int j = li & 1;
        if (!mbar_wait(&acc_empty[j], (uint32_t)(((li >> 1) & 1) ^ 1), p.err)) break;
        tc_fence_after();
        const uint32_t acc = tmem + (uint32_t)(j * kTileN);
        int m0, n0, cols;
        tiles.at(t, m0, n0, cols);
        const uint32_t idesc = umma_idesc(cols);
        for (int k = 0; k < kIters; k++, it++) {
          const int s = (int)(it % kStages);
          if (!mbar_wait(&full[s], (uint32_t)((it / kStages) & 1), p.err)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a = smem_u32(ring + s * kStageBytes);
          const uint32_t b = a + kBytesA;
#pragma unroll
          for (int kk = 0; kk < kTileK / kUmmaK; kk++) {
            /* +32 bytes along K inside the 128-byte swizzled row */
            umma(acc, smem_desc(a + kk * 32), smem_desc(b + kk * 32), idesc, (k > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&acc_full[j]);
      }
    }
  } else if (setup_ok) {
    /* ---------------- epilogue: one replicate row per thread ---------------- */
    const int q = warp & 3; /* TMEM lane quarter this warp may access */
    int li = 0;
    for (int t = blockIdx.x; t < n_tiles; t += ctas, li++) {
      const int j = li & 1;
      int m0, n0, cols;
      tiles.at(t, m0, n0, cols);
      const int row = m0 + q * 32 + lane;
      const size_t base = (size_t)row * p.N + n0;
      float4 e[8];
#pragma unroll
      for (int i = 0; i < 8; i++) e[i] = *reinterpret_cast<const float4*>(p.epsc_prev + base + 4 * i);
      /* warp-uniform: tcgen05.ld is .sync.aligned */
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[j], (uint32_t)((li >> 1) & 1), p.err) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after();
      for (int c = 0; c < cols; c += 32) {
        float acc[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(j * kTileN + c), acc);
        if (c > 0) {
#pragma unroll
          for (int i = 0; i < 8; i++) e[i] = *reinterpret_cast<const float4*>(p.epsc_prev + base + c + 4 * i);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
          float4 o;
          o.x = e[i].x * p.one_m_kepsc + acc[4 * i];
          o.y = e[i].y * p.one_m_kepsc + acc[4 * i + 1];
          o.z = e[i].z * p.one_m_kepsc + acc[4 * i + 2];
          o.w = e[i].w * p.one_m_kepsc + acc[4 * i + 3];
          *reinterpret_cast<float4*>(p.epsc_cur + base + c + 4 * i) = o;
        }
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[j]);
    }
  }
  /* every tcgen05 operation of this CTA completes before TMEM is freed: the
     MMA thread's last commit (all MMAs it issued) is waited for, bounded */
  if (warp == 1 && lane == 0) {
    umma_commit(mma_done);
    unsigned long long t0 = gtimer();
    while (!mbar_try_wait(mma_done, 0) && gtimer() - t0 < kWaitNs) {
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

using TickFn = void (*)(CUtensorMap, WMaps, Params, int, int);

constexpr int kF32BM = 128, kF32BN = 128, kF32BK = 16, kF32Threads = 256;

/* FP32 SIMT contraction with the epsc epilogue of recall_tick_kernel:
   epsc(t)[r][j] = epsc(t-1)[r][j] * (1 - kepsc) + sum_i S(t-3)[r][i] * W[i][j]
   with W in FP32 ([source i][destination j], row-major) and S the 0/1 spike
   bits.  The dense form: it multiplies every weight, so it is taken only where
   recall_events_kernel is not (see bcpnn_recall_run).

   One CTA per 128 x 128 output tile (blockIdx.x = M-tile * (N/128) + N-tile);
   thread (ty, tx) = (tid / 16, tid % 16) owns rows {ty*4 .. +3, 64 + ty*4 ..
   +3} and columns {tx*4 .. +3, 64 + tx*4 .. +3} of the tile, 64 FP32
   accumulators.  K stages of 16: S as [k][row] and W as [k][col] in shared
   memory, two buffers, the next stage's global loads held in registers while
   the current one is multiplied, one barrier per stage. */
__global__ void __launch_bounds__(kF32Threads, 2)
    recall_fp32_kernel(const uint32_t* __restrict__ s, const float* __restrict__ w, Params p) {
  __shared__ __align__(16) float As[2][kF32BK][kF32BM];
  __shared__ __align__(16) float Bs[2][kF32BK][kF32BN];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int nN = p.N / kF32BN, nM = p.R / kF32BM;
  const int m0 = ((int)blockIdx.x / nN) * kF32BM, n0 = ((int)blockIdx.x % nN) * kF32BN;
  /* self-check: whole tiles, the tile inside the arrays, 16-byte alignment of
     every vector access */
  {
    const bool bad = p.N % kF32BN != 0 || p.R % kF32BM != 0 || (int)blockIdx.x >= nN * nM ||
                     (reinterpret_cast<uintptr_t>(s) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) ||
                     (reinterpret_cast<uintptr_t>(p.epsc_prev) & 15) ||
                     (reinterpret_cast<uintptr_t>(p.epsc_cur) & 15);
    if (bad) {
      if (tid == 0 && atomicOr(p.err, kErrAlign) == 0) p.err[1] = -1 - (int)blockIdx.x;
      return;
    }
  }
  /* S stage: row a_row, eight spike bits at a_k (one byte); W stage: row b_k,
     eight floats at b_n (two 16-byte loads) */
  const int a_row = tid & 127, a_k = (tid >> 7) * 8;
  const int b_k = tid >> 4, b_n = (tid & 15) * 8;
  const uint8_t* ag = reinterpret_cast<const uint8_t*>(s) + ((size_t)(m0 + a_row) * p.N + a_k) / 8;
  const float* bg = w + (size_t)b_k * p.N + n0 + b_n;
  const size_t b_step = (size_t)kF32BK * p.N;
  uint32_t ra = __ldg(ag);
  float4 rb0 = __ldg(reinterpret_cast<const float4*>(bg));
  float4 rb1 = __ldg(reinterpret_cast<const float4*>(bg + 4));
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;

  auto stage = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 8; j++) As[buf][a_k + j][a_row] = (ra >> j) & 1u ? 1.0f : 0.0f;
    *reinterpret_cast<float4*>(&Bs[buf][b_k][b_n]) = rb0;
    *reinterpret_cast<float4*>(&Bs[buf][b_k][b_n + 4]) = rb1;
  };
  stage(0);
  __syncthreads();
  const int kTiles = p.N / kF32BK;
  for (int kt = 0; kt < kTiles; kt++) {
    const int buf = kt & 1;
    if (kt + 1 < kTiles) {
      ra = __ldg(ag + (size_t)(kt + 1) * (kF32BK / 8));
      const float* b = bg + (size_t)(kt + 1) * b_step;
      rb0 = __ldg(reinterpret_cast<const float4*>(b));
      rb1 = __ldg(reinterpret_cast<const float4*>(b + 4));
    }
#pragma unroll
    for (int k = 0; k < kF32BK; k++) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][k][64 + ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][k][tx * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&Bs[buf][k][64 + tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    /* the other buffer was last read in stage kt-1, before the barrier
       that ended it */
    if (kt + 1 < kTiles) stage(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int row = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const size_t o = (size_t)row * p.N + n0 + h * 64 + tx * 4;
      const float4 e = *reinterpret_cast<const float4*>(p.epsc_prev + o);
      float4 v;
      v.x = e.x * p.one_m_kepsc + acc[i][h * 4 + 0];
      v.y = e.y * p.one_m_kepsc + acc[i][h * 4 + 1];
      v.z = e.z * p.one_m_kepsc + acc[i][h * 4 + 2];
      v.w = e.w * p.one_m_kepsc + acc[i][h * 4 + 3];
      *reinterpret_cast<float4*>(p.epsc_cur + o) = v;
    }
  }
}

/* ---- FP32 contraction by events ------------------------------------------

   Each output adds the rows of W of the sources that spiked, in ascending
   source order from 0:
     epsc(t)[r][j] = epsc(t-1)[r][j] * (1 - kepsc) + (((W[i0][j] + W[i1][j]) + W[i2][j]) + ...)
   The multiply-adds of recall_fp32_kernel do the same additions in the same
   order, and fma(0, w, acc) = acc for a finite w, so both give the same bits;
   at the 1 spike in 50 sources of a recall the dense form does 50 times the
   work.

   Bound by the shared-memory reads of W: 4 bytes per spike and destination
   (128 bytes per SM and cycle).  A CTA (one per SM) takes a run of (column
   tile of 64, replicate) pairs, the same number in every CTA; 15 warps hold
   up to 24 replicates each, two columns per lane, in registers (48
   accumulators a lane), so a chunk of W serves 360 replicates once it is in
   shared memory.  W comes in chunks of 384 sources x 64 columns (TMA, two
   buffers, issued by a warp of its own); a warp reads a row of a chunk as 256
   contiguous bytes, without bank conflicts, for any spike pattern.  The
   spikes of a replicate and chunk come as a list of 16-bit source numbers
   (recall_lists_kernel), padded to a multiple of four with the number of a
   row of zeros (the sum is never -0, so adding +0 leaves it as it is), read
   four at a time with all lanes on the same replicate.  The replicates are
   walked in groups of eight whose accumulators rotate through the registers:
   one unrolled body for all 24 replicates is more code than the instruction
   caches hold.  A replicate with more than kEvCap spikes in a chunk is listed
   from its bits by the warp that needs it (walk_bits).

   At N = R = 4096, M = 64 and 20 Hz noise (2.2 % of the sources spike): 345 us
   a launch, 2815 us dense.  8.2 us are added per 0.1 % of density, of which
   the weights' reads are 8.0 at 128 bytes per SM and cycle; 184 us remain
   without spikes: per replicate and chunk the count, the loop and the padding,
   per pass the epilogue.  W's chunks alone would take 88 us and come in
   beside.  24 replicates in 15 warps were the best of 8 x 31, 16 x 19, 16 x
   23, 24 x 15 and 32 x 15; eight list entries per step were slower than four
   (435 us). */
constexpr int kEvCols = 64, kEvRows = 384, kEvBox = 192, kEvWarps = 15, kEvThreads = (kEvWarps + 1) * 32;
constexpr int kEvReps = 24;          /* replicates per warp and pass */
constexpr int kEvGroup = 8;          /* replicates of one unrolled body */
constexpr int kEvCap = 32;           /* listed spikes per replicate and chunk */
constexpr int kEvListWords = kEvCap / 2;
/* the expected share of sources spiking above which the dense kernel is the
   faster one: 2777 us by events at 0.2 (2815 us dense), 3169 us at 0.24 */
constexpr float kEvMaxDensity = 0.2f;
constexpr int kEvWords = kEvRows / 32;
constexpr uint32_t kEvRowBytes = kEvCols * 4;
constexpr uint32_t kEvChunkBytes = kEvRows * kEvRowBytes;
constexpr uint32_t kEvBufBytes = kEvChunkBytes + kEvRowBytes; /* and the row of zeros */
constexpr uint32_t kEvScratch = (kEvRows + 8) * 2; /* a warp's list of one replicate (walk_bits) */
/* the warps' lists, their scratch lists, their counts */
constexpr uint32_t kEvListBytes = kEvWarps * (kEvReps * (kEvListWords * 4 + 1) + kEvScratch);
constexpr size_t kEvSmemBytes = 2 * kEvBufBytes + kEvListBytes + 4 * sizeof(uint64_t);
static_assert(kEvReps % kEvGroup == 0 && kEvGroup == 8, "a group's counts are one 8-byte read");
static_assert(kEvReps * kEvListWords % 128 == 0, "a warp's lists are whole 16-byte words per lane");
static_assert(kEvScratch % 8 == 0 && kEvListBytes % 8 == 0 && kEvBufBytes % 128 == 0, "shared memory alignment");
static_assert(kEvWords % 4 == 0 && kEvWords <= 16, "walk_bits gives a word to each of at most 16 lanes");
static_assert(kEvSmemBytes <= 232448, "shared memory of one CTA");

/* byte offset, in a chunk of 256-byte rows, of the lane's columns of the row
   of a 16-bit list entry; lane8 = 8 * lane is the low byte */
__device__ __forceinline__ uint32_t ev_row0(uint32_t two, uint32_t lane8) { return __byte_perm(two, lane8, 0x7104); }
__device__ __forceinline__ uint32_t ev_row1(uint32_t two, uint32_t lane8) { return __byte_perm(two, lane8, 0x7324); }

__device__ __forceinline__ unsigned long long lds64(uint32_t a) {
  unsigned long long v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}

__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

/* the spike lists of one tick, [chunk][replicate][kEvCap], and their counts,
   [chunk][replicate]: one thread per list; the sources of the chunk that
   spiked, ascending, padded with row kEvRows (count: kEvCap + 1 if more) */
__global__ void __launch_bounds__(256) recall_lists_kernel(const uint32_t* __restrict__ bits, uint4* __restrict__ lists,
                                                           uint8_t* __restrict__ counts, int R, int N) {
  __shared__ uint16_t buf[256][kEvCap + 2]; /* 17 words a row: no bank conflicts */
  const int W32 = N / 32;
  const long long n = (long long)R * ((N + kEvRows - 1) / kEvRows);
  const long long x = (long long)blockIdx.x * 256 + threadIdx.x;
  uint16_t* mine = buf[threadIdx.x];
  if (x < n) {
    const int c = (int)(x / R), r = (int)(x - (long long)c * R);
    const uint32_t* b = bits + (size_t)r * W32 + c * kEvWords;
    const int nw = min(kEvWords, W32 - c * kEvWords);
    int cnt = 0;
    for (int v = 0; v < nw; v++) {
      uint32_t w = __ldg(b + v);
      while (w) {
        const int k = __ffs(w) - 1;
        w &= w - 1;
        if (cnt < kEvCap) mine[cnt] = (uint16_t)(v * 32 + k);
        cnt++;
      }
    }
    for (int k = cnt; k < kEvCap; k++) mine[k] = (uint16_t)kEvRows;
    counts[x] = (uint8_t)(cnt <= kEvCap ? cnt : kEvCap + 1);
  }
  __syncthreads();
  /* the block's lists are contiguous */
  uint32_t* out = reinterpret_cast<uint32_t*>(lists) + (size_t)blockIdx.x * 256 * kEvListWords;
  const long long left = n - (long long)blockIdx.x * 256;
  const int words = (int)(left < 256 ? left : 256) * kEvListWords;
  for (int k = threadIdx.x; k < words; k += 256)
    out[k] = reinterpret_cast<const uint32_t*>(buf[k / kEvListWords])[k % kEvListWords];
}

/* a replicate with more than kEvCap spikes in a chunk: its nw words of bits
   (global memory) listed in the warp's scratch (kEvRows + 4 entries at byte
   address l), padded to a multiple of four with row kEvRows, and their rows
   added to acc as from a list of its own */
__device__ __noinline__ unsigned long long walk_bits(unsigned long long acc, const uint32_t* words, int nw, uint32_t l,
                                                     uint32_t w0, uint32_t lane8) {
  const int lane = (int)lane8 >> 3;
  uint32_t w = lane < nw ? __ldg(words + lane) : 0u;
  int at = __popc(w);
  const int own = at;
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += y;
  }
  const int n = __shfl_sync(0xffffffffu, at, 15); /* kEvWords <= 16 lanes hold words */
  uint32_t d = l + 2 * (uint32_t)(at - own);
  while (w) {
    const int b = __ffs(w) - 1;
    w &= w - 1;
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(d), "h"((unsigned short)(lane * 32 + b)) : "memory");
    d += 2;
  }
  if (lane < 4)
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(l + 2 * (uint32_t)(n + lane)), "h"((unsigned short)kEvRows) : "memory");
  __syncwarp();
#pragma unroll 1
  for (const uint32_t end = l + 2 * (uint32_t)n; l < end; l += 8) {
    const unsigned long long x = lds64(l);
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    const unsigned long long v0 = lds64(w0 + ev_row0(x0, lane8)), v1 = lds64(w0 + ev_row1(x0, lane8));
    const unsigned long long v2 = lds64(w0 + ev_row0(x1, lane8)), v3 = lds64(w0 + ev_row1(x1, lane8));
    acc = add2(add2(add2(add2(acc, v0), v1), v2), v3);
  }
  __syncwarp();
  return acc;
}

/* the passes of one CTA: (column tile, replicates [a, e)) for its run of pairs */
struct EvPass {
  long long pair, end;
  int R, tile, a, e, seg_r0, seg_len, npass, k;
  __device__ __forceinline__ void init(long long p0, long long p1, int R_) {
    pair = p0;
    end = p1;
    R = R_;
    npass = k = 0;
  }
  __device__ __forceinline__ bool next() {
    if (k == npass) {
      if (pair >= end) return false;
      tile = (int)(pair / R);
      seg_r0 = (int)(pair - (long long)tile * R);
      const long long left = end - pair;
      seg_len = left < R - seg_r0 ? (int)left : R - seg_r0;
      npass = (seg_len + kEvWarps * kEvReps - 1) / (kEvWarps * kEvReps);
      pair += seg_len;
      k = 0;
    }
    a = seg_r0 + (int)((long long)seg_len * k / npass);
    e = seg_r0 + (int)((long long)seg_len * (k + 1) / npass);
    k++;
    return true;
  }
};

__global__ void __launch_bounds__(kEvThreads, 1)
    recall_events_kernel(const __grid_constant__ CUtensorMap map_w, const uint32_t* __restrict__ bits,
                         const uint4* __restrict__ lists, const uint8_t* __restrict__ counts, Params p) {
  extern __shared__ __align__(128) uint8_t ev_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(ev_smem + 2 * kEvBufBytes + kEvListBytes);
  uint64_t* empty = full + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N, W32 = N / 32, n_chunks = (N + kEvRows - 1) / kEvRows;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kEvWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 2 * kEvCols)
    reinterpret_cast<float*>(ev_smem + (threadIdx.x / kEvCols) * kEvBufBytes + kEvChunkBytes)[threadIdx.x % kEvCols] = 0.0f;
  __syncthreads();
  /* self-check: whole column tiles, alignment of the ring and of every vector access */
  const bool ok0 = N % kEvCols == 0 && W32 % 4 == 0 && (smem_u32(ev_smem) & 127u) == 0 &&
                   (reinterpret_cast<uintptr_t>(lists) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.epsc_prev) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(p.epsc_cur) & 15) == 0;
  if (!ok0) {
    if (threadIdx.x == 0 && atomicOr(p.err, kErrAlign) == 0) p.err[1] = -1 - (int)blockIdx.x;
    return;
  }
  const long long T = (long long)(N / kEvCols) * p.R;
  EvPass ps;
  ps.init(T * blockIdx.x / gridDim.x, T * (blockIdx.x + 1) / gridDim.x, p.R);
  uint32_t it = 0; /* chunks so far: buffer it & 1, phase (it >> 1) & 1 */

  if (warp == kEvWarps) {
    if (lane == 0) {
      bool ok = true;
      while (ok && ps.next()) {
        for (int c = 0; c < n_chunks; c++, it++) {
          const uint32_t s = it & 1;
          if (!mbar_wait(&empty[s], ((it >> 1) & 1) ^ 1, p.err)) {
            ok = false;
            break;
          }
          uint8_t* dst = ev_smem + s * kEvBufBytes;
          const int row = c * kEvRows;
          const bool two = row + kEvBox < N; /* no box starts past the last row */
          mbar_expect_tx(&full[s], two ? kEvChunkBytes : kEvChunkBytes / 2);
          tma_load_2d(dst, &map_w, &full[s], ps.tile * kEvCols, row);
          if (two) tma_load_2d(dst + kEvBox * kEvRowBytes, &map_w, &full[s], ps.tile * kEvCols, row + kEvBox);
        }
      }
      /* leave no copy in flight */
      for (uint32_t j = (it > 2 ? it - 2 : 0); j < it; j++) {
        const unsigned long long t0 = gtimer();
        while (!mbar_try_wait(&full[j & 1], (j >> 1) & 1) && gtimer() - t0 < kWaitNs) {
        }
      }
    }
    return;
  }

  uint8_t* const my_lists = ev_smem + 2 * kEvBufBytes + warp * (kEvReps * kEvListWords * 4);
  uint8_t* const my_scratch = ev_smem + 2 * kEvBufBytes + kEvWarps * kEvReps * kEvListWords * 4 + warp * kEvScratch;
  uint8_t* const my_counts =
      ev_smem + 2 * kEvBufBytes + kEvWarps * (kEvReps * kEvListWords * 4 + kEvScratch) + warp * kEvReps;
  const uint32_t scratch_a = smem_u32(my_scratch);
  const uint32_t lists_a = smem_u32(my_lists), counts_a = smem_u32(my_counts), lane8 = (uint32_t)lane * 8;
  while (ps.next()) {
    const int q = (ps.e - ps.a + kEvWarps - 1) / kEvWarps;
    const int r0 = ps.a + warp * q;
    const int nr = max(0, min(q, ps.e - r0)); /* this warp's replicates */
    unsigned long long acc[kEvReps]; /* two columns each */
#pragma unroll
    for (int i = 0; i < kEvReps; i++) acc[i] = 0ull;
    /* the warp's lists of a chunk, contiguous: a few 16-byte words per lane, one chunk ahead */
    constexpr int kListLoads = kEvReps * (kEvListWords / 4) / 32;
    uint4 b[kListLoads];
    uint8_t bc = 0; /* lists of no replicate: count 0 */
    auto fetch = [&](int c) {
      const uint4* src = lists + ((size_t)c * p.R + r0) * (kEvListWords / 4);
#pragma unroll
      for (int v = 0; v < kListLoads; v++)
        if (lane + 32 * v < nr * (kEvListWords / 4)) b[v] = __ldg(src + lane + 32 * v);
      if (lane < nr) bc = __ldg(counts + (size_t)c * p.R + r0 + lane);
    };
    fetch(0);
    for (int c = 0; c < n_chunks; c++, it++) {
#pragma unroll
      for (int v = 0; v < kListLoads; v++)
        if (lane + 32 * v < nr * (kEvListWords / 4)) *reinterpret_cast<uint4*>(my_lists + (lane + 32 * v) * 16) = b[v];
      if (lane < kEvReps) my_counts[lane] = bc;
      __syncwarp();
      if (c + 1 < n_chunks) fetch(c + 1);
      const uint32_t s = it & 1;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (it >> 1) & 1, p.err) ? 1 : 0) != 0;
      if (!ok) return;
      const uint32_t w0 = smem_u32(ev_smem) + s * kEvBufBytes;
      uint32_t l = lists_a;
      /* groups of replicates: after each, the accumulators rotate by one group */
#pragma unroll 1
      for (int g = 0; g < kEvReps; g += kEvGroup) {
        const unsigned long long cnts = lds64(counts_a + g);
        unsigned long long xn = lds64(l);
#pragma unroll
        for (int i = 0; i < kEvGroup; i++, l += kEvListWords * 4) {
          const uint32_t cnt = (uint32_t)(cnts >> (8 * i)) & 0xffu;
          unsigned long long x = xn;
          if (i + 1 < kEvGroup) xn = lds64(l + kEvListWords * 4);
          if (cnt <= kEvCap) {
            unsigned long long a = acc[i];
            const uint32_t end = l + 2 * cnt;
            uint32_t e = l;
#pragma unroll 1
            while (e < end) {
              const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
              const unsigned long long v0 = lds64(w0 + ev_row0(x0, lane8)), v1 = lds64(w0 + ev_row1(x0, lane8));
              const unsigned long long v2 = lds64(w0 + ev_row0(x1, lane8)), v3 = lds64(w0 + ev_row1(x1, lane8));
              e += 8;
              x = lds64(e);
              a = add2(add2(add2(add2(a, v0), v1), v2), v3);
            }
            acc[i] = a;
          } else {
            const int w = c * kEvWords;
            acc[i] = walk_bits(acc[i], bits + (size_t)(r0 + g + i) * W32 + w, min(kEvWords, W32 - w), scratch_a, w0,
                               lane8);
          }
        }
        unsigned long long t[kEvGroup];
#pragma unroll
        for (int i = 0; i < kEvGroup; i++) t[i] = acc[i];
#pragma unroll
        for (int i = 0; i < kEvReps - kEvGroup; i++) acc[i] = acc[i + kEvGroup];
#pragma unroll
        for (int i = 0; i < kEvGroup; i++) acc[kEvReps - kEvGroup + i] = t[i];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    /* epilogue: 256 contiguous bytes per replicate row and warp, four rows' loads at a time */
    const size_t col = (size_t)ps.tile * kEvCols + 2 * lane;
#pragma unroll
    for (int i0 = 0; i0 < kEvReps; i0 += 4) {
      if (i0 >= nr) break;
      float2 ev[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i0 + i < nr) ev[i] = *reinterpret_cast<const float2*>(p.epsc_prev + (size_t)(r0 + i0 + i) * N + col);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i0 + i < nr) {
          float2 o;
          o.x = ev[i].x * p.one_m_kepsc + __uint_as_float((uint32_t)acc[i0 + i]);
          o.y = ev[i].y * p.one_m_kepsc + __uint_as_float((uint32_t)(acc[i0 + i] >> 32));
          *reinterpret_cast<float2*>(p.epsc_cur + (size_t)(r0 + i0 + i) * N + col) = o;
        }
    }
  }
}

/* sets *flag when a weight is infinite or NaN: 0 * w is then not 0, and only
   the dense contraction gives what the products give */
__global__ void nonfinite_kernel(const float* w, size_t n, int* flag) {
  bool bad = false;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    bad |= !(fabsf(w[i]) <= 3.402823466e38f);
  if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 1;
}

/* one row of spikes to every replicate's row of bits */
__global__ void broadcast_bits_kernel(uint32_t* s, int R, int N, const int8_t* row) {
  const int W32 = N / 32;
  const size_t n = (size_t)R * W32;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int8_t* x = row + (i % W32) * 32;
    uint32_t w = 0;
    for (int k = 0; k < 32; k++) w |= (x[k] ? 1u : 0u) << k;
    s[i] = w;
  }
}

__global__ void broadcast_spikes_kernel(uint16_t* s, int R, int N, const int8_t* row) {
  size_t n = (size_t)R * N;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    s[i] = row[i % N] ? 0x3F80u : 0u;
}

__global__ void broadcast_f32_kernel(float* dst, int R, int N, const float* row) {
  size_t n = (size_t)R * N;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = row[i % N];
}

}  // namespace bcpnn_recall_dev

using namespace bcpnn_recall_dev;

struct bcpnn_recall {
  host_copy::Users copies;
  bcpnn_recall_desc d;
  int N = 0;
  cudaStream_t stream = nullptr;      /* contraction + epsc; the handle's stream */
  cudaStream_t pop_stream = nullptr;  /* population update, concurrent with it */
  cudaEvent_t ev_pop = nullptr, ev_gemm = nullptr;
  float* dsup[2] = {nullptr, nullptr};
  float* epsc[2] = {nullptr, nullptr};
  uint16_t* s[4] = {nullptr, nullptr, nullptr, nullptr}; /* spike ring, by tick mod 4 (BF16 contraction) */
  uint32_t* sb[4] = {nullptr, nullptr, nullptr, nullptr}; /* the same as bits [R][N/32] (FP32 contraction) */
  uint16_t* wt = nullptr; /* W^T BF16 [N][N] (BF16 contraction) */
  float* wf = nullptr;    /* W FP32 [N][N], [source][destination] (FP32 contraction) */
  uint8_t* counts = nullptr;
  float* bj = nullptr;
  int32_t* lgidx = nullptr;
  float* wmask = nullptr;
  int* err = nullptr;
  float lg_hit = 0.f, lg_miss = 0.f;
  bool loaded = false, cued = false;
  long long kk = 0; /* ticks run since load */
  int counted = 0;   /* counted ticks since the counters were cleared */
  CUtensorMap map_s[4];
  WMaps map_w;           /* BF16: boxes of a tile's columns and of its parts */
  CUtensorMap map_wf;    /* FP32: boxes of the event kernel */
  uint4* lists[2] = {nullptr, nullptr}; /* spike lists of a tick, by tick parity (recall_lists_kernel) */
  uint8_t* list_cnt[2] = {nullptr, nullptr};
  bool finite_w = false; /* FP32 contraction: every loaded weight is finite */
  uint64_t launches = 0;
  int sms = 148;
  /* in-place timing of the contraction launches (bcpnn_recall_timing) */
  bool timing = false;
  std::vector<cudaEvent_t> tev;
  double contraction_ms = 0.0;
  uint64_t contraction_launches = 0;
  std::string last_error;
  std::vector<void*> allocs;
};

namespace {

int fail(bcpnn_recall* r, int code, const std::string& msg) {
  if (r) r->last_error = msg;
  return code;
}

#define RCU(call)                                                                             \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) {                                                                  \
      cudaGetLastError(); /* reported once, see CU (bcpnn_capi.cu) */                         \
      return fail(r, BCPNN_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));     \
    }                                                                                         \
  } while (0)

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

/* tensor map over a row-major [rows][cols] matrix: BF16 in 128-byte swizzled
   boxes of kTileK columns, or FP32 (f32) in plain boxes of kEvCols columns */
int encode_map(bcpnn_recall* r, CUtensorMap* map, void* base, int rows, int cols, int box_rows, bool f32 = false) {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    RCU(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p) return fail(r, BCPNN_ERR_CUDA, "cuTensorMapEncodeTiled not available");
    fn = (EncodeTiled)p;
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * (f32 ? 4 : 2)};
  cuuint32_t box[2] = {(cuuint32_t)(f32 ? kEvCols : kTileK), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult e = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  f32 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (e != CUDA_SUCCESS) return fail(r, BCPNN_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)e));
  return BCPNN_OK;
}

template <typename T>
int dalloc(bcpnn_recall* r, T** p, size_t count) {
  *p = nullptr;
  RCU(cudaMalloc((void**)p, (count ? count : 1) * sizeof(T)));
  r->allocs.push_back((void*)*p);
  return BCPNN_OK;
}

/* a copy to the device, on the handle's stream and complete on return (not
   cudaMemcpy: its stream is not ordered with the handle's) */
cudaError_t upload(bcpnn_recall* r, void* dst, const void* src, size_t bytes) {
  const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, r->stream);
  return e == cudaSuccess ? cudaStreamSynchronize(r->stream) : e;
}

uint16_t to_bf16(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7F800000u) == 0x7F800000u) return (uint16_t)((u >> 16) | ((u & 0xFFFFu) ? 0x40u : 0u));
  u += 0x7FFFu + ((u >> 16) & 1u); /* round to nearest even */
  return (uint16_t)(u >> 16);
}

int check_err(bcpnn_recall* r) {
  int e[2] = {0, 0};
  RCU(cudaMemcpyAsync(e, r->err, sizeof(e), cudaMemcpyDeviceToHost, r->stream));
  RCU(cudaStreamSynchronize(r->stream));
  if (e[0]) {
    RCU(cudaMemsetAsync(r->err, 0, sizeof(e), r->stream));
    std::string why;
    if (e[0] & kErrWait) why += " an mbarrier wait timed out;";
    if (e[0] & kErrAlign) why += " a self-check skipped a misaligned or out-of-range access (thread " + std::to_string(e[1]) + ");";
    return fail(r, BCPNN_ERR_DEVICE, "recall kernel reported error word " + std::to_string(e[0]) + ":" + why);
  }
  return BCPNN_OK;
}

int mod4(long long v) { return (int)(v & 3); }

}  // namespace

extern "C" {

int bcpnn_recall_create(const bcpnn_recall_desc* d, bcpnn_recall** out) {
  if (!d || !out) return BCPNN_ERR_INVALID;
  *out = nullptr;
  const int H = d->hcu_num, M = d->mcu_num, R = d->replicates;
  if (H < 1 || M < 1 || R < kTileM || R % kTileM) return BCPNN_ERR_INVALID;
  const long long N = (long long)H * M;
  if (N % kTileN || kTileN % M || (M != 16 && M != 32 && M != 64) || N > 65536) return BCPNN_ERR_INVALID;
  if (!(d->dt > 0.f) || !(d->pop.taum > 0.f) || d->poisson_noise_hz < 0.f) return BCPNN_ERR_INVALID;
  if (d->contraction != BCPNN_RECALL_BF16 && d->contraction != BCPNN_RECALL_FP32) return BCPNN_ERR_INVALID;
  const bool fp32 = d->contraction == BCPNN_RECALL_FP32;
  bcpnn_recall* r = new bcpnn_recall();
  r->d = *d;
  r->N = (int)N;
  auto bad = [&](int rc) {
    if (rc == BCPNN_ERR_CUDA) cudaGetLastError(); /* reported here, see CU (bcpnn_capi.cu) */
    bcpnn_recall_destroy(r);
    return rc;
  };
  if (cudaSetDevice(d->device) != cudaSuccess) return bad(BCPNN_ERR_CUDA);
  int major = 0, minor = 0;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, d->device);
  cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, d->device);
  if (major != 10 || minor != 0) return bad(BCPNN_ERR_DEVICE);
  cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, d->device);
  if (r->sms < 1) r->sms = 1;
  /* the contraction's stream first in the block scheduler's order: its CTAs
     (one per SM) take their SMs before the population update fills the rest */
  int prio_low = 0, prio_high = 0;
  cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
  if (cudaStreamCreateWithPriority(&r->stream, cudaStreamNonBlocking, prio_high) != cudaSuccess)
    return bad(BCPNN_ERR_CUDA);
  size_t RN = (size_t)R * N;
  int rc = BCPNN_OK;
  for (int i = 0; i < 2 && !rc; i++) rc = dalloc(r, &r->dsup[i], RN);
  for (int i = 0; i < 2 && !rc; i++) rc = dalloc(r, &r->epsc[i], RN);
  for (int i = 0; i < 4 && !rc; i++) rc = fp32 ? dalloc(r, &r->sb[i], RN / 32) : dalloc(r, &r->s[i], RN);
  if (!rc && !fp32) rc = dalloc(r, &r->wt, (size_t)N * N);
  if (!rc && fp32) rc = dalloc(r, &r->wf, (size_t)N * N);
  if (!rc) rc = dalloc(r, &r->counts, RN);
  if (!rc) rc = dalloc(r, &r->bj, (size_t)N);
  if (!rc) rc = dalloc(r, &r->lgidx, (size_t)R * H);
  if (!rc) rc = dalloc(r, &r->wmask, (size_t)R * H);
  if (!rc) rc = dalloc(r, &r->err, 4);
  if (rc) return bad(rc);
  if (cudaMemsetAsync(r->err, 0, 4 * sizeof(int), r->stream) != cudaSuccess ||
      cudaMemsetAsync(r->counts, 0, RN, r->stream) != cudaSuccess)
    return bad(BCPNN_ERR_CUDA);
  if (!fp32) {
    for (int i = 0; i < 4 && !rc; i++) rc = encode_map(r, &r->map_s[i], r->s[i], R, (int)N, kTileM);
    for (int i = 0; i <= kMaxPartsLog && !rc; i++) rc = encode_map(r, &r->map_w.of[i], r->wt, (int)N, (int)N, kTileN >> i);
    if (rc) return bad(rc);
    for (TickFn f : {recall_tick_kernel<0>, recall_tick_kernel<16>, recall_tick_kernel<32>, recall_tick_kernel<64>})
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) != cudaSuccess)
        return bad(BCPNN_ERR_CUDA);
  } else {
    if ((rc = encode_map(r, &r->map_wf, r->wf, (int)N, (int)N, kEvBox, true))) return bad(rc);
    for (int i = 0; i < 2; i++)
      if ((rc = dalloc(r, &r->lists[i], (size_t)R * ((N + kEvRows - 1) / kEvRows) * (kEvListWords / 4))) ||
          (rc = dalloc(r, &r->list_cnt[i], (size_t)R * ((N + kEvRows - 1) / kEvRows))))
        return bad(rc);
    if (cudaFuncSetAttribute(recall_events_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEvSmemBytes) !=
        cudaSuccess)
      return bad(BCPNN_ERR_CUDA);
  }
  if (cudaStreamCreateWithPriority(&r->pop_stream, cudaStreamNonBlocking, prio_low) != cudaSuccess ||
      cudaEventCreateWithFlags(&r->ev_pop, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&r->ev_gemm, cudaEventDisableTiming) != cudaSuccess)
    return bad(BCPNN_ERR_CUDA);
  *out = r;
  return BCPNN_OK;
}

int bcpnn_recall_destroy(bcpnn_recall* r) {
  if (!r) return BCPNN_ERR_INVALID;
  cudaSetDevice(r->d.device);
  if (r->stream) cudaStreamSynchronize(r->stream);
  if (r->pop_stream) cudaStreamSynchronize(r->pop_stream);
  for (void* p : r->allocs) cudaFree(p);
  for (cudaEvent_t e : r->tev) cudaEventDestroy(e);
  if (r->ev_pop) cudaEventDestroy(r->ev_pop);
  if (r->ev_gemm) cudaEventDestroy(r->ev_gemm);
  if (r->pop_stream) cudaStreamDestroy(r->pop_stream);
  if (r->stream) cudaStreamDestroy(r->stream);
  delete r;
  return BCPNN_OK;
}

int bcpnn_recall_load(bcpnn_recall* r, const float* w, const float* bj, const float* epsc, const float* dsup,
                      const int8_t* spikes_tm3, const int8_t* spikes_tm2, const int8_t* spikes_tm1) {
  if (!r) return BCPNN_ERR_INVALID;
  if (!w || !bj || !epsc || !dsup || !spikes_tm3 || !spikes_tm2 || !spikes_tm1)
    return fail(r, BCPNN_ERR_INVALID, "null buffer");
  const int N = r->N, R = r->d.replicates;
  RCU(cudaSetDevice(r->d.device));
  if (r->wf) {
    /* FP32 contraction: W as given, [source][destination] */
    RCU(upload(r, r->wf, w, (size_t)N * N * 4));
    int* flag = r->err + 2;
    int bad = 0;
    RCU(cudaMemsetAsync(flag, 0, sizeof(int), r->stream));
    nonfinite_kernel<<<592, 256, 0, r->stream>>>(r->wf, (size_t)N * N, flag);
    RCU(cudaGetLastError());
    RCU(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, r->stream));
    RCU(cudaStreamSynchronize(r->stream));
    r->finite_w = bad == 0;
    r->launches++;
  } else {
    /* W^T in BF16: row j = destination MCU, K-contiguous over source MCUs */
    std::vector<uint16_t> wt((size_t)N * N);
    for (int i = 0; i < N; i++)
      for (int j = 0; j < N; j++) wt[(size_t)j * N + i] = to_bf16(w[(size_t)i * N + j]);
    RCU(upload(r, r->wt, wt.data(), wt.size() * 2));
  }
  RCU(upload(r, r->bj, bj, (size_t)N * 4));
  float* row_f = nullptr;
  int8_t* row_s = nullptr;
  RCU(cudaMalloc((void**)&row_f, (size_t)N * 4));
  cudaError_t e = cudaMalloc((void**)&row_s, (size_t)N * 3);
  if (e != cudaSuccess) {
    cudaFree(row_f);
    return fail(r, BCPNN_ERR_CUDA, std::string("recall load: ") + cudaGetErrorString(e));
  }
  r->kk = 0;
  const int prev = 1; /* parity buffer read by the next tick (kk = 0) */
  e = upload(r, row_f, epsc, (size_t)N * 4);
  if (e == cudaSuccess) {
    broadcast_f32_kernel<<<592, 256, 0, r->stream>>>(r->epsc[prev], R, N, row_f);
    e = cudaStreamSynchronize(r->stream);
  }
  if (e == cudaSuccess) e = upload(r, row_f, dsup, (size_t)N * 4);
  if (e == cudaSuccess) {
    broadcast_f32_kernel<<<592, 256, 0, r->stream>>>(r->dsup[prev], R, N, row_f);
    e = cudaStreamSynchronize(r->stream);
  }
  if (e == cudaSuccess) e = upload(r, row_s, spikes_tm3, (size_t)N);
  if (e == cudaSuccess) e = upload(r, row_s + N, spikes_tm2, (size_t)N);
  if (e == cudaSuccess) e = upload(r, row_s + 2 * N, spikes_tm1, (size_t)N);
  if (e == cudaSuccess) {
    for (int k = 0; k < 3; k++) {
      if (r->wf)
        broadcast_bits_kernel<<<592, 256, 0, r->stream>>>(r->sb[mod4(k - 3)], R, N, row_s + (size_t)k * N);
      else
        broadcast_spikes_kernel<<<592, 256, 0, r->stream>>>(r->s[mod4(k - 3)], R, N, row_s + (size_t)k * N);
    }
    e = cudaStreamSynchronize(r->stream);
  }
  cudaFree(row_f);
  cudaFree(row_s);
  if (e != cudaSuccess) return fail(r, BCPNN_ERR_CUDA, std::string("recall load: ") + cudaGetErrorString(e));
  r->launches += 5;
  r->loaded = true;
  return BCPNN_OK;
}

int bcpnn_recall_set_cues(bcpnn_recall* r, const int32_t* lgidx, float eps, const float* wmask) {
  if (!r) return BCPNN_ERR_INVALID;
  if (!lgidx || !wmask) return fail(r, BCPNN_ERR_INVALID, "null buffer");
  const size_t n = (size_t)r->d.replicates * r->d.hcu_num;
  RCU(cudaSetDevice(r->d.device));
  RCU(cudaMemcpyAsync(r->lgidx, lgidx, n * 4, cudaMemcpyHostToDevice, r->stream));
  RCU(cudaMemcpyAsync(r->wmask, wmask, n * 4, cudaMemcpyHostToDevice, r->stream));
  RCU(cudaStreamSynchronize(r->stream));
  r->lg_hit = bx_extgen_logf(1 + eps);
  r->lg_miss = bx_extgen_logf(0 + eps);
  r->cued = true;
  return BCPNN_OK;
}

int bcpnn_recall_clear_counts(bcpnn_recall* r) {
  if (!r) return BCPNN_ERR_INVALID;
  RCU(cudaSetDevice(r->d.device));
  RCU(cudaMemsetAsync(r->counts, 0, (size_t)r->d.replicates * r->N, r->stream));
  r->counted = 0;
  return BCPNN_OK;
}

int bcpnn_recall_run(bcpnn_recall* r, int32_t first, int32_t n_ticks, int32_t count_first, int32_t count_last) {
  if (!r) return BCPNN_ERR_INVALID;
  if (!r->loaded || !r->cued) return fail(r, BCPNN_ERR_STATE, "bcpnn_recall_run before load and set_cues");
  if (n_ticks < 0 || first < 0 || (long long)first + n_ticks > 0x7fffffffLL)
    return fail(r, BCPNN_ERR_INVALID, "bad tick range");
  int counted = 0;
  for (int t = first; t < first + n_ticks; t++) counted += (t >= count_first && t <= count_last);
  if (r->counted + counted > 255)
    return fail(r, BCPNN_ERR_INVALID, "more than 255 counted ticks since the last clear (uint8 counters)");
  RCU(cudaSetDevice(r->d.device));
  const bcpnn_recall_desc& d = r->d;
  Params p;
  p.counts = r->counts;
  p.bj = r->bj;
  p.lgidx = r->lgidx;
  p.wmask = r->wmask;
  p.lg_hit = r->lg_hit;
  p.lg_miss = r->lg_miss;
  p.N = r->N;
  p.H = d.hcu_num;
  p.R = d.replicates;
  p.taumdt = d.dt / d.pop.taum;   /* Pop.cpp:34 */
  p.maxfqdt = d.pop.maxfq * d.dt; /* Pop.cpp:36 */
  p.wtagain = d.pop.wtagain;
  p.igain = d.pop.igain;
  p.wgain = d.pop.wgain;
  p.lgbias = d.pop.lgbias;
  p.snoise = d.pop.snoise;
  p.one_m_kepsc = 1.0f - d.kepsc;
  p.pr = d.poisson_noise_hz * d.dt;
  p.poisson = d.poisson_noise_hz > 0.f;
  p.one = 1.0f;
  p.bound1 = p.maxfqdt * (0x1p32f * (1.0f + 0x1p-20f));
  p.pr_count = !p.poisson ? 0u : p.pr >= 1.0f ? 1u << 24 : (uint32_t)std::ceil((double)p.pr * 0x1p24);
  p.seed_base = d.seed_base;
  p.err = r->err;
  const Tiles tiles(d.replicates, r->N, r->sms);
  const int grid = tiles.total < r->sms ? tiles.total : r->sms;
  const int f32_tiles = (r->N / kF32BN) * (d.replicates / kF32BM);
  const int pop_blocks = (int)((size_t)d.replicates * d.hcu_num * 4 / 256);
  void (*pop)(Params) = nullptr;
  if (d.mcu_num == 16) pop = r->wf ? recall_pop_kernel<16, true> : recall_pop_kernel<16, false>;
  if (d.mcu_num == 32) pop = r->wf ? recall_pop_kernel<32, true> : recall_pop_kernel<32, false>;
  if (d.mcu_num == 64) pop = r->wf ? recall_pop_kernel<64, true> : recall_pop_kernel<64, false>;
  /* FP32: the contraction by events unless a weight is not finite, or so many
     MCUs can spike (an HCU's activities sum to at most 1) that the dense form
     is the faster one */
  const bool events = r->wf && r->finite_w && p.maxfqdt / (float)d.mcu_num + p.pr <= kEvMaxDensity;
  const long long ev_pairs = (long long)(r->N / kEvCols) * d.replicates;
  const int ev_grid = (int)(ev_pairs / kEvWarps < r->sms ? ev_pairs / kEvWarps : r->sms);
  const int list_blocks =
      (int)(((long long)d.replicates * ((r->N + kEvRows - 1) / kEvRows) + 255) / 256);
  /* BF16 in one launch per tick: tile CTAs and population CTAs with an SM each
     (not while the contraction is timed by itself) */
  const int pop_ctas = (int)(((long long)d.replicates * d.hcu_num * 4 + kThreads - 1) / kThreads);
  const bool together = !r->wf && !r->timing && grid + pop_ctas <= r->sms;
  const TickFn both = d.mcu_num == 16 ? recall_tick_kernel<16> : d.mcu_num == 32 ? recall_tick_kernel<32> : recall_tick_kernel<64>;
  /* Tick kk: the population update needs epsc(kk-1) and dsup(kk-1); the
     contraction needs S(kk-3) and epsc(kk-1).  So both wait only for tick
     kk-1 and run side by side: pop(kk) after gemm(kk-1) (it also must not
     overwrite S(kk) = S(kk-4) while gemm(kk-1) reads it), gemm(kk) after
     pop(kk-1) (which last read the epsc buffer gemm(kk) writes). */
  if (r->timing) {
    while (r->tev.size() < 2 * (size_t)n_ticks) {
      cudaEvent_t e;
      RCU(cudaEventCreate(&e));
      r->tev.push_back(e);
    }
  }
  if (events && n_ticks > 0) /* later ticks' lists are made beside the contraction of the tick before */
    recall_lists_kernel<<<list_blocks, 256, 0, r->stream>>>(r->sb[mod4(r->kk - 3)], r->lists[r->kk & 1],
                                                             r->list_cnt[r->kk & 1], d.replicates, r->N);
  RCU(cudaGetLastError());
  if (!together) {
    RCU(cudaEventRecord(r->ev_gemm, r->stream));
    RCU(cudaStreamWaitEvent(r->pop_stream, r->ev_gemm, 0));
  }
  for (int i = 0; i < n_ticks; i++) {
    const long long kk = r->kk + i;
    const int cur = (int)(kk & 1), prev = cur ^ 1;
    p.dsup_prev = r->dsup[prev];
    p.dsup_cur = r->dsup[cur];
    p.epsc_prev = r->epsc[prev];
    p.epsc_cur = r->epsc[cur];
    p.s_out = r->s[mod4(kk)];
    p.s_bits = r->sb[mod4(kk)];
    p.simstep = first + i;
    p.count_on = (first + i >= count_first && first + i <= count_last) ? 1 : 0;
    if (together) {
      cudaLaunchAttribute early = {};
      early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      early.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid + pop_ctas);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmemBytes;
      cfg.stream = r->stream;
      cfg.attrs = &early;
      cfg.numAttrs = 1;
      RCU(cudaLaunchKernelEx(&cfg, both, r->map_s[mod4(kk - 3)], r->map_w, p, r->sms, grid));
      continue;
    }
    pop<<<pop_blocks, 256, 0, r->pop_stream>>>(p);
    if (events && i + 1 < n_ticks)
      recall_lists_kernel<<<list_blocks, 256, 0, r->pop_stream>>>(r->sb[mod4(kk - 2)], r->lists[cur ^ 1],
                                                                   r->list_cnt[cur ^ 1], d.replicates, r->N);
    RCU(cudaGetLastError());
    if (r->timing) RCU(cudaEventRecord(r->tev[2 * i], r->stream));
    if (events)
      recall_events_kernel<<<ev_grid, kEvThreads, kEvSmemBytes, r->stream>>>(r->map_wf, r->sb[mod4(kk - 3)], r->lists[cur],
                                                                           r->list_cnt[cur], p);
    else if (r->wf)
      recall_fp32_kernel<<<f32_tiles, kF32Threads, 0, r->stream>>>(r->sb[mod4(kk - 3)], r->wf, p);
    else
      recall_tick_kernel<0><<<grid, kThreads, kSmemBytes, r->stream>>>(r->map_s[mod4(kk - 3)], r->map_w, p, r->sms, grid);
    RCU(cudaGetLastError());
    if (r->timing) RCU(cudaEventRecord(r->tev[2 * i + 1], r->stream));
    /* both kernels of tick kk are queued: each stream waits for the other's
       kernel of this tick before its kernel of tick kk+1 */
    RCU(cudaEventRecord(r->ev_pop, r->pop_stream));
    RCU(cudaEventRecord(r->ev_gemm, r->stream));
    RCU(cudaStreamWaitEvent(r->stream, r->ev_pop, 0));
    RCU(cudaStreamWaitEvent(r->pop_stream, r->ev_gemm, 0));
  }
  r->kk += n_ticks;
  r->counted += counted;
  r->launches += (together ? 1 : events ? 3 : 2) * (uint64_t)n_ticks;
  int rc = check_err(r); /* synchronises the stream: every timing event has completed */
  if (rc == BCPNN_OK && r->timing) {
    for (int i = 0; i < n_ticks; i++) {
      float ms = 0.f;
      RCU(cudaEventElapsedTime(&ms, r->tev[2 * i], r->tev[2 * i + 1]));
      r->contraction_ms += ms;
    }
    r->contraction_launches += (uint64_t)n_ticks;
  }
  return rc;
}

static int resolve_rows(bcpnn_recall* r, const char* name, int32_t row0, int32_t n_rows, size_t bytes, void** base,
                        size_t* elem, int* kind) {
  if (!name) return fail(r, BCPNN_ERR_INVALID, "null name");
  const int R = r->d.replicates;
  if (row0 < 0 || n_rows < 0 || row0 + (long long)n_rows > R) return fail(r, BCPNN_ERR_INVALID, "rows out of range");
  std::string s(name);
  const long long last = r->kk - 1; /* last tick run */
  *kind = 0;
  auto spikes = [&](long long tick) {
    *base = r->wf ? (void*)r->sb[mod4(tick)] : (void*)r->s[mod4(tick)];
    *elem = 2;
    *kind = r->wf ? 2 : 1;
  };
  if (s == "dsup") {
    *base = r->dsup[(int)(last & 1) & 1];
    *elem = 4;
  } else if (s == "epsc") {
    *base = r->epsc[(int)(last & 1) & 1];
    *elem = 4;
  } else if (s == "counts") {
    *base = r->counts;
    *elem = 1;
  } else if (s == "spike" || s == "spike_tm1") {
    spikes(last);
  } else if (s == "spike_tm2") {
    spikes(last - 1);
  } else if (s == "spike_tm3") {
    spikes(last - 2);
  } else {
    return fail(r, BCPNN_ERR_NOT_FOUND, "unknown recall array " + s);
  }
  size_t want = (size_t)n_rows * r->N * (*kind ? 1 : *elem);
  if (bytes != want) return fail(r, BCPNN_ERR_SIZE, "buffer size does not match rows x N");
  return BCPNN_OK;
}

int bcpnn_recall_read(bcpnn_recall* r, const char* name, int32_t row0, int32_t n_rows, void* host, size_t bytes) {
  if (!r || !host) return BCPNN_ERR_INVALID;
  void* base;
  size_t elem;
  int kind;
  int rc = resolve_rows(r, name, row0, n_rows, bytes, &base, &elem, &kind);
  if (rc) return rc;
  RCU(cudaSetDevice(r->d.device));
  const size_t off = (size_t)row0 * r->N * elem, n = (size_t)n_rows * r->N;
  if (kind == 2) {
    /* N is a multiple of 32: whole words per row */
    std::vector<uint32_t> tmp(n / 32);
    RCU(host_copy::to_host(tmp.data(), (uint32_t*)base + (size_t)row0 * r->N / 32, n / 8, r->stream));
    int8_t* o = (int8_t*)host;
    for (size_t i = 0; i < n; i++) o[i] = (int8_t)((tmp[i / 32] >> (i % 32)) & 1u);
  } else if (kind == 1) {
    std::vector<uint16_t> tmp(n);
    RCU(host_copy::to_host(tmp.data(), (uint8_t*)base + off, n * 2, r->stream));
    int8_t* o = (int8_t*)host;
    for (size_t i = 0; i < n; i++) o[i] = tmp[i] ? 1 : 0;
  } else {
    RCU(host_copy::to_host(host, (uint8_t*)base + off, n * elem, r->stream));
  }
  return BCPNN_OK;
}

int bcpnn_recall_write(bcpnn_recall* r, const char* name, int32_t row0, int32_t n_rows, const void* host,
                       size_t bytes) {
  if (!r || !host) return BCPNN_ERR_INVALID;
  if (name && std::string(name) == "counts") return fail(r, BCPNN_ERR_INVALID, "counts are cleared, not written");
  void* base;
  size_t elem;
  int kind;
  int rc = resolve_rows(r, name, row0, n_rows, bytes, &base, &elem, &kind);
  if (rc) return rc;
  RCU(cudaSetDevice(r->d.device));
  const size_t off = (size_t)row0 * r->N * elem, n = (size_t)n_rows * r->N;
  if (kind == 2) {
    std::vector<uint32_t> tmp(n / 32, 0u);
    const int8_t* in = (const int8_t*)host;
    for (size_t i = 0; i < n; i++) tmp[i / 32] |= (in[i] ? 1u : 0u) << (i % 32);
    RCU(cudaMemcpyAsync((uint32_t*)base + (size_t)row0 * r->N / 32, tmp.data(), n / 8, cudaMemcpyHostToDevice, r->stream));
    RCU(cudaStreamSynchronize(r->stream));
  } else if (kind == 1) {
    std::vector<uint16_t> tmp(n);
    const int8_t* in = (const int8_t*)host;
    for (size_t i = 0; i < n; i++) tmp[i] = in[i] ? 0x3F80u : 0u;
    RCU(cudaMemcpyAsync((uint8_t*)base + off, tmp.data(), n * 2, cudaMemcpyHostToDevice, r->stream));
    RCU(cudaStreamSynchronize(r->stream));
  } else {
    RCU(cudaMemcpyAsync((uint8_t*)base + off, host, n * elem, cudaMemcpyHostToDevice, r->stream));
    RCU(cudaStreamSynchronize(r->stream));
  }
  return BCPNN_OK;
}

int bcpnn_recall_get_stream(const bcpnn_recall* r, void** stream) {
  if (!r || !stream) return BCPNN_ERR_INVALID;
  *stream = (void*)r->stream;
  return BCPNN_OK;
}

int bcpnn_recall_launches(const bcpnn_recall* r, uint64_t* out) {
  if (!r || !out) return BCPNN_ERR_INVALID;
  *out = r->launches;
  return BCPNN_OK;
}

int bcpnn_recall_timing(bcpnn_recall* r, int32_t on) {
  if (!r) return BCPNN_ERR_INVALID;
  r->timing = on != 0;
  r->contraction_ms = 0.0;
  r->contraction_launches = 0;
  return BCPNN_OK;
}

int bcpnn_recall_contraction_time(const bcpnn_recall* r, double* total_ms, uint64_t* n_launches) {
  if (!r || !total_ms || !n_launches) return BCPNN_ERR_INVALID;
  *total_ms = r->contraction_ms;
  *n_launches = r->contraction_launches;
  return BCPNN_OK;
}

const char* bcpnn_recall_last_error(const bcpnn_recall* r) { return r ? r->last_error.c_str() : ""; }

}  // extern "C"
