/*
 * bcpnn_flow.cuh -- the tick of the plain FP32 path, and of its variant
 * ProcUpdMulti, as a dataflow inside and between CTAs: one CTA per (population,
 * destination HCU), persistent over a run, without a grid-wide barrier.  HCUs of
 * at most 128 MCUs; the others, and external spike replay, take tick_kernel
 * (bcpnn_tick.cuh) and the kernels of bcpnn_multi.cuh.
 *
 * What a tick t of HCU h needs (ProcUpdLazy.cpp:88-124):
 *   P(t)  population update  Pop.cpp:229-323: epsc(t-1), bj(t-1), and the
 *         softmax seed of the tick, the new dsup of the population's MCU 0
 *         (Pop.cpp:270), which HCU 0 computes first thing in its P(t);
 *   W(t)  rows  Proj.cpp:365-479, 667-720: the active rows listed by Q(t-1),
 *         pj(t), and the columns of t-1 (same cells); it gives epsc(t).  It
 *         does not need the spikes of t: zj alone takes them (Proj.cpp:349);
 *         columns  Proj.cpp:481-536, 722-760: the spikes of t, after its rows;
 *   Q(t)  delay queue  Proj.cpp:621-630, 645-664: it lists the active rows of
 *         t+1, then puts the spikes of t-1 of every source HCU into the queue.
 * The row traces (Proj.cpp:397-416) belong to the rows alone, so a warp of its
 * own, R(t), does those of the listed rows beside the decays of their cells.
 * The four groups run side by side and meet at shared-memory mbarriers: E(t) (W
 * -> P, Q: epsc(t), and the lists of t are free), S(t) (P -> W: spikes of t,
 * pj(t+1)), L(t+1) (Q -> W, R: the active rows of t+1), T(t) (R -> W: their new
 * pi).  A cell's thread goes from its decay to its weight without a barrier; one
 * barrier before the ordered sum is the only one of the rows.  A CTA
 * whose HCU spikes does its whole columns itself while its next population
 * update runs; only its rows of t+1 wait, and through them its P(t+2).
 *
 * Between CTAs a spike word carries its own flag: 32 spikes and the tick's tag
 * in 64 bits, one relaxed store, polled by every CTA's Q.  Q waits for the
 * words of all HCUs of the network, its sources or not, which bounds how far
 * CTAs run apart: P(t) needs the list of Q(t-2), which comes after all of
 * Q(t-3), so a CTA that publishes t has seen every word of t-4, and a CTA that
 * published t-4 has read the words of t-8 and the seed of t-4.  Words are kept
 * for 8 ticks and seeds for 4.
 *
 * Bound by the longest cycle of dependences: P(t) -> columns(t) -> rows(t+1) ->
 * P(t+2) takes two ticks, E(t-1) -> P(t) one.  Per tick, against tick_kernel with
 * its grid barrier and its columns spread over the grid: 10 x 10 1.8 us (7.4),
 * 50 x 50 2.4 (8.8), 100 x 100 with C = 1000 3.75 (9.9), 256 x 50 with C = 1000
 * 6.0 (13.8), 296 x 20 with C = 400 3.3 (11.3).  With the row traces in W and two
 * more barriers before the sum, decays as calls, and a queue word of every slot
 * shifted every tick: 2.8, 3.7, 6.0, 9.7 and 5.7.  The decays and their exact
 * division are those of bcpnn_device.cuh, so every value is bit-identical to
 * tick_kernel's and to the oracle's.
 *
 * The delay queue is kept by bit planes, a ring of 32 over the ticks: the rows
 * due are the set bits of one plane, 32 slots a word, and a spike sets one bit of
 * the plane its delay names.  Shifting every slot's own word took a warp 900
 * cycles per 128 slots, on the path from one tick's rows to the next (100 x 100
 * 4.4 -> 4.0 us per tick, 256 x 50 7.4 -> 6.3, 20 x 20 2.6 -> 2.2); and the list
 * of the due rows no longer waits for the other HCUs' spikes.
 *
 * Every wait is bounded (Args::wait_ns, kWaitNs but for the self-test): one that
 * runs out sets kErrBarrier and the CTA's abort flag, the groups of that CTA and,
 * at their next wait for it, the other CTAs leave their tick loops together.  The
 * network's state is undefined then, until a reset: such a CTA does not write
 * back what it keeps in shared memory, but its cells and row traces are in global
 * memory already, and a CTA that had finished did write.
 */
#ifndef BCPNN_FLOW_CUH
#define BCPNN_FLOW_CUH

#include "bcpnn_device.cuh"

namespace bcpnn {
namespace flow {

constexpr int kMaxM = 128;        /* one MCU per thread of up to four warps */
constexpr int kWordTicks = 8, kSeedTicks = 4;
constexpr int kMaxWords = 2047;   /* word and bit of a source MCU in 16 bits; word n_words: none */
constexpr unsigned long long kWaitNs = 2000000000ull;

struct Args {
  unsigned long long* words; /* [kWordTicks][n_words]: tag << 32 | 32 spikes */
  unsigned long long* seeds; /* [n_pops][kSeedTicks]: tag << 32 | float bits */
  const int* word0;          /* [n_pops] first word of a population */
  int n_words;
  unsigned long long wait_ns; /* limit of every wait */
  int si_mask; /* source-spike buffers by tick & si_mask: 1, or 3 (the block of four of ProcUpdMulti's resident launch) */
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

/* An event of every tick: four mbarriers by tick, so that a group which is up to
   three ticks behind the one that signals still finds its tick's phase (a phase
   is told by its parity; no group falls more than two behind). */
constexpr int kEventTicks = 4;

__device__ __forceinline__ void mb_init(unsigned long long* ev, int arrivals) {
  for (int k = 0; k < kEventTicks; ++k)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(ev + k)), "r"(arrivals) : "memory");
}

__device__ __forceinline__ void mb_arrive(unsigned long long* ev, int k) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(ev + k % kEventTicks)) : "memory");
}

__device__ __forceinline__ bool mb_try(unsigned long long* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

/* wait for the event of tick k >= 0; false when another group gave up, or after limit_ns */
__device__ __forceinline__ bool mb_wait(unsigned long long* ev, int k, volatile int* abort_flag, int* err,
                                        unsigned long long limit_ns) {
  unsigned long long* const b = ev + k % kEventTicks;
  const uint32_t parity = (uint32_t)(k / kEventTicks) & 1u;
  if (mb_try(b, parity)) return true;
  const unsigned long long t0 = now_ns();
  while (!mb_try(b, parity)) {
    if (*abort_flag) return false;
    if (now_ns() - t0 > limit_ns) {
      atomicOr(err, kErrBarrier);
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_word(unsigned long long* p, uint32_t tag, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | v) : "memory");
}

/* poll *p for the tag; false when a group or another CTA gave up a wait (no other error ends a run: a slot whose
   index is out of range is left out of it), or after limit_ns */
__device__ __forceinline__ bool poll_word(const unsigned long long* p, uint32_t tag, uint32_t& v, volatile int* abort_flag,
                                          int* err, unsigned long long limit_ns) {
  unsigned long long w = ld_word(p);
  if ((uint32_t)(w >> 32) != tag) {
    const unsigned long long t0 = now_ns();
    do {
      if (*abort_flag || (*(volatile int*)err & kErrBarrier)) {
        *abort_flag = 1;
        return false;
      }
      if (now_ns() - t0 > limit_ns) {
        atomicOr(err, kErrBarrier);
        *abort_flag = 1;
        return false;
      }
      w = ld_word(p);
    } while ((uint32_t)(w >> 32) != tag);
  }
  v = (uint32_t)w;
  return true;
}

/* barrier of one group of n threads; bar_any also gives the OR of a flag */
__device__ __forceinline__ void bar(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__device__ __forceinline__ bool bar_any(int id, int n, bool flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(id), "r"(n), "r"((uint32_t)flag)
      : "memory");
  return r != 0;
}

/* a cell's table entry for fewer than no ticks */
__device__ __noinline__ Entry entry_before(const TabRef& T, int pdt) {
  Entry e;
  table_pair(T.k.kp, T.k.ke, T.k.kzi, T.k.kzj, pdt, 0, e.A, e.B, T.k.fp64);
  recip_part(e.A, e.B, 0, e.R0, e.R1);
  return e;
}

/* shared-memory layout of a CTA, in 4-byte words */
struct Layout {
  int act;                 /* [M rounded up to 4] */
  int bits;                /* [n_words] the previous tick's spikes of the network, and a word of 0 */
  int w;                   /* [chunk cells] weights to add */
  int q[kMaxIn];           /* blocks of the incoming projections */
  int total;
};

/* slots per queue warp, a multiple of 64 */
__host__ __device__ inline int queue_part(int C, int qw) { return ((C + qw - 1) / qw + 63) & ~63; }

/* a projection's block: pj ej zj bj [M], epsc [2][M], pjn [2][M]; pi [2][C] (by list entry); then, of the n = qw * part
   slots: bit planes of the delay queue [32][n / 32], 16-bit list [2][n] and src [n], bytes di [n].  ProcUpdMulti: then
   the ti and zi that a tick's rows start from, [2][C] by list entry */
__host__ __device__ inline int block_words(int M, int C, int qw, bool multi) {
  const int n = qw * queue_part(C, qw);
  return 8 * M + (multi ? 6 : 2) * C + n + n + n / 2 + n / 4;
}

__host__ __device__ inline int chunk_rows(int M, int cells) { return cells / M < 1 ? 1 : cells / M; }

__host__ __device__ inline void layout(int M, int n_in, const int* C, int n_words, int cells, int qw, bool multi, Layout& L) {
  int o = 0;
  L.act = o; o += (M + 3) & ~3;
  L.bits = o; o += (n_words + 4) & ~3;
  const int rows = chunk_rows(M, cells);
  const int n = rows * M > cells ? rows * M : cells;
  L.w = o; o += n;
  for (int k = 0; k < kMaxIn; ++k) {
    L.q[k] = o;
    if (k < n_in) o += block_words(M, C[k], qw, multi);
  }
  L.total = o;
}

struct Block {
  float *pj, *ej, *zj, *bj, *epsc, *pjn, *pi;
  uint32_t* plane;
  uint16_t *list, *src;
  uint8_t* di;
  int* ti0;
  float* zi0;
};

template <int kQW>
__device__ __forceinline__ Block block(float* sm, const Layout& L, int k, int M, int C) {
  Block b;
  float* f = sm + L.q[k];
  b.pj = f;
  b.ej = f + M;
  b.zj = f + 2 * M;
  b.bj = f + 3 * M;
  b.epsc = f + 4 * M;
  b.pjn = f + 6 * M;
  const int n = kQW * queue_part(C, kQW);
  b.pi = f + 8 * M;
  b.plane = (uint32_t*)(b.pi + 2 * C);
  b.list = (uint16_t*)(b.plane + n);
  b.src = b.list + 2 * n;
  b.di = (uint8_t*)(b.src + n);
  b.ti0 = (int*)(b.di + n); /* ProcUpdMulti alone has these */
  b.zi0 = (float*)(b.ti0 + 2 * C);
  return b;
}

constexpr int kBarP = 1, kBarW = 2, kBarQ = 3;
/* delay byte: delay (1-31, or 0 for 32) in bits 0-4; bit 5: the source population is not published, and bits 6 and 7 are its constant flags
   by tick parity; else bit 6 is the source's spike before the launch */
constexpr int kUnfed = 32;

/* The loops of a tick are not unrolled: the four groups run through all of their
   code every tick, one dependent instruction after the other, and what does not
   stay in the instruction caches is fetched again each time (296 x 20, C = 400:
   4.7 -> 3.8 us per tick, 10 x 10: 2.4 -> 2.2).

   kThreads: 512 (one CTA per SM) or 256 (two); kPW warps of population update (M <= 32 kPW), kQW of delay queue, one of
   row traces, the others rows and columns.

   kMulti: ProcUpdMulti (Pop.cpp:222-311, 403-421, Proj.cpp:409-488, 557-706 of
   that variant).  The softmax is seeded by the HCU's own MCU 0; there are no
   columns: a row's cells start from the ti and zi that the row had before this
   tick (R puts them beside the list first, event O), replay the HCU's spikes
   since, which s_hist holds as a mask per MCU (bit b: b ticks before the tick
   after), and take a spike of this tick last, with the rows done and epsc given.
   Only then are the lists free (event F, for Q).  Bound by the longer of P and W:
   both start from E and S of the tick before.  us per tick with a ring of 25,
   against the launch with a grid barrier (res_tick_loop) or, for 256 x 50, two
   launches per tick: 10 x 10 5.8 -> 2.3, 50 x 50 6.3 -> 2.6, 100 x 100 with
   C = 1000 6.3 -> 3.0, 256 x 50 with C = 1000 31.3 -> 4.4. */
template <int kThreads, int kPW, int kQW, bool kMulti>
__global__ void __launch_bounds__(kThreads, 512 / kThreads)
    flow_kernel(const NetDev* __restrict__ net_g, const RunParams* __restrict__ rp_g, Args fa, int n_ticks) {
  constexpr int kP = kPW * 32, kQ = kQW * 32, kW = kThreads - kP - kQ - 32;
  constexpr int kCells = kThreads; /* row cells of one chunk */
  extern __shared__ __align__(16) float sm[];
  __shared__ NetDev s_net;
  __shared__ RunParams s_rp;
  __shared__ PopDev s_pop;
  __shared__ ProjDev s_proj[kMaxIn];
  __shared__ TabRef s_tab[kMaxIn];
  __shared__ int s_inp[kMaxIn], s_srcM[kMaxIn], s_src0[kMaxIn], s_fed[kMaxIn];
  __shared__ Layout s_L;
  __shared__ unsigned long long s_E[kEventTicks], s_S[kEventTicks], s_Lst[kEventTicks], s_T[kEventTicks];
  __shared__ unsigned long long s_O[kEventTicks], s_F[kEventTicks];
  __shared__ uint32_t s_hist[2][kMulti ? kP : 1]; /* by tick parity */
  __shared__ int s_abort;
  __shared__ int s_nl[kMaxIn][2][kQW]; /* list lengths by tick parity */
  __shared__ uint32_t s_spk[2][kPW];   /* spikes of this HCU by tick parity */
  __shared__ float s_red[kPW];
  __shared__ float s_seed;
  __shared__ unsigned long long s_rows, s_cols;

  const int tid = threadIdx.x;
  if (tid == 0) {
    s_net = *net_g;
    s_rp = *rp_g;
    s_abort = 0;
    s_rows = s_cols = 0;
    mb_init(s_E, kW / 32 + 1);
    mb_init(s_S, 1);
    mb_init(s_Lst, 1);
    mb_init(s_T, 1);
    mb_init(s_O, 1);
    mb_init(s_F, kW / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const NetDev* __restrict__ net = &s_net;
  const RunParams* __restrict__ rp = &s_rp;
  const int P = net->cta_pop[blockIdx.x], h = net->cta_hcu[blockIdx.x];
  if (tid == 0) s_pop = net->pops[P];
  __syncthreads();
  const PopDev& pop = s_pop;
  const int M = pop.M, n = pop.n, n_in = pop.n_in;
  if (tid < kMaxIn && tid < n_in) {
    const int p = pop.in_proj[tid];
    s_inp[tid] = p;
    s_proj[tid] = net->projs[p];
    s_tab[tid] = rp->tabs[p];
    const PopDev& src = net->pops[s_proj[tid].src];
    s_srcM[tid] = src.M;
    s_src0[tid] = fa.word0[s_proj[tid].src];
    int fed = 0;
#pragma unroll 1
    for (int k = 0; k < src.n_out; ++k) fed |= src.out_proj[k] == p;
    s_fed[tid] = fed;
  }
  __syncthreads();
  if (tid == 0) {
    int c[kMaxIn];
#pragma unroll
    for (int k = 0; k < kMaxIn; ++k) c[k] = k < n_in ? s_proj[k].C : 0;
    layout(M, n_in, c, fa.n_words, kCells, kQW, kMulti, s_L);
  }
  __syncthreads();
  const Layout& L = s_L;
  float* s_act = sm + L.act;
  uint32_t* s_bits = (uint32_t*)(sm + L.bits);

  /* ---- load the state the previous tick left ---- */
  const int cur0 = rp->k0 & 1, prev0 = cur0 ^ 1;
  const float prn = rp->prn;
  /* the source of an empty slot: a word that is always 0; none | 1: of a slot that no spike reaches */
  const uint32_t none = (uint32_t)fa.n_words << 5;
  if (tid == 0) s_bits[fa.n_words] = 0u;
#pragma unroll 1
  for (int k = 0; k < n_in; ++k) {
    const ProjDev& J = s_proj[k];
    Block B = block<kQW>(sm, L, k, M, J.C);
    const size_t eoff = (size_t)J.proj_in_pop * n;
    const float kp = J.taupdt * prn;
#pragma unroll 1
    for (int j = tid; j < M; j += kThreads) {
      const int idx = h * M + j;
      const float pj = J.pj[idx], ej = J.ej[idx];
      B.pj[j] = pj;
      B.ej[j] = ej;
      B.zj[j] = J.zj[idx];
      B.bj[j] = pop.bj[prev0][eoff + idx];
      B.epsc[prev0 * M + j] = pop.epsc[prev0][eoff + idx];
      B.pjn[cur0 * M + j] = pj + (ej - pj) * kp;
    }
    /* a queue entry's bit b, due in b ticks, is bit `slot` of plane b; whole warps, a word of slots each */
    const int part = queue_part(J.C, kQW), slots = kQW * part;
#pragma unroll 1
    for (int s = tid; s < slots; s += kThreads) {
      const int r = h * J.C + s, ii = s < J.C ? J.ii[r] : -1;
      uint32_t src = none, di = 0, qi = 0;
      if (ii >= J.Ns) atomicOr(net->err, kErrIndex);
      if (ii >= 0 && ii < J.Ns) {
        qi = (uint32_t)J.qi[r];
        const int hs = ii / s_srcM[k], ms = ii - hs * s_srcM[k];
        const int delay = J.di[r];
        if (delay >= 1 && delay <= 32) {
          src = (uint32_t)(s_src0[k] + hs * ((s_srcM[k] + 31) >> 5) + (ms >> 5)) << 5 | (uint32_t)(ms & 31);
          di = (uint32_t)delay & 31u;
          if (s_fed[k]) di |= J.si[0][(size_t)((rp->k0 + fa.si_mask) & fa.si_mask) * J.Ns + ii] > 0 ? 64u : 0u;
          else di |= kUnfed | (J.si[0][ii] > 0 ? 64u : 0u) | (J.si[1][ii] > 0 ? 128u : 0u);
        } else { /* written into the state: bit delay - 1 is none of the word's, no spike arrives */
          src = none | 1u;
        }
      }
      B.src[s] = (uint16_t)src;
      B.di[s] = (uint8_t)di;
#pragma unroll 1
      for (int b = 0; b < 32; ++b) {
        const uint32_t m = __ballot_sync(0xffffffffu, (qi >> b) & 1u);
        if ((tid & 31) == b) B.plane[b * (slots >> 5) + (s >> 5)] = m;
      }
    }
    /* the listed rows, ascending, by queue warp: the first part's are the first n0 */
    const int cnt = J.list_cnt[h];
    const int* rows = J.list + h * J.C;
    int n0 = cnt;
    if (kQW > 1) {
      int lo = 0, hi = cnt; /* first entry of the second part */
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (rows[mid] - h * J.C < part) lo = mid + 1;
        else hi = mid;
      }
      n0 = lo;
    }
    if (tid < kQW) s_nl[k][cur0][tid] = tid == 0 ? n0 : cnt - n0;
#pragma unroll 1
    for (int e = tid; e < cnt; e += kThreads)
      B.list[cur0 * kQW * part + (e < n0 ? e : part + e - n0)] = (uint16_t)(rows[e] - h * J.C);
  }
  if (tid < ((M + 3) & ~3) - M) s_act[M + tid] = 0.0f; /* read by the serial sum */
  if (kMulti)
#pragma unroll 1
    for (int j = tid; j < M; j += kThreads) {
      /* bit b: the ring's entry for tick simstep0 - 1 - b (at most 32 ticks) */
      uint32_t m = 0;
#pragma unroll 1
      for (int b = 0; b < pop.ring_len - 1; ++b) {
        const int t = rp->simstep0 - 1 - b;
        if (t >= 0 && pop.ring[(size_t)(t % pop.ring_len) * n + h * M + j] > 0) m |= 1u << b;
      }
      s_hist[prev0][j] = m;
    }
  __syncthreads();

  if (tid < kP) {
    /* ================= P: population update, j-traces ================= */
    const int j = tid, warp = tid >> 5, lane = tid & 31;
    const bool active = j < M;
    const int idx = h * M + (active ? j : 0);
    float dsup = pop.dsup[prev0][idx], act = pop.act[idx];
    int cnt = pop.counter[idx];
    float ada = kMulti ? pop.ada[idx] : 0.0f;
    bool spk = false;
    const float lg = rp->lginp[pop.mcu_start + idx], wm = rp->wmask[pop.hcu_start + h];
    const int wph = (M + 31) >> 5;
    const float pr = net->poisson_hz * net->dt;
    bool bad = false;
#pragma unroll 1
    for (int it = 0; it < n_ticks; ++it) {
      const int simstep = rp->simstep0 + it, cur = (rp->k0 + it) & 1, prev = cur ^ 1;
      const uint32_t tag = rp->serial0 + (uint32_t)it;
      unsigned long long* const slot = fa.seeds + P * kSeedTicks + (tag & (kSeedTicks - 1));
      const bool own_seed = kMulti || h == 0;
      /* HCU 0, which waits for no seed, is mostly ahead: its seed is there already (10 x 10 2.07 -> 1.84 us per tick) */
      unsigned long long early = 0;
      if (!own_seed && lane == 0) early = ld_word(slot);
      /* what depends on tick and MCU only, before the wait */
      const float u = bx_uniform01(pop.rng_seed, pop.rng_pop, (uint32_t)simstep, (uint32_t)idx);
      bool extra = false;
      if (net->poisson_hz > 0.0f)
        extra = bx_uniform01_poisson(pop.rng_seed, pop.rng_pop, (uint32_t)simstep, (uint32_t)idx) < pr;
      float noise = 0.0f;
      if (pop.snoise != 0.0f)
        noise = pop.snoise * dev_normal01(pop.rng_seed, pop.rng_pop, (uint32_t)simstep, (uint32_t)idx);
      float sup = pop.lgbias + pop.igain * lg + noise;
      if (it > 0 && !bad) bad = !mb_wait(s_E, it - 1, &s_abort, net->err, fa.wait_ns);
      float wsup = 0.0f;
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const Block B = block<kQW>(sm, L, k, M, s_proj[k].C);
        if (active) wsup += B.bj[j] + B.epsc[prev * M + j];
      }
      sup += (pop.wgain * wm) * wsup;
      if (kMulti) {
        sup -= wm * ada;
        sup = (float)((double)sup + 6.9 * (double)wm); /* a double constant in gsbn */
      }
      const float d = dsup + (sup - dsup) * pop.taumdt;
      /* the softmax seed (Pop.cpp:270) */
      float seed = 0.0f;
      if (own_seed) {
        if (tid == 0) {
          if (!kMulti) st_word(slot, tag, __float_as_uint(d));
          s_seed = d;
        }
      } else if (lane == 0) {
        if (it == 0) {
          float ws = 0.0f;
          int offset = 0;
#pragma unroll 1
          for (int m = 0; m < pop.dim_proj; m++) {
            ws += __ldcg(pop.bj[prev] + offset) + __ldcg(pop.epsc[prev] + offset);
            offset += n;
          }
          float nz = 0.0f;
          if (pop.snoise != 0.0f) nz = pop.snoise * dev_normal01(pop.rng_seed, pop.rng_pop, (uint32_t)simstep, 0u);
          float sp = pop.lgbias + pop.igain * rp->lginp[pop.mcu_start] + nz;
          sp += (pop.wgain * rp->wmask[pop.hcu_start]) * ws;
          const float d0 = __ldcg(pop.dsup[prev]);
          seed = d0 + (sp - d0) * pop.taumdt;
        } else if (!bad) {
          uint32_t v = (uint32_t)early;
          if ((uint32_t)(early >> 32) != tag) bad = !poll_word(slot, tag, v, &s_abort, net->err, fa.wait_ns);
          seed = __uint_as_float(v);
        }
      }
      /* pj of the next tick (Proj.cpp:340: it takes ej and pj only); its buffer is free, the rows that read it are done */
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const ProjDev& J = s_proj[k];
        const Block B = block<kQW>(sm, L, k, M, J.C);
        if (active) {
          const float pj = B.pjn[cur * M + j];
          float ej = B.ej[j];
          ej += (B.zj[j] - ej) * J.ke;
          B.pj[j] = pj;
          B.ej[j] = ej;
          B.pjn[prev * M + j] = pj + (ej - pj) * (J.taupdt * prn);
        }
      }
      /* the maximum: of the HCU's MCUs, then against the seed, which a NaN never replaces and which stays if it is NaN */
      float mx = __int_as_float(0xff800000);
      if (active && d > mx) mx = d;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float w = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = (w > mx) ? w : mx;
      }
      seed = __shfl_sync(0xffffffffu, seed, 0);
      if (kPW > 1) {
        if (lane == 0) s_red[warp] = mx;
        bar(kBarP, kP);
        if (own_seed) seed = s_seed;
        float m = seed;
#pragma unroll
        for (int w = 0; w < kPW; ++w) m = (s_red[w] > m) ? s_red[w] : m;
        mx = m;
      } else {
        if (own_seed) seed = __shfl_sync(0xffffffffu, d, 0);
        mx = (mx > seed) ? mx : seed;
      }
      const float maxact = bx_expf(pop.wtagain * mx);
      float a = bx_expf(pop.wtagain * (d - mx));
      if (maxact < 1.0f) a *= maxact;
      if (active) s_act[j] = a;
      if (kPW > 1) bar(kBarP, kP);
      else __syncwarp();
      /* serial, in MCU order (Pop.cpp:281-293), by every thread; the padding adds +0 to a sum that is never -0 */
      float vsum = 0.0f;
      {
        const float4* v = (const float4*)s_act;
        float4 x = v[0];
#pragma unroll 1
        for (int m = 4; m < M; m += 4) {
          const float4 y = v[m >> 2];
          vsum += x.x;
          vsum += x.y;
          vsum += x.z;
          vsum += x.w;
          x = y;
        }
        vsum += x.x;
        vsum += x.y;
        vsum += x.z;
        vsum += x.w;
      }
      if (vsum > 1.0f) a /= vsum;
      spk = active && ((u < a * pop.maxfqdt) || extra);
      const uint32_t word = __ballot_sync(0xffffffffu, spk);
      if (lane == 0 && warp < wph) {
        st_word(fa.words + (size_t)(tag & (kWordTicks - 1)) * fa.n_words + fa.word0[P] + h * wph + warp, tag, word);
        s_spk[cur][warp] = word;
      }
      if (kMulti) s_hist[cur][j] = (s_hist[prev][j] << 1) | (spk ? 1u : 0u);
      if (kPW > 1) {
        bad = bar_any(kBarP, kP, bad);
      } else {
        bad = __any_sync(0xffffffffu, bad);
        __syncwarp();
      }
      if (tid == 0) mb_arrive(s_S, it); /* the group's writes happen before: barrier above */
      /* in the shadow of the rows and columns: state, traces, bias, records */
      dsup = d;
      act = a;
      cnt += spk ? 1 : 0;
      if (kMulti) {
        ada += (pop.adgain * a - ada) * pop.tauadt;
        /* the ring holds the last ticks: what this run would overwrite itself is not written */
        if (active && n_ticks - it <= pop.ring_len) pop.ring[(size_t)(simstep % pop.ring_len) * n + idx] = spk ? 1 : 0;
      }
      if (spk) {
        atomicOr(&pop.spk_log[(size_t)it * pop.log_words + (idx >> 5)], 1u << (idx & 31));
        if (idx == 9)
#pragma unroll 1
          for (int k = 0; k < n_in; ++k) atomicOr(&net->ss_log[(size_t)it * net->n_projs + s_inp[k]], 2u);
      }
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const ProjDev& J = s_proj[k];
        const Block B = block<kQW>(sm, L, k, M, J.C);
        if (active) {
          float zj = B.zj[j];
          zj *= (1 - J.kzj);
          if (spk) zj += J.kftj;
          B.zj[j] = zj;
          if (J.taupdt * prn != 0.0f) B.bj[j] = J.bgain * bx_logf(B.pj[j] + J.eps);
        }
      }
      if (bad) break;
    }
    bar(0, kThreads);
    if (!s_abort && active) {
      const int last = (rp->k0 + n_ticks - 1) & 1;
      pop.dsup[last][idx] = dsup;
      pop.act[idx] = act;
      pop.counter[idx] = cnt;
      pop.spike[idx] = spk ? 1 : 0;
      if (kMulti) pop.ada[idx] = ada;
      const size_t si_last = (size_t)((rp->k0 + n_ticks - 1) & fa.si_mask) * n;
#pragma unroll 1
      for (int k = 0; k < pop.n_out; ++k) net->projs[pop.out_proj[k]].si[0][si_last + idx] = spk ? 1 : 0;
    }
  } else if (tid < kP + kQ) {
    /* ================= Q: delay queue, spike words ================= */
    const int qt = tid - kP, warp = qt >> 5, lane = qt & 31;
    bool bad = false;
#pragma unroll 1
    for (int it = 0; it < n_ticks; ++it) {
      const int prev = (rp->k0 + it + 1) & 1, nxt = prev;
      /* the lists written below were read by the rows of it - 1 */
      if (it > 0 && !bad) bad = !mb_wait(s_E, it - 1, &s_abort, net->err, fa.wait_ns);
      if (kMulti && it > 0 && !bad) bad = !mb_wait(s_F, it - 1, &s_abort, net->err, fa.wait_ns);
      if (kQW > 1) bar(kBarQ, kQ);
      else __syncwarp();
      /* the slots due, from plane `it`, a word of 32 per lane; then the planes are one tick further: what was plane 0 is
         the last one, and takes what was the last (the queue word is shifted with its sign, Proj.cpp:621) */
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const int C = s_proj[k].C;
        const Block B = block<kQW>(sm, L, k, M, C);
        const int part = queue_part(C, kQW), words = kQW * part >> 5;
        uint32_t* const due = B.plane + (it & 31) * words;
        const uint32_t* const last = B.plane + ((it + 31) & 31) * words;
        uint16_t* out = B.list + (nxt * kQW + warp) * part;
        int total = 0;
#pragma unroll 1
        for (int x0 = warp * (part >> 5); x0 < (warp + 1) * (part >> 5); x0 += 32) {
          const int x = x0 + lane;
          uint32_t m = 0;
          if (x < (warp + 1) * (part >> 5)) {
            m = due[x];
            due[x] = last[x];
          }
          const int c = __popc(m);
          int at = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += v;
          }
          const int sum = __shfl_sync(0xffffffffu, at, 31);
          at += total - c;
#pragma unroll 1
          for (; m; m &= m - 1) out[at++] = (uint16_t)(x * 32 + __ffs(m) - 1);
          total += sum;
        }
        if (lane == 0) s_nl[k][nxt][warp] = total;
      }
      if (kQW > 1) {
        bad = bar_any(kBarQ, kQ, bad);
      } else {
        bad = __any_sync(0xffffffffu, bad);
        __syncwarp();
      }
      if (qt == 0) mb_arrive(s_Lst, it);
      if (bad) break;
      if (it > 0) {
        const uint32_t tag = rp->serial0 + (uint32_t)(it - 1);
        const unsigned long long* w = fa.words + (size_t)(tag & (kWordTicks - 1)) * fa.n_words;
#pragma unroll 1
        for (int x0 = 0; x0 < fa.n_words; x0 += 4 * kQ) {
          /* four words' loads at once; the late ones are polled */
          unsigned long long v[4];
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            const int x = x0 + y * kQ + qt;
            if (x < fa.n_words) v[y] = ld_word(w + x);
          }
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            const int x = x0 + y * kQ + qt;
            if (x < fa.n_words) {
              uint32_t b = (uint32_t)v[y];
              if ((uint32_t)(v[y] >> 32) != tag && !bad) bad = !poll_word(w + x, tag, b, &s_abort, net->err, fa.wait_ns);
              s_bits[x] = b;
            }
          }
        }
        __syncwarp();
        if (kQW > 1) bar(kBarQ, kQ);
      }
      /* the slots whose source has spiked: most have not, so eight are looked at together */
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const int C = s_proj[k].C;
        const Block B = block<kQW>(sm, L, k, M, C);
        const int part = queue_part(C, kQW), words = kQW * part >> 5;
        const bool words_tell = it > 0 && s_fed[k];
#pragma unroll 1
        for (int s0 = warp * part; s0 < (warp + 1) * part; s0 += 64) {
          const int s = s0 + 2 * lane;
          const uint32_t src = *(const uint32_t*)(B.src + s);
          uint32_t hit;
          if (words_tell) {
            hit = (s_bits[(src & 0xffffu) >> 5] >> (src & 31u)) & 1u;
            hit |= ((s_bits[src >> 21] >> ((src >> 16) & 31u)) & 1u) << 1;
          } else {
            hit = 0;
#pragma unroll 1
            for (int y = 0; y < 2; ++y) {
              const uint32_t di = B.di[s + y];
              hit |= ((di >> (di & kUnfed ? 6 + prev : 6)) & 1u) << y;
            }
          }
#pragma unroll 1
          for (; hit; hit &= hit - 1) {
            const int e = s + __ffs(hit) - 1;
            /* due in di - 1 ticks, seen from the next one */
            atomicOr(B.plane + ((it + (B.di[e] & 31)) & 31) * words + (e >> 5), 1u << (e & 31));
          }
        }
      }
    }
    bar(0, kThreads);
  } else if (tid < kP + kQ + 32) {
    /* ================= R: row traces ================= */
    const int lane = tid & 31;
    bool bad = false;
#pragma unroll 1
    for (int it = 0; it < n_ticks; ++it) {
      const int simstep = rp->simstep0 + it, cur = (rp->k0 + it) & 1;
      if (it > 0) bad = !mb_wait(s_Lst, it - 1, &s_abort, net->err, fa.wait_ns);
      if (__any_sync(0xffffffffu, bad)) break;
      if (kMulti) {
#pragma unroll 1
        for (int k = 0; k < n_in; ++k) {
          const ProjDev& J = s_proj[k];
          const Block B = block<kQW>(sm, L, k, M, J.C);
          const int part = queue_part(J.C, kQW);
          const uint16_t* l0 = B.list + cur * kQW * part;
          const int n0 = s_nl[k][cur][0], nrow = kQW > 1 ? n0 + s_nl[k][cur][kQW - 1] : n0;
#pragma unroll 1
          for (int e = lane; e < nrow; e += 32) {
            const int r = h * J.C + (int)(e < n0 ? l0[e] : l0[part + e - n0]);
            B.ti0[cur * J.C + e] = J.ti[r];
            B.zi0[cur * J.C + e] = J.zi[r];
          }
        }
        __syncwarp();
        if (lane == 0) mb_arrive(s_O, it);
      }
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const ProjDev& J = s_proj[k];
        const Block B = block<kQW>(sm, L, k, M, J.C);
        const TabRef& T = s_tab[k];
        const int part = queue_part(J.C, kQW);
        const uint16_t* l0 = B.list + cur * kQW * part;
        const int n0 = s_nl[k][cur][0], nrow = kQW > 1 ? n0 + s_nl[k][cur][kQW - 1] : n0;
#pragma unroll 1
        for (int e = lane; e < nrow; e += 32) {
          const int r = h * J.C + (int)(e < n0 ? l0[e] : l0[part + e - n0]);
          if (r == 9) atomicOr(&net->ss_log[(size_t)it * net->n_projs + s_inp[k]], 1u);
          const int pdt = simstep - J.ti[r];
          const float4 tr = make_float4(J.pi[r], J.ei[r], J.zi[r], 0.0f);
          float pi = tr.x;
          if (pdt <= 0) {
            if (!kMulti) J.zi[r] = tr.z + J.kfti;
          } else {
            float4 A, Bt;
            double2 R0, R1;
            entry(T, pdt, 2, A, Bt, R0, R1);
            const float4 rt = row_step(tr, T, A, Bt, R0, R1);
            pi = rt.x;
            J.pi[r] = pi;
            J.ei[r] = rt.y;
            J.zi[r] = rt.z + J.kfti;
          }
          J.ti[r] = simstep;
          B.pi[cur * J.C + e] = pi;
        }
      }
      __syncwarp();
      if (lane == 0) {
        mb_arrive(s_T, it);
        mb_arrive(s_E, it); /* the rows wait for T only where a weight needs it */
      }
    }
    bar(0, kThreads);
  } else {
    /* ================= W: rows, columns ================= */
    const int wt = tid - kP - kQ - 32, lane = tid & 31;
    float* s_w = sm + L.w;
    const int rch = chunk_rows(M, kCells);
    bool bad = false;
#pragma unroll 1
    for (int it = 0; it < n_ticks; ++it) {
      const int simstep = rp->simstep0 + it, cur = (rp->k0 + it) & 1, prev = cur ^ 1;
      if (it > 0) {
        if (!bad) bad = !mb_wait(s_Lst, it - 1, &s_abort, net->err, fa.wait_ns);
        /* together: a list that is not there is not read.  Also: the columns of it - 1 are in place */
        bad = bar_any(kBarW, kW, bad);
        if (bad) break;
      }
      bool traces = false, start = false;
#pragma unroll 1
      for (int k = 0; k < n_in; ++k) {
        const ProjDev& J = s_proj[k];
        const int C = J.C;
        const Block B = block<kQW>(sm, L, k, M, C);
        const TabRef& T = s_tab[k];
        const float kp = J.taupdt * prn;
        const int part = queue_part(C, kQW);
        const uint16_t* l0 = B.list + cur * kQW * part;
        const int n0 = s_nl[k][cur][0], nrow = kQW > 1 ? n0 + s_nl[k][cur][kQW - 1] : n0;
        if (nrow == 0)
#pragma unroll 1
          for (int j = wt; j < M; j += kW) B.epsc[cur * M + j] = B.epsc[prev * M + j] * (1 - J.kepsc);
#pragma unroll 1
        for (int base = 0; base < nrow; base += rch) {
          const int nr = min(rch, nrow - base);
#pragma unroll 1
          for (int c = wt; c < nr * M; c += kW) {
            const int rr = c / M, j = c - rr * M, e = base + rr;
            const size_t index = (size_t)(h * C + (int)(e < n0 ? l0[e] : l0[part + e - n0])) * M + j;
            if constexpr (kMulti) {
              float4 q = J.cell[index];
              if (!start) {
                if (!mb_wait(s_O, it, &s_abort, net->err, fa.wait_ns)) bad = true;
                start = true;
              }
              int tij = B.ti0[cur * C + e];
              float zi2 = B.zi0[cur * C + e];
              /* the spikes after max(tij, simstep - ring) and before this tick, ascending; bit b: tick simstep - b */
              const int span = min(simstep - tij, pop.ring_len - 1);
              uint32_t m = span > 1 ? (s_hist[prev][j] << 1) & (0xffffffffu >> (32 - span)) : 0u;
#pragma unroll 1
              for (;;) {
                const int b = m ? 31 - __clz(m) : 0, pdt = simstep - b - tij;
                float4 A, Bt;
                double2 R0, R1;
                if (pdt >= 0) {
                  entry(T, pdt, 0, A, Bt, R0, R1);
                } else { /* a row written with a later tick: gsbn's expressions all the same */
                  const Entry x = entry_before(T, pdt);
                  A = x.A;
                  Bt = x.B;
                  R0 = x.R0;
                  R1 = x.R1;
                }
                const float4 d = cell_step(make_float4(q.x, q.y, zi2, q.w), T, A, Bt, R0, R1);
                q.x = d.x;
                q.y = d.y;
                q.w = d.w;
                if (m == 0) break; /* the cell keeps the zi2 of its last replay */
                zi2 = d.z;
                q.w += J.kftj;
                tij = simstep - b;
                m &= ~(1u << b);
              }
              q.z = zi2;
              float w;
              if (kp != 0.0f) {
                if (!traces) {
                  if (!mb_wait(s_T, it, &s_abort, net->err, fa.wait_ns)) bad = true;
                  traces = true;
                }
                w = J.wgain * bx_logf((q.x + J.eps2) / ((B.pi[cur * C + e] + J.eps) * (B.pjn[cur * M + j] + J.eps)));
                J.wij[index] = w;
              } else {
                w = J.wij[index];
              }
              J.cell[index] = q;
              s_w[c] = w;
              continue;
            }
            const int pdt = simstep - J.tij[index];
            float4 q = J.cell[index];
            float w = kp == 0.0f ? J.wij[index] : 0.0f; /* without plasticity the weights stay */
            if (pdt <= 0) {
              q.z += J.kfti;
              w = -0.0f; /* adds nothing, to any sum */
            } else {
              float4 A, Bt;
              double2 R0, R1;
              entry(T, pdt, 0, A, Bt, R0, R1);
              q = cell_step(q, T, A, Bt, R0, R1);
              q.z = q.z + J.kfti;
              if (kp != 0.0f) { /* Proj.cpp:458-462 */
                if (!traces) {
                  if (!mb_wait(s_T, it, &s_abort, net->err, fa.wait_ns)) bad = true;
                  traces = true;
                }
                w = J.wgain * bx_logf((q.x + J.eps2) / ((B.pi[cur * C + e] + J.eps) * (B.pjn[cur * M + j] + J.eps)));
                J.wij[index] = w;
              }
            }
            J.cell[index] = q;
            J.tij[index] = simstep;
            s_w[c] = w;
          }
          bar(kBarW, kW);
          /* epsc in row order */
#pragma unroll 1
          for (int j = wt; j < M; j += kW) {
            float e = base == 0 ? B.epsc[prev * M + j] * (1 - J.kepsc) : B.epsc[cur * M + j];
#pragma unroll 1
            for (int rr = 0; rr < nr; ++rr) e += s_w[rr * M + j];
            B.epsc[cur * M + j] = e;
          }
          if (base + rch < nrow || k + 1 < n_in) bar(kBarW, kW);
        }
        if (wt == 0) s_rows += (unsigned long long)nrow * M;
      }
      __syncwarp();
      if (lane == 0) mb_arrive(s_E, it);
      /* columns of this tick's spikes */
      if (!bad) bad = !mb_wait(s_S, it, &s_abort, net->err, fa.wait_ns);
      if (!bad) {
        uint32_t sp[kPW];
        int nspk = 0;
#pragma unroll
        for (int w = 0; w < kPW; ++w) {
          sp[w] = w * 32 < M ? s_spk[cur][w] : 0u;
          nspk += __popc(sp[w]);
        }
#pragma unroll 1
        for (int k = 0; k < n_in && nspk > 0; ++k) {
          const ProjDev& J = s_proj[k];
          const int C = J.C;
          const Block B = block<kQW>(sm, L, k, M, C);
          const TabRef& T = s_tab[k];
#pragma unroll 1
          for (int w = 0; w < kPW; ++w)
#pragma unroll 1
            for (uint32_t m = s_spk[cur][w]; m && w * 32 < M; m &= m - 1) {
              const int j = w * 32 + __ffs(m) - 1;
              if constexpr (kMulti) {
                /* the cells of this tick's rows: written by other threads of the group, before its last barrier */
                const int part = queue_part(C, kQW);
                const uint16_t* l0 = B.list + cur * kQW * part;
                const int n0 = s_nl[k][cur][0], nrow = kQW > 1 ? n0 + s_nl[k][cur][kQW - 1] : n0;
#pragma unroll 1
                for (int e = wt; e < nrow; e += kW)
                  J.cell[(size_t)(h * C + (int)(e < n0 ? l0[e] : l0[part + e - n0])) * M + j].w += J.kftj;
                continue;
              }
              float4* const cell = J.cell + (size_t)h * C * M + j;
              int* const tij = J.tij + (size_t)h * C * M + j;
              /* a cell at a time, with the loads of the thread's next one in flight.  Two at a time was more code to
                 fetch every tick and spilled: 100 x 100 4.0 -> 3.75 us per tick, 10 x 10 2.13 -> 2.02, 296 x 20 3.65 ->
                 3.3; with the next one's table entry in flight too 4.1, 2.09 and 3.5 */
              int pn;
              float4 next;
              auto load = [&](int s) {
                pn = -1;
                if (s < C && B.src[s] != none) {
                  pn = max(simstep - tij[(size_t)s * M], 0);
                  next = cell[(size_t)s * M];
                }
              };
              load(wt);
#pragma unroll 1
              for (int s = wt; s < C; s += kW) {
                const int pdt = pn;
                float4 q = next;
                load(s + kW);
                if (pdt < 0) continue;
                if (pdt > 0) {
                  float4 A, Bt;
                  double2 R0, R1;
                  entry(T, pdt, 0, A, Bt, R0, R1);
                  q = cell_step(q, T, A, Bt, R0, R1);
                }
                q.w += J.kftj;
                cell[(size_t)s * M] = q;
                tij[(size_t)s * M] = simstep;
              }
            }
          if (!kMulti && wt == 0) s_cols += (unsigned long long)nspk * C;
        }
      }
      if (kMulti) {
        __syncwarp();
        if (lane == 0) mb_arrive(s_F, it);
      }
    }
    bar(0, kThreads);
  }

  /* ---- the state back to the buffers of the last tick.  Q has seen every
     CTA's words of the tick before the last, so no CTA still reads what the
     launch began with (its first softmax seed, the spikes before it) ---- */
  if (s_abort) return;
  if (tid == 0) {
    if (s_rows) atomicAdd(&net->counters[0], s_rows);
    if (s_cols) atomicAdd(&net->counters[1], s_cols);
  }
  const int last = (rp->k0 + n_ticks - 1) & 1, next = last ^ 1;
#pragma unroll 1
  for (int k = 0; k < n_in; ++k) {
    const ProjDev& J = s_proj[k];
    const Block B = block<kQW>(sm, L, k, M, J.C);
    const size_t eoff = (size_t)J.proj_in_pop * n;
#pragma unroll 1
    for (int j = tid; j < M; j += kThreads) {
      const int idx = h * M + j;
      J.pj[idx] = B.pj[j];
      J.ej[idx] = B.ej[j];
      J.zj[idx] = B.zj[j];
      pop.epsc[last][eoff + idx] = B.epsc[last * M + j];
      pop.bj[last][eoff + idx] = B.bj[j];
    }
    const int part = queue_part(J.C, kQW), n0 = s_nl[k][next][0], words = kQW * part >> 5;
#pragma unroll 1
    for (int s = tid; s < J.C; s += kThreads) {
      if (B.src[s] == none) continue;
      uint32_t q = 0;
#pragma unroll 4
      for (int b = 0; b < 32; ++b) q |= ((B.plane[((n_ticks + b) & 31) * words + (s >> 5)] >> (s & 31)) & 1u) << b;
      J.qi[h * J.C + s] = (int)q;
    }
    const int cnt = kQW > 1 ? n0 + s_nl[k][next][kQW - 1] : n0;
    const uint16_t* l = B.list + next * kQW * part;
#pragma unroll 1
    for (int e = tid; e < cnt; e += kThreads) J.list[h * J.C + e] = h * J.C + (int)(e < n0 ? l[e] : l[part + e - n0]);
    if (tid == 0) J.list_cnt[h] = cnt;
  }
}

/* dynamic shared memory, in bytes, for the network's populations; kQW queue warps, `cells` per chunk */
inline size_t smem_bytes(int M, int n_in, const int* C, int n_words, int cells, int qw, bool multi) {
  Layout L;
  layout(M, n_in, C, n_words, cells, qw, multi, L);
  return (size_t)L.total * 4;
}

}  // namespace flow
}  // namespace bcpnn

#endif /* BCPNN_FLOW_CUH */
