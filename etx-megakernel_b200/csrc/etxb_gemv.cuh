// bf16 streaming GEMV family of the B200 megakernel: plain / norm-folded projections (QKV, O, router, lm_head),
// MoE gate+up with the SiLU*mul epilogue, MoE down with the routing-weight epilogue, and the softmax top-k.
//
// Function of the reference these tiles take over (same argument block, same task -> row mapping):
//   dsl_gemv / dsl_gemv_fold      etx/ops/gemv.py:816-840   (+ norm fold dsl_stage_norm_at, gemv.py:552-700)
//   dsl_moe_up[_fold]             etx/ops/gemv.py:841-911
//   dsl_moe_down[_fold]           etx/ops/gemv.py:912-953
//   dsl_topk / dsl_topk_lds       etx/ops/topk.py:35-156, etx/ops/gemv.py:712-749
// Rounding points are those of the reference's CPU numerical path (examples/llm/ref_numpy.py:105-158): every
// materialised vector is rounded to bf16, RMSNorm rounds twice, SiLU is rounded before the product, the routing
// weight is a bf16 value, expert outputs are accumulated in bf16 in ascending expert id.
//
// Weight streaming.  The weight rows of a task are one or two contiguous byte ranges.  The CTA's producer warp walks
// the task queue AHEAD of the consumer warps and copies those ranges, whole rows at a time, into a ring of
// ETXB_NSTAGE x 24 KB shared-memory stages with bulk asynchronous copies (cp.async.bulk, the TMA engine; completion
// on an mbarrier per stage).  Weights depend on no event (expert weights: only on the routing), so the stream keeps
// running while the consumers wait for their activations: HBM stays busy across phase boundaries.  A stage
// belongs to a group of 1 .. 16 consumer warps (GemvGeom), consecutive stages to different groups; a warp of the group
// multiplies 1, 3 or 4 of the stage's rows at once: 16-byte weight and activation vectors from shared memory, fp32
// accumulators in a fixed order (lane-strided, then xor butterfly), and hands the row results to the tile's epilogue.
#pragma once
#include "etxb_prims.cuh"

namespace etxb {

// ---------------------------------------------------------------------------------------------- what a task streams
// The weight rows of a task: `nranges` contiguous ranges of `n` rows each (row_bytes per row), taken range by range.
//   plain GEMV   one range: rows [r0, r0 + n) of W
//   MoE gate+up  per expert slot of the task: the gate rows, then the up rows (2 * spt ranges)
//   MoE down     per expert slot of the task: rows [r0, r0 + n) of that expert's W2 (spt ranges)
struct GemvTask {
  int nranges, n, row_bytes, r0, group, spt;
};
// How the consumer warps share a task's stages.  Worked out by one warp while the task's event is being waited for (the
// few integer divisions in it take longer than a short task's multiplications) and read by all through shared memory.
//   rps    rows per stage,  ns  stages of the task
//   W      warps per stage (a divisor of ETXB_EMPTY_COUNT),  NG <= min(16 / W, ETXB_NSTAGE) groups: group g takes stages g, g + NG, ..
//   R      rows a warp multiplies at once: rows wi, wi + W, .. of the stage
struct GemvGeom {
  GemvTask t;
  int rps, ns, W, NG, R, wmul;                                     // wmul: warp w belongs to group (w * wmul) >> 8
};

// What the tiles read of the running launch and task now and then: kept in shared memory, where it costs no registers.
struct CtaVars {
  int32_t* ctrl;
  uint64_t* tr;              // 8 stamps of the running task when tracing, else null (slots 4..7 are in-body marks)
  uint32_t epoch;            // the step (sharded sessions: the flag of this step's exchanged words derives from it)
  int cur;                   // the running task's index in the queue order (reported when a wait gives up)
  int q0, q1;                // the CTA's queue
  int done;                  // tasks of the queue before this one are over (kernels whose other tiles use the ring's memory too)
  int halt;                  // thread 0's word before a task: the step is being abandoned, everybody leaves the loop
  int hold;                  // the running task's results are on their way out: the producer starts no further stage (see produce_task)
};
struct Smem {
  float* xs;                 // general region (ETXB_GEN_BYTES): fp32 scratch, bf16 activations, row results
  float* scr;                // ETXB_SCR_FLOATS of reduction / routing scratch
  unsigned char* ring;       // ETXB_NSTAGE stages
  uint64_t* full;            // [ETXB_NSTAGE] stage filled (transaction bytes landed)
  uint64_t* empty;           // [ETXB_NSTAGE] stage drained by the warps it belongs to; behind it [8] uint32: the use the producer fills it for
  int32_t* prod;             // producer-warp scratch: 16 expert ids; from word 32 on the argument block of the task it copies for
  const unsigned long long* deadline;
  int* stop;                 // CTA-local: a wait inside a body gave up (the body's results are not to be announced)
  const GemvGeom* geo;       // the running GEMV-family task's rows and how the warps share them
  CtaVars* vars;       // null outside the persistent kernel
  __device__ __forceinline__ int32_t* ctrl() const { return vars->ctrl; }
  __device__ __forceinline__ uint64_t* tr() const { return vars ? vars->tr : nullptr; }
  __device__ __forceinline__ uint32_t epoch() const { return vars ? vars->epoch : 0u; }
  __device__ __forceinline__ int cur() const { return vars->cur; }
};
// in-body time stamp k (0..3) of the running task; thread 0 only, no-op unless tracing
__device__ __forceinline__ void mark(const Smem& sm, int k) { if (sm.tr() != nullptr && tidx() == 0) sm.tr()[4 + k] = globaltimer(); }
__device__ __forceinline__ __nv_bfloat16* smem_xb(const Smem& sm) { return (__nv_bfloat16*)((unsigned char*)sm.xs + ETXB_XB_OFF); }
__device__ __forceinline__ float* smem_g(const Smem& sm) { return (float*)((unsigned char*)sm.xs + ETXB_G_OFF); }

// Bounded mbarrier wait: true when the phase completed; false when the step is being abandoned (another thread gave
// up, the host aborted, or the deadline passed -- then this thread records it).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const Smem& sm, int where) {
  uint32_t n = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++n & 255u) == 0) {
      if (ld_relaxed(sm.ctrl()) != 0) { *(volatile int*)sm.stop = 1; return false; }
      if ((n & 4095u) == 0 && globaltimer() > *sm.deadline) {
        if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) { sm.ctrl()[1] = where; sm.ctrl()[2] = -1; sm.ctrl()[3] = (int32_t)parity; sm.ctrl()[4] = -1; }
        *(volatile int*)sm.stop = 1;
        return false;
      }
    }
  }
  return true;
}

// Bounded wait until the producer fills use k of a ring stage (its running stage count); gives up like mbar_wait.
__device__ __forceinline__ bool wait_use(volatile const uint32_t* use, uint32_t k, const Smem& sm, int where) {
  uint32_t n = 0;
  while (*use != k) {
    if ((++n & 255u) == 0) {
      if (ld_relaxed(sm.ctrl()) != 0) { *(volatile int*)sm.stop = 1; return false; }
      if ((n & 4095u) == 0 && globaltimer() > *sm.deadline) {
        if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) { sm.ctrl()[1] = where; sm.ctrl()[2] = -1; sm.ctrl()[3] = (int32_t)*use; sm.ctrl()[4] = (int32_t)k; }
        *(volatile int*)sm.stop = 1;
        return false;
      }
    }
  }
  return true;
}
// Bounded wait until the tasks of the queue before `cur` are over; gives up like mbar_wait.
__device__ __forceinline__ bool wait_done(const Smem& sm, int cur) {
  volatile const int* done = &sm.vars->done;
  uint32_t n = 0;
  while (*done < cur) {
    __nanosleep(20);
    if ((++n & 255u) == 0) {
      if (ld_relaxed(sm.ctrl()) != 0) return false;
      if ((n & 1023u) == 0 && globaltimer() > *sm.deadline) {
        if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) { sm.ctrl()[1] = cur; sm.ctrl()[2] = -1; sm.ctrl()[3] = *done; sm.ctrl()[4] = cur; }
        *(volatile int*)sm.stop = 1;
        return false;
      }
    }
  }
  return true;
}
// ---------------------------------------------------------------------------------------------- top-k
// softmax over E bf16 logits (fp32), K rounds of argmax with the lower index winning ties, optional renormalisation
// over the selected weights (numpy's summation order for <= 16 values), optional bf16 rounding of the weights.
// One warp (all 32 lanes call); E <= 256, K <= 16.  ids / wts / tei may point to shared or global memory.
template <int NK>
__device__ __forceinline__ void warp_topk_n(const void* logits, int E, int K, bool renorm, bool bf16w,
                                            int32_t* ids, float* wts, int32_t* tei) {
  const int lane = tidx() & 31;
  float p[NK];
  float m = -INFINITY;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const int e = lane + 32 * k;
    p[k] = e < E ? ld_bf(logits, e) : -INFINITY;
    m = fmaxf(m, p[k]);
  }
  m = warp_max(m);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < NK; ++k) { p[k] = (lane + 32 * k < E) ? expf(__fsub_rn(p[k], m)) : 0.f; s = __fadd_rn(s, p[k]); }
  s = warp_sum(s);
  // Selection keys: a probability is a non-negative float, so its bit pattern orders like the value; + 1 keeps a valid
  // zero probability above "no candidate" (0).  A candidate is the 64-bit pair (key, ~expert): the larger pair is the
  // larger probability or, on a tie, the lower expert.  Each lane sorts its NK candidates once (descending), so a
  // round only looks at the lanes' heads: a warp reduction (redux.sync) finds the winner, whose lane pops its head.
  // A NaN anywhere in the row makes the sum, and so every probability, NaN: no candidate is valid then and every round
  // writes id 0x7fffffff with weight -1 (the behaviour the reference's model pins for its wave path,
  // etx/ops/topk_key32.py:122-147; the expert tiles map such an id to expert 0 before they form an address).
  unsigned long long c[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const int e = lane + 32 * k;
    const float pq = __fdiv_rn(p[k], s);
    const uint32_t key = (e < E && pq == pq) ? __float_as_uint(pq) + 1u : 0u;
    c[k] = ((unsigned long long)key << 32) | (uint32_t)(0xffffffffu - (uint32_t)e);
  }
#pragma unroll
  for (int i = 1; i < NK; ++i)                                      // insertion network: c[0] >= c[1] >= ...
#pragma unroll
    for (int j = i; j > 0; --j) {
      const unsigned long long hi = c[j - 1] > c[j] ? c[j - 1] : c[j], lo = c[j - 1] > c[j] ? c[j] : c[j - 1];
      c[j - 1] = hi; c[j] = lo;
    }
  float myw = 0.f; int myid = 0x7fffffff;
#pragma unroll 1
  for (int t = 0; t < K; ++t) {
    const uint32_t hk = (uint32_t)(c[0] >> 32), hi_ = (uint32_t)c[0];
    const uint32_t top = __reduce_max_sync(0xffffffffu, hk);
    const uint32_t who = __ballot_sync(0xffffffffu, hk == top);
    uint32_t wl;
    if (who & (who - 1u)) wl = __reduce_max_sync(0xffffffffu, hk == top ? hi_ : 0u);    // (several lanes' heads are as probable)
    else wl = __shfl_sync(0xffffffffu, hi_, __ffs(who) - 1);
    const bool any = top != 0u;
    if (any && hk == top && hi_ == wl) {                            // the winner's lane pops its head
#pragma unroll
      for (int k = 0; k + 1 < NK; ++k) c[k] = c[k + 1];
      c[NK - 1] = 0ull;
    }
    if (lane == t) { myw = any ? __uint_as_float(top - 1u) : -1.f; myid = any ? (int)(0xffffffffu - wl) : 0x7fffffff; }
  }
  if (wts != nullptr && renorm) {
    // numpy's order for the sum of the K selected weights: K < 8 left to right, else 8 accumulators + tree + tail
    float tot;
    if (K < 8) {
      tot = 0.f;
#pragma unroll 1
      for (int t = 0; t < K; ++t) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, myw, t));
    } else {
      float r = lane < 8 ? myw : 0.f;                              // accumulator j = lane j
      const float second = __shfl_sync(0xffffffffu, myw, (lane & 7) + 8);
      if (K >= 16 && lane < 8) r = __fadd_rn(r, second);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, o));
      tot = __shfl_sync(0xffffffffu, r, 0);
#pragma unroll 1
      for (int t = (K >= 16 ? 16 : 8); t < K; ++t) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, myw, t));
    }
    myw = __fdiv_rn(myw, tot);
  }
  if (bf16w) myw = bfr(myw);
  if (lane < K) { ids[lane] = myid; if (wts != nullptr) wts[lane] = myw; if (tei) tei[lane] = lane; }
  __syncwarp();
}

// LEAN: the form the host picks when every top-k of the plan has E <= 128 (no code for more experts in that kernel).
template <bool LEAN>
__device__ __noinline__ void warp_topk(const void* logits, int E, int K, bool renorm, bool bf16w,
                                       int32_t* ids, float* wts, int32_t* tei) {
  if (LEAN || E <= 128) warp_topk_n<4>(logits, E, K, renorm, bf16w, ids, wts, tei);
  else warp_topk_n<8>(logits, E, K, renorm, bf16w, ids, wts, tei);
}

__device__ __forceinline__ void tile_topk(const unsigned char* a, int blk, const Smem& sm) {
  const etxb_topk_args& d = *(const etxb_topk_args*)a;
  if (blk >= (int)d.nblocks) return;
  const int nb = (d.nbsv & 0xff) ? (d.nbsv & 0xff) : 1, sv = d.nbsv >> 8;
  const int w = tidx() >> 5;
  if (w >= nb) return;
  warp_topk<false>((const __nv_bfloat16*)d.logits + (size_t)w * d.E, d.E, d.K, (d.mode & 0xff) == 1, (d.mode & ETXB_MODE_BF16_WTS) != 0,
            d.ids + (size_t)w * sv, d.wts + (size_t)w * sv, d.tei ? d.tei + (size_t)w * sv : nullptr);
}

// Decode task `blk` of a GEMV-family tile (pure arithmetic on the argument block).  Slots per task: mode bits 16..23
// (0 = 1): task blk covers slots [group * spt, (group + 1) * spt), group = blk / tpe, row chunk j = blk % tpe.
__device__ __forceinline__ GemvTask gemv_task(int body, const etxb_gemv_args& d, int blk) {
  GemvTask t;
  t.nranges = 0; t.n = 0; t.row_bytes = d.K * 2; t.r0 = 0; t.group = 0; t.spt = 1;
  if (blk >= (int)d.nblocks) return t;
  if (body == 3) {
    const int r0 = blk * d.rpt, r1 = min(d.M, r0 + d.rpt);
    if (r0 < r1) { t.nranges = 1; t.n = r1 - r0; t.r0 = r0; }
    return t;
  }
  const int spt = ((d.mode >> 16) & 0xff) ? ((d.mode >> 16) & 0xff) : 1;
  const int group = blk / d.tpe, j = blk - group * d.tpe;
  const int r0 = j * d.rpt, r1 = min(d.M, r0 + d.rpt);
  if (r0 < r1) { t.nranges = (body == 4 ? 2 : 1) * spt; t.n = r1 - r0; t.r0 = r0; t.group = group; t.spt = spt; }
  return t;
}

// a / b for 0 <= a < 2^22, b > 0: one approximate reciprocal and an exact correction (the compiler's integer division is
// several times as long).
__device__ __forceinline__ int udiv_small(int a, int b) {
  int q = __float2int_rz(__fdividef((float)a, (float)b));
  const int r = a - q * b;
  if (r < 0) --q; else if (r >= b) ++q;
  return q;
}
// Rows at once (R) and warps per stage (W): one row at a time is a chain of waits, shared-memory latencies and shuffles that
// 4 warps per scheduler do not hide; several rows share the activation vector with its unpacking and are reduced together.
// Rows of up to 1792 values (7 vectors per lane): 4 at once; of 2048 (6 rows per stage): 3; longer ones: a stage holds 5
// rows or fewer (of 4096: 3), one warp each (so too where every range has its own activation vector and 3 rows share nothing).  Clocks
// per task, weights already in the ring, against one row per warp and every warp on every stage:
// 35 rows of 2048: 5816 -> 3786; 8 x 14 rows of 768: 8972 -> 6486; 48 of 1536: 6277 -> 3701; 18 of 4096: 5420 -> 5293.
__device__ __forceinline__ void gemv_geom(int body, GemvGeom& g) {
  const int total = g.t.nranges * g.t.n;
  const int nvl = ((g.t.row_bytes >> 4) + 31) >> 5;
  g.rps = g.t.row_bytes > 0 && g.t.row_bytes <= ETXB_STAGE_BYTES ? udiv_small(ETXB_STAGE_BYTES, g.t.row_bytes) : 0;
  g.ns = 0; g.W = 1; g.NG = ETXB_NSTAGE; g.R = 1;
  if (total > 0 && g.rps > 0) {
    g.ns = total < (1 << 21) ? udiv_small(total + g.rps - 1, g.rps) : (total + g.rps - 1) / g.rps;
    g.R = nvl <= 7 ? 4 : (nvl <= 8 && !(body == 5 && g.t.nranges > 1) ? 3 : 1);
    const int m = min(g.rps, total);
    const int w = g.R == 4 ? (m + 3) >> 2 : (g.R == 3 ? udiv_small(m + 2, 3) : m);
    g.W = w <= 4 ? w : w <= 6 ? 6 : w <= 8 ? 8 : w <= 12 ? 12 : 16;
    g.NG = g.W <= 2 ? ETXB_NSTAGE : g.W == 3 ? 5 : g.W == 4 ? 4 : g.W <= 8 ? 2 : 1;
  }
  g.wmul = udiv_small(255 + g.W, g.W);                              // ceil(256 / W): exact for 16 warps and for ETXB_EMPTY_COUNT / W
}

// Expert ids (and routing weights, unless lwts is null) of the task's slots into `lids` / `lwts` (indexed by global slot).  One warp, all
// lanes call.  Top-k fold: recomputed from the logits; else read from the ids / wts buffers; no ids: expert 0.
// SH: the kernel variant supports always-on (shared) experts -- mode bits 24..27: ns experts that every token uses, stored
// after the E routed ones; they take the last ns slots with weight 1, the top-k picks the others.  (A template parameter
// and not a run-time branch: the lean kernels of the models without shared experts measured 1.4 % slower with it.)
template <bool LEAN, bool SH = !LEAN>
__device__ __forceinline__ void gemv_routing(const etxb_gemv_args& d, int32_t* lids, float* lwts) {
  const int fold = d.mode & 0xff, lane = tidx() & 31;
  if (fold >= 2) {
    if constexpr (SH) {
      const int ns = (d.mode >> 24) & 0xf;
      warp_topk<LEAN>(d.logits, d.E, d.R - ns, fold == 3, (d.mode & ETXB_MODE_BF16_WTS) != 0, lids, lwts, nullptr);
      if (ns > 0) {
        if (lane < ns) { lids[d.R - ns + lane] = d.E + lane; if (lwts != nullptr) lwts[d.R - ns + lane] = 1.f; }
        __syncwarp();
      }
    } else {
      warp_topk<LEAN>(d.logits, d.E, d.R, fold == 3, (d.mode & ETXB_MODE_BF16_WTS) != 0, lids, lwts, nullptr);
    }
  } else {
    if (lane < 16) {
      lids[lane] = (d.ids && lane < d.R) ? __ldcg(d.ids + lane) : 0;
      if (lwts != nullptr) lwts[lane] = (d.wts && lane < d.R) ? __ldcg(d.wts + lane) : 1.f;
    }
    __syncwarp();
  }
}

template <bool SH = true>
__device__ __forceinline__ const unsigned char* gemv_range_base(int body, const etxb_gemv_args& d, const GemvTask& t, int i, const int32_t* lids) {
  if (body == 3) return (const unsigned char*)d.W + (size_t)t.r0 * t.row_bytes;
  const int slot = t.group * t.spt + (body == 4 ? i >> 1 : i);
  int e = lids[slot];
  if (d.E > 0 && (unsigned)e >= (unsigned)(d.E + (SH ? ((d.mode >> 24) & 0xf) : 0))) e = 0;   // "no candidate" (a NaN row): never an address
  const unsigned char* We = (const unsigned char*)d.W + (size_t)e * d.estride * 2;
  const int row = t.r0 + ((body == 4 && (i & 1)) ? d.M : 0);        // up rows follow the M gate rows
  return We + (size_t)row * t.row_bytes;
}

// ---------------------------------------------------------------------------------------------- producer side
// Issue the bulk copies of one task.  One warp; lane 0 issues.  n = running stage counter of this CTA.
// ptr: the task's trace row when tracing (slot 7 <- time the first stage was issued, slot 6 <- the last), else null.
template <bool SH = true>
__device__ __forceinline__ bool produce_task(int body, const etxb_gemv_args& d, const GemvTask& t, int rps, const int32_t* lids, uint32_t& n,
                                             const Smem& sm, int where, uint64_t* ptr = nullptr) {
  const int total = t.nranges * t.n;
  if (total <= 0) return true;
  bool ok = true;
  if (rps < 1) {                                                   // a row longer than a stage: refused by the host; never loop on it
    if ((tidx() & 31) == 0) { atomicOr(sm.ctrl(), ETXB_CTRL_BADTASK); *(volatile int*)sm.stop = 1; }
    return false;
  }
  if ((tidx() & 31) == 0) {
    const uint64_t pol = l2_policy_evict_first();
    int rg = 0, r = 0;                                             // the range and the row in it that come next
    for (int q0 = 0; q0 < total && ok; q0 += rps) {
      const uint32_t st = n % ETXB_NSTAGE, par = (n / ETXB_NSTAGE) & 1;
      ok = mbar_wait(sm.empty + st, par ^ 1, sm, where);           // a fresh barrier passes the first round
      if (!ok) break;
      // A task's release waits for its stores to be acknowledged, and behind a full load queue that takes longer: after the
      // summed down tiles of a 128-expert model 2.4 us instead of 0.8, because the next layer's first projection streams into
      // every stage that falls free.  The last of those stages wait for the release (bounded: it is a matter of time only).
      // Asked of what follows a down tile and can be ahead of it, nothing else: in the expert grids' own streams the question
      // costs more than it gives (gate+up 12.5 -> 13.6 us).  (Not unrolled: the compiler's four copies of the wait are 4 KB of
      // code in this loop, and a step pays for them in instruction fetch whether it waits or not: 12 layers of a dense 4096-wide
      // model 1270 -> 1252 us without them, 9 of a latent-attention one 719 -> 709, 12 of a 128-expert one 700 -> 695.)
      if (body == 3 && q0 < ETXB_NSTAGE * rps)
#pragma unroll 1
        for (int spin = 0; spin < 64 && *(volatile const int*)&sm.vars->hold != 0; ++spin) __nanosleep(40);
      const int nr = min(rps, total - q0);
      unsigned char* dst = sm.ring + (size_t)st * ETXB_STAGE_BYTES;
      *((volatile uint32_t*)(sm.full + 2 * ETXB_NSTAGE) + st) = n;  // (see wait_use)
      mbar_expect_tx(sm.full + st, (uint32_t)(nr * t.row_bytes));
      for (int j = 0; j < nr;) {                                   // one copy per piece of a range that falls into this stage
        const int cnt = min(t.n - r, nr - j);
        bulk_g2s_hint(dst + (size_t)j * t.row_bytes, gemv_range_base<SH>(body, d, t, rg, lids) + (size_t)r * t.row_bytes,
                      (uint32_t)(cnt * t.row_bytes), sm.full + st, pol);
        j += cnt;
        r += cnt;
        if (r == t.n) { r = 0; ++rg; }
      }
      if (ptr != nullptr) { if (q0 == 0) ptr[7] = globaltimer(); ptr[6] = globaltimer(); }
      ++n;
    }
  }
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  n = __shfl_sync(0xffffffffu, n, 0);
  return ok;
}

// ---------------------------------------------------------------------------------------------- consumer side
__device__ __forceinline__ float dot8(const uint4 w, const uint4 x, float a) {
  a = __fmaf_rn(bf_lo(w.x), bf_lo(x.x), a); a = __fmaf_rn(bf_hi(w.x), bf_hi(x.x), a);
  a = __fmaf_rn(bf_lo(w.y), bf_lo(x.y), a); a = __fmaf_rn(bf_hi(w.y), bf_hi(x.y), a);
  a = __fmaf_rn(bf_lo(w.z), bf_lo(x.z), a); a = __fmaf_rn(bf_hi(w.z), bf_hi(x.z), a);
  a = __fmaf_rn(bf_lo(w.w), bf_lo(x.w), a); a = __fmaf_rn(bf_hi(w.w), bf_hi(x.w), a);
  return a;
}

// What happens to a row's result: the epilogue of the three tiles (held in registers: a pointer to a struct would put it
// on the stack, and beside 227 KB of shared memory the L1 that backs the stack is small).
struct GemvEpi {
  int body;                  // 3, 4, 5
  int M;                     // down: rows of an expert's output
  __nv_bfloat16* out;        // gemv: row 0 of the task;  down, not summed: slot 0, row 0 of the task
  const void* aux;           // gemv: bias of row 0 of the task (bf16);  down: routing weight per slot of the task (fp32);  or null
  float* g;                  // up: bf16-rounded results per row;  down: weighted results per row when they are summed, else null
};
__device__ __forceinline__ void gemv_epi(const GemvEpi& e, int q, int rg, int rows, float v) {
  if (e.body == 3) {
    e.out[q] = __float2bfloat16_rn(e.aux ? __fadd_rn(v, __bfloat162float(((const __nv_bfloat16*)e.aux)[q])) : v);
  } else {
    float y = bfr(v);
    if (e.aux) y = bfr(__fmul_rn(y, ((const float*)e.aux)[rg]));
    if (e.g) e.g[q] = y;
    else e.out[(size_t)rg * e.M + (q - rg * rows)] = __float2bfloat16_rn(y);
  }
}

// Rows j, j + W, .. (R of them, those past the stage's nr repeat the last one and are dropped) of one stage by one warp.
// XS: a row's activation vector is its range's (xb + range * xstride), else one vector serves all.  rg, rgend: the range
// of the warp's current row and the row where it ends.
template <int R, bool XS>
__device__ __forceinline__ void gemv_rows(const unsigned char* stage, int row_bytes, int j, int W, int nr, int q0, int rows, int& rg, int& rgend,
                                          const __nv_bfloat16* xb, int xstride, const GemvEpi& e) {
  const int lane = tidx() & 31, nvec = row_bytes >> 4;
  const uint4* wv[R];
  const uint4* xv[XS ? R : 1];
  int rgu[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int jj = min(j + u * W, nr - 1);
    wv[u] = (const uint4*)(stage + (size_t)jj * row_bytes);
    rgu[u] = 0;
    if (XS) {
      while (q0 + jj >= rgend) { ++rg; rgend += rows; }
      rgu[u] = rg;
      xv[u] = (const uint4*)(xb + (size_t)rg * xstride);
    }
  }
  if (!XS) xv[0] = (const uint4*)xb;
  float a[R];
#pragma unroll
  for (int u = 0; u < R; ++u) a[u] = 0.f;
  constexpr int U = R == 1 ? 4 : 1;
#pragma unroll U
  for (int v = lane; v < nvec; v += 32) {
    if (XS) {
#pragma unroll
      for (int u = 0; u < R; ++u) a[u] = dot8(wv[u][v], xv[u][v], a[u]);
    } else {
      const uint4 x = xv[0][v];
#pragma unroll
      for (int u = 0; u < R; ++u) a[u] = dot8(wv[u][v], x, a[u]);
    }
  }
  if constexpr (R == 1) {
    const float s = warp_sum(a[0]);
    if (lane == 0) gemv_epi(e, q0 + j, rgu[0], rows, s);
  } else {
    // the butterfly of warp_sum on R values at once: the lanes split the values between them at distances 16 and 8, then
    // 4, 2, 1 as usual -- the same sums in the same order, 6 shuffles instead of 5 R
    static_assert(R == 3 || R == 4, "the exchange below splits up to four values");
    const bool h16 = lane & 16, h8 = lane & 8;
    const float a3 = R == 4 ? a[R - 1] : 0.f;
    float k0 = h16 ? a[2] : a[0], k1 = h16 ? a3 : a[1];
    k0 += __shfl_xor_sync(0xffffffffu, h16 ? a[0] : a[2], 16);
    k1 += __shfl_xor_sync(0xffffffffu, h16 ? a[1] : a3, 16);
    float k = h8 ? k1 : k0;
    k += __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    const int u = (h16 ? 2 : 0) + (h8 ? 1 : 0), jj = j + u * W;
    if ((lane & 7) == 0 && u < R && jj < nr) {
      int r = rgu[0];
#pragma unroll
      for (int i = 1; i < R; ++i) r = u == i ? rgu[i] : r;
      gemv_epi(e, q0 + jj, r, rows, k);
    }
  }
}

// Consume the stages of one task: row q (0 .. total-1, range q / rows) . its activation vector -> gemv_epi.
// Range i uses the vector at xb + i * xstride (xstride = 0: one vector for all).  A stage is waited for, read and given
// back by its group's W warps only (each arrives ETXB_EMPTY_COUNT / W times); the stage counter runs on by the task's
// stages in every warp.
// (Measured and not kept: the packed fma.rn.f32x2 form of the inner loop, +1.3 % step time; the mixed fma.rn.f32.bf16,
// which needs no unpacking but issues at about a quarter of the rate: 39 -> 41 bytes per clock with one row; a lane's
// share of the activations in registers, which spills at the 96 registers this kernel gets; a ring of 7 stages instead of 6,
// +0.6 %; mma.sync m16n8k16 with conflict-free unpadded rows (row r reads the 16-byte chunks in the order c ^ r and column r
// of B holds the activations in that order): 3800 clocks for 35 rows of 2048, with an error 1.2 times as large; this function as a
// call, one copy for all tiles: its arguments and saved registers on the stack cost 2 us per phase.)
__device__ __forceinline__ void consume_task(uint32_t& n, const Smem& sm, const __nv_bfloat16* xb, int xstride, int where, const GemvEpi& e) {
  const int lane = tidx() & 31, cw = tidx() >> 5;
  const GemvGeom& geo = *sm.geo;
  const int W = geo.W, NG = geo.NG, g = (cw * geo.wmul) >> 8, wi = cw - g * W;
  const int rows = geo.t.n, total = geo.t.nranges * rows, rps = geo.rps, row_bytes = geo.t.row_bytes, R = geo.R;
  const uint32_t n0 = n;
  n += (uint32_t)geo.ns;
  if (g >= NG) return;
  const uint32_t cnt = (uint32_t)ETXB_EMPTY_COUNT * (uint32_t)geo.wmul >> 8;   // 48 / W
  uint32_t st = n0 % ETXB_NSTAGE, par = (n0 / ETXB_NSTAGE) & 1, k = n0 + g;
  st += g;
  while (st >= ETXB_NSTAGE) { st -= ETXB_NSTAGE; par ^= 1; }
  volatile const uint32_t* use = (volatile const uint32_t*)(sm.full + 2 * ETXB_NSTAGE);
  int rg = 0, rgend = rows;
  for (int q0 = g * rps; q0 < total; q0 += NG * rps) {
    // A parity wait tells use k of a stage from use k - 1 only, and with a number of groups that does not divide the ring
    // the use before this one may be another group's that is still being filled: the wait would be answered by use k - 2.
    // So the producer's note of the use it fills is looked at first (when it names k, k - 1 is over).
    if (ETXB_NSTAGE % NG != 0 && !wait_use(use + st, k, sm, where)) return;
    if (!mbar_wait(sm.full + st, par, sm, where)) return;          // step abandoned: touch nothing
    if (q0 == 0) mark(sm, 1);
    const int nr = min(rps, total - q0);
    const unsigned char* stage = sm.ring + (size_t)st * ETXB_STAGE_BYTES;
    for (int j = wi; j < nr; j += R * W) {
      if (xstride != 0) {
        if (R == 4) gemv_rows<4, true>(stage, row_bytes, j, W, nr, q0, rows, rg, rgend, xb, xstride, e);
        else gemv_rows<1, true>(stage, row_bytes, j, W, nr, q0, rows, rg, rgend, xb, xstride, e);
      } else if (R == 4) gemv_rows<4, false>(stage, row_bytes, j, W, nr, q0, rows, rg, rgend, xb, 0, e);
      else if (R == 3) gemv_rows<3, false>(stage, row_bytes, j, W, nr, q0, rows, rg, rgend, xb, 0, e);
      else gemv_rows<1, false>(stage, row_bytes, j, W, nr, q0, rows, rg, rgend, xb, 0, e);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_n(sm.empty + st, cnt);
    st += NG; k += NG;
    while (st >= ETXB_NSTAGE) { st -= ETXB_NSTAGE; par ^= 1; }
  }
}

// ---------------------------------------------------------------------------------------------- activation staging
// K bf16 values (written by other CTAs) -> shared memory, K % 8 == 0.
__device__ __forceinline__ void stage_xb(const void* x, int K, __nv_bfloat16* xb) {
  const int nv = K >> 3;
  for (int i = tidx(); i < nv; i += ETXB_CONSUMERS) ((uint4*)xb)[i] = ld_act16((const __nv_bfloat16*)x + 8 * i);
  csync();
}

// Norm fold: z = bf16(resid_in + acc), acc = the R rows added one by one in bf16 in ascending id order (R == 1: the row
// itself; rows == null: z = resid_in), then x = bf16(ln * bf16(z * r)), r = 1 / sqrt(mean(z^2) + eps) with the mean summed
// in numpy's order.  x goes to shared memory (xb); `store`: this task also writes resid_out (z) and xout (x).  K <= 8192.
// LEAN: the form the host picks when every norm fold of the plan adds at most one row (R <= 1): no ordering, no row loop.
// fl != 0 (sharded model): `rows` holds R rows of K flagged words published by the ranks (row r by rank r); every word is
// re-read until its flag is `fl` (bounded like every wait: on a give-up the step is abandoned through sm.stop), then the
// rows are added in rank order -- every rank adds the same values in the same order and gets the same bits.
// XCH: the kernel variant of a sharded session; without it the flagged form is compiled out (the single-GPU kernels
// carry none of the exchange code: it cost them about 5 % when it was a run-time branch).
template <bool LEAN, bool XCH = false>
__device__ __forceinline__ void stage_norm_col(const void* rows, const void* rin, void* rout, void* xout, const void* ln,
                                            const int32_t* ids, int R, int K, float eps, float* xf, __nv_bfloat16* xb, float* scr, bool store,
                                            uint32_t fl = 0u, const Smem* smp = nullptr) {
  int* order = (int*)(scr + 64);
  if (!LEAN && R > 1 && (!XCH || fl == 0u)) {
    if (R <= 32) {
      // one load per lane, the other ids by shuffle (no loop of R loads from L2 in front of the rows)
      if (tidx() < 32) {
        const int lane = tidx();
        const int mine = (ids && lane < R) ? __ldcg(ids + lane) : 0;
        int rank = ids ? 0 : lane;
        if (ids)
          for (int j = 0; j < R; ++j) {
            const int o = __shfl_sync(0xffffffffu, mine, j);
            rank += (o < mine) || (o == mine && j < lane);
          }
        if (lane < R) order[rank] = lane;
      }
    } else if (tidx() < R) {
      int rank = tidx();
      if (ids) {
        const int mine = __ldcg(ids + tidx());
        rank = 0;
        for (int j = 0; j < R; ++j) {
          const int o = __ldcg(ids + j);
          rank += (o < mine) || (o == mine && j < tidx());
        }
      }
      order[rank] = tidx();
    }
    csync();
  }
  const int nv = K >> 3, pad = K <= 4096 ? 8 : 0;                  // (blocks of 128 values apart: see sumsq_numpy_order)
  uint4 lw0 = make_uint4(0, 0, 0, 0), lw1 = lw0;                   // norm weights of this thread's (at most two) vectors, fetched with the rows
#pragma unroll 1
  for (int i = tidx(), it = 0; i < nv; i += ETXB_CONSUMERS, ++it) {
    float z[8];
    const uint4 lwi = __ldg((const uint4*)((const __nv_bfloat16*)ln + 8 * i));
    if (it == 0) lw0 = lwi; else lw1 = lwi;
    const uint4 ri = ld_act16((const __nv_bfloat16*)rin + 8 * i);
    const float rf[8] = {bf_lo(ri.x), bf_hi(ri.x), bf_lo(ri.y), bf_hi(ri.y), bf_lo(ri.z), bf_hi(ri.z), bf_lo(ri.w), bf_hi(ri.w)};
    if (rows == nullptr || R == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) z[j] = rf[j];
    } else if (XCH && fl != 0u) {
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll 1
      for (int s0 = 0; s0 < R; ++s0) {
        const uint32_t* src = (const uint32_t*)rows + (size_t)s0 * K + 8 * i;
        uint4 a, b;
        uint32_t spins = 0;
        for (;;) {
          a = ld_volatile16(src); b = ld_volatile16(src + 4);
          if ((((a.x ^ fl) | (a.y ^ fl) | (a.z ^ fl) | (a.w ^ fl) | (b.x ^ fl) | (b.y ^ fl) | (b.z ^ fl) | (b.w ^ fl)) >> 16) == 0u) break;
          if ((++spins & 63u) == 0) {
            if (ld_relaxed(smp->ctrl()) != 0) { *(volatile int*)smp->stop = 1; break; }
            if ((spins & 1023u) == 0 && globaltimer() > *smp->deadline) {
              if (atomicOr(smp->ctrl(), ETXB_CTRL_TIMEOUT) == 0) { smp->ctrl()[1] = smp->cur(); smp->ctrl()[2] = -2 - s0; smp->ctrl()[3] = (int32_t)(a.x >> 16); smp->ctrl()[4] = (int32_t)(fl >> 16); }
              *(volatile int*)smp->stop = 1;
              break;
            }
            __nanosleep(32);
          }
        }
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = bfr(__fadd_rn(acc[j], __uint_as_float(w[j] << 16)));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) z[j] = bfr(__fadd_rn(rf[j], acc[j]));
    } else if (LEAN) {
      const uint4 rv = ld_act16((const __nv_bfloat16*)rows + 8 * i);
      const float v[8] = {bf_lo(rv.x), bf_hi(rv.x), bf_lo(rv.y), bf_hi(rv.y), bf_lo(rv.z), bf_hi(rv.z), bf_lo(rv.w), bf_hi(rv.w)};
#pragma unroll
      for (int j = 0; j < 8; ++j) z[j] = bfr(__fadd_rn(rf[j], v[j]));      // bf16(0 + row) = row: the one-row case of the loop below
    } else {
      constexpr int NF = 8;
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll 1
      for (int s0 = 0; s0 < R; s0 += NF) {                      // NF rows in flight, added in order
        uint4 rv[NF];
#pragma unroll
        for (int u = 0; u < NF; ++u) {
          const int row = R > 1 ? order[min(s0 + u, R - 1)] : 0;
          rv[u] = ld_act16((const __nv_bfloat16*)rows + (size_t)row * K + 8 * i);
        }
#pragma unroll
        for (int u = 0; u < NF; ++u)
          if (s0 + u < R) {
            const float v[8] = {bf_lo(rv[u].x), bf_hi(rv[u].x), bf_lo(rv[u].y), bf_hi(rv[u].y),
                                bf_lo(rv[u].z), bf_hi(rv[u].z), bf_lo(rv[u].w), bf_hi(rv[u].w)};
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = bfr(__fadd_rn(acc[j], v[j]));
          }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) z[j] = bfr(__fadd_rn(rf[j], acc[j]));
    }
    float* zx = xf + 8 * i + (i >> 4) * pad;
    *(float4*)zx = make_float4(z[0], z[1], z[2], z[3]);
    *(float4*)(zx + 4) = make_float4(z[4], z[5], z[6], z[7]);
    if (store && rout != nullptr)
      *(uint4*)((__nv_bfloat16*)rout + 8 * i) = make_uint4(pack_bf(z[0], z[1]), pack_bf(z[2], z[3]), pack_bf(z[4], z[5]), pack_bf(z[6], z[7]));
  }
  csync();
  const float ss = sumsq_numpy_order<true>(xf, K, scr, pad);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
#pragma unroll 1
  for (int i = tidx(), it = 0; i < nv; i += ETXB_CONSUMERS, ++it) {
    const uint4 w = it == 0 ? lw0 : lw1;
    const float wf[8] = {bf_lo(w.x), bf_hi(w.x), bf_lo(w.y), bf_hi(w.y), bf_lo(w.z), bf_hi(w.z), bf_lo(w.w), bf_hi(w.w)};
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bfr(__fmul_rn(wf[j], bfr(__fmul_rn(xf[8 * i + (i >> 4) * pad + j], r))));
    const uint4 o = make_uint4(pack_bf(v[0], v[1]), pack_bf(v[2], v[3]), pack_bf(v[4], v[5]), pack_bf(v[6], v[7]));
    ((uint4*)xb)[i] = o;
    if (store && xout != nullptr) *(uint4*)((__nv_bfloat16*)xout + 8 * i) = o;
  }
  csync();
}

// ---------------------------------------------------------------------------------------------- the tiles
// body 3, plain / folded GEMV: out[r] = bf16(W[r,:].x + bias[r]).
// body 4, MoE gate+up.  task blk: expert slots [group * spt, ...), row chunk j = blk % tpe; expert e = ids[slot] (no ids and
//   no fold: expert 0, the dense SwiGLU MLP); act[slot][r] = bf16(bf16(silu(bf16 g)) * bf16 u), g = W_e[r,:].x, u = W_e[M + r,:].x.
// body 5, MoE down.  y[slot][r] = bf16(bf16(W_e[r,:] . act_slot) * wts[slot]) (no weights, the dense MLP: bf16(W_e[r,:] . act)).
//   Plain form: out[slot][r] = y.  Summed form (mode bit ETXB_MODE_SUM_SLOTS, the task covers every slot): out[r] = the
//   y of all slots added one by one in bf16 in ascending expert id -- the expert combine of the CPU path
//   (examples/llm/ref_numpy.py:142-148), which the reference leaves to the next layer's norm fold.
// One function with one copy of the multiplication: the phases of a step share its code, so it stays in the instruction
// cache from one to the next.
template <bool LEAN, bool XCH = false, bool SH = !LEAN>
__device__ __forceinline__ void tile_gemv_family(int body, const unsigned char* a, int blk, const Smem& sm, uint32_t& n, int where) {
  const etxb_gemv_args& d = *(const etxb_gemv_args*)a;
  const GemvTask& t = sm.geo->t;
  if (t.n <= 0) return;
  int32_t* lids = (int32_t*)(sm.scr + 96); float* lwts = sm.scr + 112;
  const int fold = d.mode & 0xff, rows = t.n, K = d.K, spt = t.spt;
  __nv_bfloat16* xb = smem_xb(sm);
  float* g = smem_g(sm);                                           // up: per slot, rows gate results, then rows up results;  down: rows per slot
  GemvEpi e;
  e.body = body; e.M = d.M; e.out = (__nv_bfloat16*)d.out; e.aux = nullptr; e.g = nullptr;
  const bool sum = body == 5 && (d.mode & ETXB_MODE_SUM_SLOTS) != 0;
  if (body != 3 && tidx() < 32) {
    if (body == 5 && fold >= 2 && (d.mode & ETXB_MODE_ROUTE_READY) && d.ids != nullptr && d.wts != nullptr) {
      if (tidx() < 16) {
        lids[tidx()] = tidx() < d.R ? __ldcg(d.ids + tidx()) : 0;
        lwts[tidx()] = tidx() < d.R ? __ldcg(d.wts + tidx()) : 1.f;
      }
      __syncwarp();
    } else if (body == 5 || (fold >= 2 && blk - t.group * d.tpe == 0)) {    // (gate+up needs the routing only to publish it)
      gemv_routing<LEAN, SH>(d, lids, lwts);
    }
    if (body == 4 && fold >= 2 && blk - t.group * d.tpe == 0 && tidx() < spt) {   // the group's first chunk publishes its slots' routing
      const int sl = t.group * spt + tidx();
      if (d.ids) ((int32_t*)d.ids)[sl] = lids[sl];
      if (d.wts) ((float*)d.wts)[sl] = lwts[sl];
    }
    // the slots in ascending expert id, for the summed form (as the row of g where the slot's results begin): known as soon
    // as the routing is, so it is worked out here, under the weight stream, and not after it
    if (sum && tidx() < spt) {
      const int mine = lids[t.group * spt + tidx()];
      int rank = 0;
      for (int j = 0; j < spt; ++j) {
        const int o = lids[t.group * spt + j];
        rank += (o < mine) || (o == mine && j < tidx());
      }
      ((int*)(sm.scr + 64))[rank] = tidx() * rows;
    }
  }
  if (body == 5) {
    for (int i = tidx(); i < spt * (K >> 3); i += ETXB_CONSUMERS)             // the task's slots' activation vectors, one behind the other
      ((uint4*)xb)[i] = ld_act16((const __nv_bfloat16*)d.x + (size_t)t.group * spt * K + 8 * i);
    csync();
    e.out += (size_t)t.group * spt * d.M + t.r0;
    e.g = sum ? g : nullptr;
    e.aux = fold >= 2 || d.wts != nullptr ? lwts + t.group * spt : nullptr;
    if (sum) e.out -= (size_t)t.group * spt * d.M;                 // (the summed form writes one row)
  } else {
    if (fold == ETXB_MODE_NORM)                                    // (a dense MLP's gate+up: the post-attention norm folded in)
      stage_norm_col<LEAN, XCH>(d.rows, d.resid_in, d.resid_out, (void*)d.x, d.ln, body == 3 ? d.ids : nullptr, d.R, K, d.eps, sm.xs, xb, sm.scr, blk == 0,
                                (XCH && (d.mode & ETXB_MODE_FLAGGED)) ? row_flag(sm.epoch()) : 0u, &sm);
    else
      stage_xb(d.x, K, xb);
    if (body == 3) {
      e.out += t.r0;
      e.aux = (d.mode & ETXB_MODE_BIAS) ? (const __nv_bfloat16*)d.wts + t.r0 : nullptr;
    } else {
      e.g = g;
    }
  }
  mark(sm, 0);
  consume_task(n, sm, xb, body == 5 && t.nranges > 1 ? K : 0, where, e);
  if (body == 3 || (body == 5 && !sum)) return;
  csync();
  if (body == 5 && tidx() == 0) *(volatile int*)&sm.vars->hold = 1;
  mark(sm, 2);
  if (body == 4) {
    __nv_bfloat16* act = e.out + (size_t)t.group * spt * e.M + t.r0;
    for (int s = 0, r = tidx(); s < spt; ++s, r -= rows, act += e.M, g += 2 * rows)
      for (; r < rows; r += ETXB_CONSUMERS) act[r] = __float2bfloat16_rn(__fmul_rn(bfr(silu_f(g[r])), g[rows + r]));
  } else {
    const int* order = (const int*)(sm.scr + 64);
    for (int r = tidx(); r < rows; r += ETXB_CONSUMERS) {
      float acc = 0.f;
      for (int k0 = 0; k0 < spt; k0 += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = g[order[min(k0 + k, spt - 1)] + r];
#pragma unroll
        for (int k = 0; k < 8; ++k) if (k0 + k < spt) acc = bfr(__fadd_rn(acc, v[k]));
      }
      e.out[r] = __float2bfloat16_rn(acc);
    }
  }
}

}  // namespace etxb
