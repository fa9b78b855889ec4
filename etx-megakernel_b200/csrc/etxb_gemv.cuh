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
// multiplies 1, 3 or 4 of the stage's rows at once, or a part of them: 16-byte weight and activation vectors from shared memory, fp32
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
//   rps    rows per stage (at most),  ns  stages of the task,  spr  stages per range where no stage crosses a range's end, else 0
//   W      warps per stage (a divisor of ETXB_EMPTY_COUNT),  NG <= min(16 / W, ETXB_NSTAGE) groups: group g takes stages g, g + NG, ..
//   S      warps that share a row: warp h of them multiplies the vectors h * 32 + lane, (h + S) * 32 + lane, ..
//   R      rows a warp multiplies at once: rows wi / S, wi / S + rw, .. of the stage, rw = W / S
struct __align__(16) GemvGeom {
  GemvTask t;
  int rps, ns, W, NG, R, S, rw, spr;
  int wmul;                                                        // warp w belongs to group (w * wmul) >> 8
  int cnt, shared;                                                 // arrivals of a warp per stage; a stage's uses may belong to different groups (see consume_task)
  int few;                                                         // at most 16 rows, of at most 2048 values
  int direct;                                                      // results go straight to memory: a plain task whose vector nobody takes as words
  int one;                                                         // rows longer than 2048 values that go one at a time
  float rspr;                                                      // 1 / spr (0: no ranges): stage s belongs to range (s + 0.5) * rspr
};

// What the tiles read of the running launch and task now and then: kept in shared memory, where it costs no registers.
struct CtaVars {
  int32_t* ctrl;
  uint64_t* tr;              // 8 stamps of the running task when tracing, else null (slots 4..7 are in-body marks)
  uint32_t serial;           // number of the launch in the process (flags of attention partials)
  uint32_t flag;             // flag of this step's words: of the hand-off on this GPU, and of the rows a sharded session exchanges
  int cur;                   // the running task's index in the queue order (reported when a wait gives up)
  int q0, q1;                // the CTA's queue
  int done;                  // tasks of the queue before this one are over (kernels whose other tiles use the ring's memory too)
  int halt;                  // thread 0's word before a task: the step is being abandoned, everybody leaves the loop
  int hold;                  // the running task's results are on their way out: the producer starts no further stage (see produce_task)
};
struct Smem {
  float* xs;                 // general region (ETXB_GEN_BYTES): fp32 scratch, then the rows' results; bf16 activations behind it
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
  __device__ __forceinline__ uint32_t serial() const { return vars ? vars->serial : 0u; }
  __device__ __forceinline__ int cur() const { return vars->cur; }
};
// The persistent kernel's shared memory beside the dynamic part.  At namespace scope so that the tiles that are calls find
// it at known addresses too: passed by reference, Smem would live on the stack; passed by value, in registers.
__shared__ int s_stop;
__shared__ unsigned long long s_deadline;
__shared__ GemvGeom s_geo;
__shared__ CtaVars s_vars;
// in-body time stamp k (0..3) of the running task; thread 0 only, no-op unless tracing
__device__ __forceinline__ void mark(const Smem& sm, int k) { if (tidx() == 0 && sm.tr() != nullptr) sm.tr()[4 + k] = globaltimer(); }
__device__ __forceinline__ __nv_bfloat16* smem_xb(const Smem& sm) { return (__nv_bfloat16*)((unsigned char*)sm.xs + ETXB_XB_OFF); }

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
// Between two looks at words that are not there yet: false when the step is being abandoned (see mbar_wait).
__device__ __noinline__ bool words_again(uint32_t& spins, uint32_t fl) {
  if ((++spins & 63u) == 0) {
    int32_t* ctrl = s_vars.ctrl;
    if (ld_relaxed(ctrl) != 0) { *(volatile int*)&s_stop = 1; return false; }
    if ((spins & 1023u) == 0 && globaltimer() > s_deadline) {
      if (atomicOr(ctrl, ETXB_CTRL_TIMEOUT) == 0) { ctrl[1] = s_vars.cur; ctrl[2] = -4; ctrl[3] = 0; ctrl[4] = (int32_t)(fl >> 16); }
      *(volatile int*)&s_stop = 1;
      return false;
    }
    __nanosleep(32);
  }
  return true;
}
__device__ __forceinline__ uint32_t poll_word(const uint32_t* p, uint32_t fl) {
  uint32_t v, spins = 0;
  do v = ld_word(p); while (((v ^ fl) >> 16) != 0u && words_again(spins, fl));
  return v;
}
__device__ __forceinline__ uint4 poll_words4(const uint32_t* p, uint32_t fl) {
  uint4 v;
  uint32_t spins = 0;
  do v = ld_words4(p); while (words_miss(v, fl) != 0u && words_again(spins, fl));
  return v;
}
// ---------------------------------------------------------------------------------------------- top-k
// softmax over E bf16 logits (fp32), K rounds of argmax with the lower index winning ties, optional renormalisation
// over the selected weights (numpy's summation order for <= 16 values), optional bf16 rounding of the weights.
// One warp (all 32 lanes call); E <= 256, K <= 16.  fl: 0, or the flag of the words that `logits` names.  ids / wts / tei may point to shared or global memory.
// The ids alone, as a stream of expert rows waits for them: ordered by the logits themselves, value and index in one 24-bit key, a reduction per round.
// The probabilities order alike unless two distinct logits among the K best and the next one become one probability: closer than 2^-14 (l - max is
// rounded to 2^-18 at most within the range asked for), or so far below the maximum that they underflow.  Then, and where a logit is NaN or the maximum
// infinite, nothing is written and false is returned.  One warp.  (Softmax, 64-bit candidates and two or three exchanges a round: the first expert rows
// of a 128-expert layer were asked for 2.9 us after the router's event, so after 2.3.)
template <int NK>
__device__ __forceinline__ bool topk_ids_by_logit(const float (&p)[NK], int E, int K, int32_t* ids) {
  const int lane = tidx() & 31;
  uint32_t c[NK];
  bool nan = false;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const int e = lane + 32 * k;
    const uint32_t u = __float_as_uint(__fadd_rn(p[k], 0.f)) >> 16;  // (-0 and +0 are one logit)
    nan = nan || (e < E && p[k] != p[k]);
    c[k] = e < E ? ((u & 0x8000u ? ~u & 0xffffu : u | 0x8000u) << 8) | (uint32_t)(255 - e) : 0u;
  }
  if (__any_sync(0xffffffffu, nan)) return false;
#pragma unroll
  for (int i = 1; i < NK; ++i)                                      // c[0] >= c[1] >= ...
#pragma unroll
    for (int j = i; j > 0; --j) { const uint32_t hi = max(c[j - 1], c[j]), lo = min(c[j - 1], c[j]); c[j - 1] = hi; c[j] = lo; }
  const int n = min(K + 1, E);
  uint32_t mine = 0u;
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    const uint32_t top = __reduce_max_sync(0xffffffffu, c[0]);
    if (c[0] == top) {                                              // (keys are unique: one lane pops its head)
#pragma unroll
      for (int k = 0; k + 1 < NK; ++k) c[k] = c[k + 1];
      c[NK - 1] = 0u;
    }
    if (lane == t) mine = top;
  }
  const uint32_t u = mine >> 8;
  const float l = __uint_as_float((u & 0x8000u ? u & 0x7fffu : ~u & 0xffffu) << 16);
  const float m = __shfl_sync(0xffffffffu, l, 0), d = __fsub_rn(l, __shfl_down_sync(0xffffffffu, l, 1));
  const bool bad = lane < n && (!(m < INFINITY) || !(__fsub_rn(l, m) >= -80.f) || (lane + 1 < n && !(d == 0.f || d >= 6.103515625e-5f)));
  if (__any_sync(0xffffffffu, bad)) return false;
  if (lane < K) ids[lane] = 255 - (int)(mine & 0xffu);
  __syncwarp();
  return true;
}

template <int NK, bool GEMV>
__device__ __forceinline__ void warp_topk_n(const void* logits, uint32_t fl, int E, int K, bool renorm, bool bf16w,
                                            int32_t* ids, float* wts, int32_t* tei) {
  const int lane = tidx() & 31;
  float p[NK];
  float m = -INFINITY;
  if (GEMV && fl != 0u) {                                          // (all loads, then a look at their flags)
    uint32_t u[NK], spins = 0, miss;
    do {
      miss = 0u;
#pragma unroll
      for (int k = 0; k < NK; ++k) u[k] = ld_word((const uint32_t*)logits + min(lane + 32 * k, E - 1));
#pragma unroll
      for (int k = 0; k < NK; ++k) miss |= (u[k] ^ fl) >> 16;
    } while (miss != 0u && words_again(spins, fl));
#pragma unroll
    for (int k = 0; k < NK; ++k) p[k] = bf_lo(u[k]);
  } else {
#pragma unroll
    for (int k = 0; k < NK; ++k) p[k] = ld_bf(logits, min(lane + 32 * k, E - 1));
  }
  if (GEMV && wts == nullptr && topk_ids_by_logit<NK>(p, E, K, ids)) return;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    if (lane + 32 * k >= E) p[k] = -INFINITY;
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
// GEMV: logits may be words, and the ids alone may be asked for.  The top-k tiles have neither, and their copy without that code is what the batched
// step's routing is bound by, its instructions being fetched anew in every layer: 3 layers with it / without, 2 sequences at 60
// positions 521.7 / 516.0 us, 5 at 700 618.5 / 615.5, 24 at 1000 961 / 958.
template <bool LEAN, bool GEMV = true>
__device__ __noinline__ void warp_topk(const void* logits, uint32_t fl, int E, int K, bool renorm, bool bf16w,
                                       int32_t* ids, float* wts, int32_t* tei) {
  if (LEAN || E <= 128) warp_topk_n<4, GEMV>(logits, fl, E, K, renorm, bf16w, ids, wts, tei);
  else warp_topk_n<8, GEMV>(logits, fl, E, K, renorm, bf16w, ids, wts, tei);
}

__device__ __forceinline__ void tile_topk(const unsigned char* a, int blk, const Smem& sm) {
  const etxb_topk_args& d = *(const etxb_topk_args*)a;
  if (blk >= (int)d.nblocks) return;
  const int nb = (d.nbsv & 0xff) ? (d.nbsv & 0xff) : 1, sv = d.nbsv >> 8;
  const int w = tidx() >> 5;
  if (w >= nb) return;
  warp_topk<false, false>((const __nv_bfloat16*)d.logits + (size_t)w * d.E, 0u, d.E, d.K, (d.mode & 0xff) == 1, (d.mode & ETXB_MODE_BF16_WTS) != 0,
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
// Rows at once (R), rows per stage and warps per stage (W).  The products are bound by the unpacking of bf16 on the integer pipe and by their
// latencies: several rows at once share the activation vector with its unpacking and are reduced together, and 12 to 16 warps have to be at it.
//   up to 16 rows of up to 2048 values: a warp each (or several, S), in stages that all have a group at once
//   longer tasks, rows of up to 1792 values (7 vectors per lane): 4 at once; of 2048 (6 rows per stage): 3
//   longer rows (5 to 1 per stage): 3 or 4 at once (of 2 or 1 per stage one) by two warps, a half of the row each; by four where the task is a stream of
//   more stages than the ring has: a stage is given back sooner, and the last one is multiplied in a quarter of the time (a stand-alone 4096 -> 12288 GEMV
//   ends 14.5 us after its start, 15.3 with a row per warp; 12 dense layers 1142 us with two warps everywhere, 1126 now)
//   down grids of several slots: every slot has its own activations, so a stage holds rows of one slot
// Clocks per task, weights already in the ring, before / now: 14 rows of 4096 (a row per warp before) 2650 / 2100; 8 x 14 rows of 768 (16-row stages
// across the slots, activations unpacked per row) 6000 / 3700; 1 row of 2048 (three times by one warp) 1800 / 500; 11 of 1536 (by four warps) 1700 / 700.
// 35 of 2048: 2400, 60 bytes per clock; the same loop without its loads 2800 (with indexing), without its products 2000.
__device__ __forceinline__ int gemv_groups(int W) { return W <= 2 ? ETXB_NSTAGE : W == 3 ? 5 : W == 4 ? 4 : W <= 8 ? 2 : 1; }
// rows per stage (0: a row longer than a stage) and stages per range: what the producer has to know
__device__ __forceinline__ void gemv_stages(int body, int mode, GemvGeom& g) {
  const int total = g.t.nranges * g.t.n;
  g.rps = g.t.row_bytes > 0 && g.t.row_bytes <= ETXB_STAGE_BYTES ? udiv_small(ETXB_STAGE_BYTES, g.t.row_bytes) : 0;
  g.spr = 0;
  // (a row's sums are the same whichever way the results go: S does not depend on it)
  g.direct = body == 3 && total > ETXB_XF_FLOATS / 4 && !(mode & ETXB_MODE_WORDS_OUT);
  g.few = total <= ETXB_CONSUMER_WARPS && g.t.row_bytes <= 4096;
  if (total <= 0 || g.rps <= 0) return;
  if (g.few) {
    int r = min(g.rps, total);
    r = r >= 16 ? 16 : r >= 12 ? 12 : r >= 8 ? 8 : r >= 6 ? 6 : r >= 4 ? 4 : r;
#pragma unroll 1
    while (r > 1 && r * gemv_groups(r) < total) r = r > 12 ? 12 : r > 8 ? 8 : r > 6 ? 6 : r > 4 ? 4 : r - 1;
    g.rps = r;
  }
  if (body == 5 && g.t.nranges > 1) {
    g.spr = udiv_small(g.t.n + g.rps - 1, g.rps);
    g.rps = udiv_small(g.t.n + g.spr - 1, g.spr);
  }
}
__device__ __forceinline__ void gemv_geom(int body, int mode, GemvGeom& g) {
  const int total = g.t.nranges * g.t.n, nvl = ((g.t.row_bytes >> 4) + 31) >> 5;
  gemv_stages(body, mode, g);
  g.ns = 0; g.W = 1; g.NG = ETXB_NSTAGE; g.R = 1; g.S = 1; g.rw = 1; g.one = 0; g.rspr = 0.f;
  if (total > 0 && g.rps > 0) {
    if (g.spr) { g.rspr = __frcp_rn((float)g.spr); g.ns = g.t.nranges * g.spr; }
    else g.ns = total < (1 << 21) ? udiv_small(total + g.rps - 1, g.rps) : (total + g.rps - 1) / g.rps;
    const int m = min(g.rps, g.spr ? g.t.n : total);
    g.R = g.few ? 1 : nvl <= 7 ? 4 : nvl == 8 ? 3 : m == 3 || m == 5 ? 3 : m == 4 ? 4 : 1;
    g.one = g.R == 1 && nvl > 8;
    int rw = g.R == 4 ? (m + 3) >> 2 : g.R == 3 ? (m + 2) * 171 >> 9 : m;       // (m + 2 < 512: rows of more than 1792 values)
    rw = rw <= 4 ? rw : rw <= 6 ? 6 : rw <= 8 ? 8 : rw <= 12 ? 12 : 16;
    if (mode & ETXB_MODE_SUM_SLOTS) {                              // (its epilogue adds slots, not parts of rows)
    } else if (g.few) {
#pragma unroll 1
      while (g.S < 4 && total * g.S <= 8 && 2 * g.S <= nvl && g.ns <= gemv_groups(2 * g.S * rw)) g.S *= 2;
    } else if (nvl > 8 && total <= ETXB_XF_FLOATS / 4) g.S = rw == 1 && g.ns > ETXB_NSTAGE ? 4 : 2;    // (rw: 1 or 2 there)
    g.rw = rw; g.W = rw * g.S;
    g.NG = gemv_groups(g.W);
  }
  g.wmul = g.W <= 4 ? (g.W == 3 ? 86 : 256 >> (g.W >> 1)) : g.W == 6 ? 43 : g.W == 8 ? 32 : g.W == 12 ? 22 : 16;   // ceil(256 / W): exact for 16 warps and for ETXB_EMPTY_COUNT / W
  g.cnt = ETXB_EMPTY_COUNT * g.wmul >> 8;                           // 48 / W
  g.shared = g.NG == 4 || g.NG == 5;                                // (the groups that do not divide ETXB_NSTAGE)
}

// Expert ids (and routing weights, unless lwts is null) of the task's slots into `lids` / `lwts` (indexed by global slot).  One warp, all
// lanes call.  Top-k fold: recomputed from the logits; else read from the ids / wts buffers; no ids: expert 0.
// SH: the kernel variant supports always-on (shared) experts -- mode bits 24..27: ns experts that every token uses, stored
// after the E routed ones; they take the last ns slots with weight 1, the top-k picks the others.  (A template parameter
// and not a run-time branch: the lean kernels of the models without shared experts measured 1.4 % slower with it.)
template <bool LEAN, bool SH = !LEAN>
__device__ __forceinline__ void gemv_routing(const etxb_gemv_args& d, int32_t* lids, float* lwts) {
  const int fold = d.mode & 0xff, lane = tidx() & 31;
  const uint32_t fl = (d.mode & ETXB_MODE_WORDS_IN) ? s_vars.flag : 0u;
  if (fold >= 2) {
    if constexpr (SH) {
      const int ns = (d.mode >> 24) & 0xf;
      warp_topk<LEAN>(d.logits, fl, d.E, d.R - ns, fold == 3, (d.mode & ETXB_MODE_BF16_WTS) != 0, lids, lwts, nullptr);
      if (ns > 0) {
        if (lane < ns) { lids[d.R - ns + lane] = d.E + lane; if (lwts != nullptr) lwts[d.R - ns + lane] = 1.f; }
        __syncwarp();
      }
    } else {
      warp_topk<LEAN>(d.logits, fl, d.E, d.R, fold == 3, (d.mode & ETXB_MODE_BF16_WTS) != 0, lids, lwts, nullptr);
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
// ranges: a stage ends with its range.  ptr: the task's trace row when tracing (slot 7 <- time the first stage was issued, slot 6 <- the last), else null.
template <bool SH = true>
__device__ __forceinline__ bool produce_task(int body, const etxb_gemv_args& d, const GemvTask& t, int rps, bool ranges, const int32_t* lids, uint32_t& n,
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
    for (int q0 = 0, i = 0; q0 < total && ok; ++i) {
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
      if (body == 3 && i < ETXB_NSTAGE)
#pragma unroll 1
        for (int spin = 0; spin < 64 && *(volatile const int*)&sm.vars->hold != 0; ++spin) __nanosleep(40);
      const int nr = min(rps, ranges ? t.n - r : total - q0);
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
      if (ptr != nullptr) { if (i == 0) ptr[7] = globaltimer(); ptr[6] = globaltimer(); }
      ++n;
      q0 += nr;
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

// Where a row's result goes: fp32 to `g` (S partial sums a row), from which the tile's epilogue takes all of them behind a barrier (in order, so
// that its stores are coalesced, and one copy of it serves every form of the multiplication); g null (GemvGeom::direct, a plain task of more rows than
// `g` holds): bf16(v + bias) to `out` at once.
struct GemvEpi {
  float* g;
  __nv_bfloat16* out;        // row 0 of the task
  const void* bias;          // bf16, row 0 of the task, or null
};
__device__ __forceinline__ void gemv_epi(const GemvEpi& e, int q, int S, int h, float v) {
  if (e.g) e.g[q * S + h] = v;
  else e.out[q] = __float2bfloat16_rn(e.bias ? __fadd_rn(v, __bfloat162float(((const __nv_bfloat16*)e.bias)[q])) : v);
}

// Rows j, j + rw, .. (R of them, those past the stage's nr repeat the last one and are dropped) of one stage by one warp, vectors h * 32 + lane,
// (h + S) * 32 + lane, .. of each, U at a time.  stage, x: shared-memory addresses of the stage and of the activation vector; q0: the stage's
// first row.  (One copy for 1 to 4 rows, told apart inside the loop: 35 rows of 2048 in 3250 clocks against 2500.)
template <int R, int U>
__device__ __forceinline__ void gemv_rows(uint32_t stage, int row_bytes, int j, int rw, int nr, int h, int S, int q0, uint32_t x, const GemvEpi& e) {
  const int lane = tidx() & 31;
  uint32_t w[R];
  float a[R];
#pragma unroll
  for (int u = 0; u < R; ++u) { w[u] = stage + (uint32_t)(min(j + u * rw, nr - 1) * row_bytes); a[u] = 0.f; }
#pragma unroll U
  for (int o = (h * 32 + lane) * 16; o < row_bytes; o += S * 512) {
    const uint4 xv = lds128(x + o);
#pragma unroll
    for (int u = 0; u < R; ++u) a[u] = dot8(lds128(w[u] + o), xv, a[u]);
  }
  if constexpr (R == 1) {
    const float s = warp_sum(a[0]);
    if (lane == 0) gemv_epi(e, q0 + j, S, h, s);
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
    const int u = (h16 ? 2 : 0) + (h8 ? 1 : 0), jj = j + u * rw;
    if ((lane & 7) == 0 && u < R && jj < nr) gemv_epi(e, q0 + jj, S, h, k);
  }
}

// Consume the stages of one task: row q (0 .. total-1, range q / rows) . its activation vector -> gemv_epi.
// Where a stage ends with its range, range i uses the vector i * K further on.  A stage is waited for, read and given
// back by its group's W warps only (each arrives ETXB_EMPTY_COUNT / W times); the stage counter runs on by the task's
// stages in every warp.
// (Measured and not kept: the packed fma.rn.f32x2 form of the inner loop, +1.3 % step time; the mixed fma.rn.f32.bf16,
// which needs no unpacking but issues at about a quarter of the rate: 39 -> 41 bytes per clock with one row; a lane's
// share of the activations in registers, which spills at the 96 registers this kernel gets; a ring of 7 stages instead of 6,
// +0.6 %; mma.sync m16n8k16 with conflict-free unpadded rows (row r reads the 16-byte chunks in the order c ^ r and column r
// of B holds the activations in that order): 3800 clocks for 35 rows of 2048, with an error 1.2 times as large; this function as a
// call, one copy for all tiles: its arguments and saved registers on the stack cost 2 us per phase.)
__device__ __forceinline__ void consume_task(uint32_t& n, const Smem& sm, const __nv_bfloat16* xb, int where, const GemvEpi& e) {
  static_assert(ETXB_NSTAGE == 6, "which numbers of groups divide the ring (GemvGeom::shared)");
  const int lane = tidx() & 31, cw = tidx() >> 5;
  const GemvGeom geo = *sm.geo;
  const int g = (cw * geo.wmul) >> 8, wi = cw - g * geo.W, h = wi & (geo.S - 1), j0 = geo.S == 1 ? wi : wi >> (geo.S == 2 ? 1 : 2);
  const int rows = geo.t.n, total = geo.t.nranges * rows, row_bytes = geo.t.row_bytes;
  const uint32_t ring = smem_u32(sm.ring), xa = smem_u32(xb);
  uint32_t k = n + (uint32_t)g;
  n += (uint32_t)geo.ns;
  if (g >= geo.NG) return;
  volatile const uint32_t* use = (volatile const uint32_t*)(sm.full + 2 * ETXB_NSTAGE);
#pragma unroll 1
  for (int i = g; i < geo.ns; i += geo.NG, k += (uint32_t)geo.NG) {
    const uint32_t rd = k / ETXB_NSTAGE, st = k - rd * ETXB_NSTAGE;
    // A parity wait tells use k of a stage from use k - 1 only, and with a number of groups that does not divide the ring
    // the use before this one may be another group's that is still being filled: the wait would be answered by use k - 2.
    // So the producer's note of the use it fills is looked at first (when it names k, k - 1 is over).
    if (geo.shared && !wait_use(use + st, k, sm, where)) return;
    if (!mbar_wait(sm.full + st, rd & 1, sm, where)) return;       // step abandoned: touch nothing
    if (i == 0) mark(sm, 1);
    const int rg = __float2int_rz(((float)i + 0.5f) * geo.rspr), r0 = (i - rg * geo.spr) * geo.rps;   // (spr = 0: range 0, row i * rps of all)
    const int nr = min(geo.rps, (geo.spr != 0 ? rows : total) - r0), q0 = rg * rows + r0;
    const uint32_t stage = ring + st * ETXB_STAGE_BYTES, x = xa + (uint32_t)(rg * row_bytes);
#pragma unroll 1
    for (int j = j0; j < nr; j += geo.R * geo.rw) {
      // (one row at a time: long rows four vectors deep; a few short ones in a loop that is short to fetch)
      if (geo.R == 4) gemv_rows<4, 1>(stage, row_bytes, j, geo.rw, nr, h, geo.S, q0, x, e);
      else if (geo.R == 3) gemv_rows<3, 1>(stage, row_bytes, j, geo.rw, nr, h, geo.S, q0, x, e);
      else if (geo.one) gemv_rows<1, 4>(stage, row_bytes, j, geo.rw, nr, h, geo.S, q0, x, e);
      else gemv_rows<1, 1>(stage, row_bytes, j, geo.rw, nr, h, geo.S, q0, x, e);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_n(sm.empty + st, (uint32_t)geo.cnt);
  }
}

// ---------------------------------------------------------------------------------------------- activation staging
// K bf16 values (written by other CTAs) -> shared memory, K % 8 == 0.
__device__ __forceinline__ void stage_xb(const void* x, int K, __nv_bfloat16* xb) {
  const int nv = K >> 3;
  for (int i = tidx(); i < nv; i += ETXB_CONSUMERS) ((uint4*)xb)[i] = ld_act16((const __nv_bfloat16*)x + 8 * i);
  csync();
}

// K words -> bf16 values in shared memory, K % 4 == 0.
__device__ __forceinline__ void stage_words(const uint32_t* w, int K, uint32_t fl, __nv_bfloat16* xb) {
  const int nv = K >> 2;
#pragma unroll 1
  for (int i = tidx(); i < nv; i += 4 * ETXB_CONSUMERS) {
    uint4 v[4];
    uint32_t spins = 0;
    for (;;) {
      uint32_t miss = 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = i + u * ETXB_CONSUMERS < nv ? ld_words4(w + 4 * (i + u * ETXB_CONSUMERS)) : make_uint4(fl, fl, fl, fl);
#pragma unroll
      for (int u = 0; u < 4; ++u) miss |= words_miss(v[u], fl);
      if (miss == 0u || !words_again(spins, fl)) break;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * ETXB_CONSUMERS < nv) ((uint2*)xb)[i + u * ETXB_CONSUMERS] = words_pack(v[u]);
  }
  csync();
}

// Norm fold (below) for the hand-off as words: z = bf16(resid_in + row) or resid_in, x = bf16(ln * bf16(z * r)) -> xb; `store`: z and x
// also to memory, as bf16 and as words.  in: rows / resid_in name words.  K % 4 == 0, K <= 8192.
// A chain of latencies in front of every phase that folds a norm, so a warp's vectors are the blocks of 128 values that numpy's order
// sums up (sumsq_numpy_order): squares are added without a barrier, and the blocks' sums meet behind the only one.  The same bits as that function's where
// K is a power of two; it takes strided chains for other widths, which are further from 64-bit sums (rms at 1536 values 6.5e-8, so 4.2e-8).
__device__ __forceinline__ void stage_norm_words(const etxb_gemv_args& d, const etxb_gemv_words& wd, uint32_t fl, bool in, bool store,
                                                 float* xf, __nv_bfloat16* xb, float* scr) {
  const int K = d.K, nv = K >> 2, nblk = (K + 127) >> 7, lane = tidx() & 31, warp = tidx() >> 5;
  const float inv = __int_as_float((127 - (31 - __clz(K))) << 23);  // 1 / K where K is a power of two: the same as dividing
  const int LD = nblk <= ETXB_XF_FLOATS / 136 ? 136 : 128;         // floats from block to block (136: the accumulators of four blocks in 32 banks)
#pragma unroll 1
  for (int i = tidx(); i < 32 * nblk; i += ETXB_CONSUMERS) {       // vector i: block i / 32
    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < nv) {
      const uint2 ln = __ldg((const uint2*)d.ln + i);
      uint4 r, a;                                                  // values in the upper halves
      if (in) {
        uint32_t spins = 0;
        do {
          r = ld_words4((const uint32_t*)d.resid_in + 4 * i);
          a = ld_words4((const uint32_t*)d.rows + 4 * i);
        } while ((words_miss(r, fl) | words_miss(a, fl)) != 0u && words_again(spins, fl));
        r = make_uint4(r.x << 16, r.y << 16, r.z << 16, r.w << 16);
        a = make_uint4(a.x << 16, a.y << 16, a.z << 16, a.w << 16);
      } else {
        const uint2 q = __ldcg((const uint2*)d.resid_in + i);
        r = make_uint4(q.x << 16, q.x & 0xffff0000u, q.y << 16, q.y & 0xffff0000u);
        if (d.rows != nullptr) {
          const uint2 p = __ldcg((const uint2*)d.rows + i);
          a = make_uint4(p.x << 16, p.x & 0xffff0000u, p.y << 16, p.y & 0xffff0000u);
        }
      }
      z = make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
      if (d.rows != nullptr) {
        z.x = bfr(__fadd_rn(z.x, __uint_as_float(a.x))); z.y = bfr(__fadd_rn(z.y, __uint_as_float(a.y)));
        z.z = bfr(__fadd_rn(z.z, __uint_as_float(a.z))); z.w = bfr(__fadd_rn(z.w, __uint_as_float(a.w)));
      }
      ((uint2*)xb)[i] = ln;                                        // (where this thread's x goes)
      if (store) {
        const uint32_t u0 = __float_as_uint(z.x), u1 = __float_as_uint(z.y), u2 = __float_as_uint(z.z), u3 = __float_as_uint(z.w);
        if (wd.z != nullptr) st_words4(wd.z + 4 * i, make_uint4((u0 >> 16) | fl, (u1 >> 16) | fl, (u2 >> 16) | fl, (u3 >> 16) | fl));
        if (d.resid_out != nullptr) ((uint2*)d.resid_out)[i] = make_uint2((u0 >> 16) | (u1 & 0xffff0000u), (u2 >> 16) | (u3 & 0xffff0000u));
      }
    }
    *(float4*)(xf + (i >> 5) * LD + 4 * lane) = z;
  }
  __syncwarp();
  {
    const int blk = warp + 16 * (lane >> 3);                       // this lane: accumulator lane % 8 of one of the warp's (up to four) blocks
    float s = 0.f;
    if (blk < nblk) {
      const float* x = xf + blk * LD + (lane & 7);
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = x[8 * i];
      s = __fmul_rn(v[0], v[0]);
#pragma unroll
      for (int i = 1; i < 16; ++i) s = __fadd_rn(s, __fmul_rn(v[i], v[i]));
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((lane & 7) == 0) scr[blk] = s;                             // (64 of them: blocks past the last one are 0)
  }
  csync();
  float ss = scr[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
  if (nblk > 32) {
    float s1 = scr[32 + lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) s1 = __fadd_rn(s1, __shfl_xor_sync(0xffffffffu, s1, o));
    ss = __fadd_rn(ss, s1);
  }
  const float mean = (K & (K - 1)) == 0 ? __fmul_rn(ss, inv) : __fdiv_rn(ss, (float)K);
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, d.eps)));
#pragma unroll 1
  for (int i = tidx(); i < nv; i += ETXB_CONSUMERS) {
    const float4 z = *(const float4*)(xf + (i >> 5) * LD + 4 * lane);
    const uint2 w = ((const uint2*)xb)[i];
    const uint2 o = make_uint2(pack_bf(__fmul_rn(bf_lo(w.x), bfr(__fmul_rn(z.x, r))), __fmul_rn(bf_hi(w.x), bfr(__fmul_rn(z.y, r)))),
                               pack_bf(__fmul_rn(bf_lo(w.y), bfr(__fmul_rn(z.z, r))), __fmul_rn(bf_hi(w.y), bfr(__fmul_rn(z.w, r)))));
    ((uint2*)xb)[i] = o;
    if (store) {
      if (wd.x != nullptr) st_words4(wd.x + 4 * i, make_uint4((o.x & 0xffffu) | fl, (o.x >> 16) | fl, (o.y & 0xffffu) | fl, (o.y >> 16) | fl));
      if (d.x != nullptr) ((uint2*)d.x)[i] = o;
    }
  }
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
// A down task whose routing comes as words, which the gate+up grid publishes when it begins: nothing the task waits for is needed to read
// it, so that is done while its event is being waited for (at the head of the body it took 4000 clocks of the phase).
__device__ __forceinline__ bool gemv_routed_early(int body, const etxb_gemv_args& d) {
  return body == 5 && (d.mode & 0xff) >= 2 && (d.mode & (ETXB_MODE_WORDS_IN | ETXB_MODE_ROUTE_READY)) == (ETXB_MODE_WORDS_IN | ETXB_MODE_ROUTE_READY);
}
// For the summed form of down: the slots in ascending expert id (where their results begin) at scr + 64, with their weights at 80; ids and
// weights of all slots are at 96 and 112.  One warp.
__device__ __forceinline__ void gemv_slot_order(const GemvTask& t, float* scr) {
  const int32_t* lids = (const int32_t*)(scr + 96) + t.group * t.spt;
  const int lane = tidx() & 31;
  if (lane < t.spt) {
    const int mine = lids[lane];
    int rank = 0;
#pragma unroll 1
    for (int j = 0; j < t.spt; ++j) { const int o = lids[j]; rank += (o < mine) || (o == mine && j < lane); }
    ((int*)(scr + 64))[rank] = lane * t.n;
    (scr + 80)[rank] = (scr + 112)[t.group * t.spt + lane];
  }
}
__device__ __forceinline__ void gemv_route_words(const etxb_gemv_args& d, const etxb_gemv_words& wd, const GemvTask& t, float* scr) {
  const int lane = tidx() & 31;
  if (lane < 16) {
    uint32_t u = 0u, spins = 0;
    uint2 v = make_uint2(__float_as_uint(1.f), 0u);
    if (lane < d.R) {
      const uint32_t fl = s_vars.flag;
      const uint2* pw = (const uint2*)(wd.route + 16) + lane;
      do { u = ld_word(wd.route + lane); v = ld_volatile8(pw); } while ((((u ^ fl) >> 16) != 0u || v.y != fl) && words_again(spins, fl));
      u &= 0xffffu;
    }
    ((int32_t*)(scr + 96))[lane] = u == 0xffffu ? 0x7fffffff : (int32_t)u;
    (scr + 112)[lane] = __uint_as_float(v.x);
  }
  __syncwarp();
  if (d.mode & ETXB_MODE_SUM_SLOTS) gemv_slot_order(t, scr);
}
// Routing of a task's slots otherwise.  One warp.  A gate+up group's first chunk also publishes its slots' routing.
template <bool LEAN, bool SH, bool WD>
__device__ __forceinline__ void gemv_route_task(int body, const etxb_gemv_args& d, const etxb_gemv_words& wd, int blk, const GemvTask& t, float* scr) {
  int32_t* lids = (int32_t*)(scr + 96); float* lwts = scr + 112;
  const int fold = d.mode & 0xff, lane = tidx() & 31;
  if (body == 4 && !(fold >= 2 && blk - t.group * d.tpe == 0)) return;    // (gate+up needs the routing only to publish it)
  if (body == 5 && fold >= 2 && (d.mode & ETXB_MODE_ROUTE_READY) && d.ids != nullptr && d.wts != nullptr) {
    if (lane < 16) {
      lids[lane] = lane < d.R ? __ldcg(d.ids + lane) : 0;
      lwts[lane] = lane < d.R ? __ldcg(d.wts + lane) : 1.f;
    }
    __syncwarp();
  } else gemv_routing<LEAN, SH>(d, lids, lwts);
  if (body == 4 && lane < t.spt) {
    const int sl = t.group * t.spt + lane;
    if (WD && (d.mode & ETXB_MODE_WORDS_OUT) && wd.route != nullptr) {
      const uint32_t fl = s_vars.flag;
      st_word(wd.route + sl, ((uint32_t)lids[sl] < 0xffffu ? (uint32_t)lids[sl] : 0xffffu) | fl);
      st_relaxed8((uint2*)(wd.route + 16) + sl, __float_as_uint(lwts[sl]), fl);
    }
    if (d.ids) ((int32_t*)d.ids)[sl] = lids[sl];
    if (d.wts) ((float*)d.wts)[sl] = lwts[sl];
  }
  // (known as soon as the routing is: worked out here, under the weight stream, and not after it)
  if (body == 5 && (d.mode & ETXB_MODE_SUM_SLOTS)) gemv_slot_order(t, scr);
}
template <bool LEAN, bool XCH = false, bool SH = !LEAN>
__device__ __forceinline__ void tile_gemv_family(int body, const unsigned char* a, int blk, const Smem& sm, uint32_t& n, int where) {
  const etxb_gemv_args& d = *(const etxb_gemv_args*)a;
  const GemvTask& t = sm.geo->t;
  if (t.n <= 0) return;
  constexpr bool WD = !XCH;                                        // (a sharded session has no words of this kind)
  const int mode = d.mode, fold = mode & 0xff, K = d.K;
  const bool win = WD && (mode & ETXB_MODE_WORDS_IN), wout = WD && (mode & ETXB_MODE_WORDS_OUT);
  const bool sum = body == 5 && (mode & ETXB_MODE_SUM_SLOTS) != 0;
  const etxb_gemv_words& wd = *(const etxb_gemv_words*)(a + sizeof(etxb_gemv_args));
  __nv_bfloat16* const xb = smem_xb(sm);
  if (body == 3 && !win && fold == 0) stage_xb(d.x, K, xb);        // (a stand-alone launch waits for its activations and for this code: the short way)
  else {
  if (body == 5 && !(WD && gemv_routed_early(body, d)) && tidx() < 32) gemv_route_task<LEAN, SH, WD>(body, d, wd, blk, t, sm.scr);
  // the activations
  if (fold == ETXB_MODE_NORM && (win || wout)) stage_norm_words(d, wd, s_vars.flag, win, blk == 0, sm.xs, xb, sm.scr);
  else if (win) {                                                  // (down: the task's slots' vectors, one behind the other)
    const bool dn = body == 5;
    stage_words((const uint32_t*)d.x + (dn ? t.group * t.spt * K : 0), dn ? t.spt * K : K, s_vars.flag, xb);
  } else if (body == 5) {
    for (int i = tidx(); i < t.spt * (K >> 3); i += ETXB_CONSUMERS) ((uint4*)xb)[i] = ld_act16((const __nv_bfloat16*)d.x + (size_t)t.group * t.spt * K + 8 * i);
    csync();
  } else if (fold == ETXB_MODE_NORM)                               // (a dense MLP's gate+up: the post-attention norm folded in)
    stage_norm_col<LEAN, XCH>(d.rows, d.resid_in, d.resid_out, (void*)d.x, d.ln, body == 3 ? d.ids : nullptr, d.R, K, d.eps, sm.xs, xb, sm.scr, blk == 0,
                              (XCH && (mode & ETXB_MODE_FLAGGED)) ? s_vars.flag : 0u, &sm);
  else stage_xb(d.x, K, xb);
  }
  const int rows = t.n, spt = t.spt, S = sm.geo->S;
  float* const g = sm.xs;                                          // results (S partial sums each): up: per slot, rows gate results, then rows up results;  down: rows per slot
  const float* const lwts = sm.scr + 112;
  GemvEpi e;
  e.g = sm.geo->direct ? nullptr : g;
  e.out = (__nv_bfloat16*)d.out + t.r0;
  e.bias = body == 3 && (mode & ETXB_MODE_BIAS) ? (const __nv_bfloat16*)d.wts + t.r0 : nullptr;
  mark(sm, 0);
  // (the top-k that a gate+up group's first chunk publishes: nothing in this task waits for it, and the last warp mostly has no rows)
  if (body == 4 && tidx() >= ETXB_CONSUMERS - 32) gemv_route_task<LEAN, SH, WD>(body, d, wd, blk, t, sm.scr);
  consume_task(n, sm, xb, where, e);
  if (e.g == nullptr) return;
  csync();
  if (sum && tidx() == 0) *(volatile int*)&sm.vars->hold = 1;
  mark(sm, 2);
  const uint32_t fl = s_vars.flag;
  uint32_t* const words = wout ? wd.out : nullptr;
  __nv_bfloat16* const out = (__nv_bfloat16*)d.out;
  auto val = [&](int q) {                                          // (partial sums pairwise)
    float v = g[q * S];
    if (S > 1) {
      v = __fadd_rn(v, g[q * S + 1]);
      if (S > 2) v = __fadd_rn(v, __fadd_rn(g[q * S + 2], g[q * S + 3]));
    }
    return v;
  };
  auto put = [&](uint32_t at, float y) {
    const uint32_t u = bf_bits(y);
    if (WD && words != nullptr) st_word(words + at, u | fl);
    if (out != nullptr) ((unsigned short*)out)[at] = (unsigned short)u;
  };
  if (body == 3) {
#pragma unroll 1
    for (int r = tidx(); r < rows; r += ETXB_CONSUMERS) {
      float y = val(r);
      if (e.bias) y = __fadd_rn(y, __bfloat162float(((const __nv_bfloat16*)e.bias)[r]));
      put((uint32_t)(t.r0 + r), y);
    }
  } else if (sum) {
    const int* order = (const int*)(sm.scr + 64);
    const bool weighted = fold >= 2 || d.wts != nullptr;
#pragma unroll 1
    for (int r = tidx(); r < rows; r += ETXB_CONSUMERS) {
      float acc = 0.f;
#pragma unroll 1
      for (int k0 = 0; k0 < spt; k0 += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int i = min(k0 + k, spt - 1);
          v[k] = bfr(g[order[i] + r]);                             // (S = 1 there)
          if (weighted) v[k] = bfr(__fmul_rn(v[k], (sm.scr + 80)[i]));
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) if (k0 + k < spt) acc = bfr(__fadd_rn(acc, v[k]));
      }
      put((uint32_t)(t.r0 + r), acc);
    }
  } else {
    uint32_t at = (uint32_t)(t.group * spt * d.M + t.r0);
    const float* const wt = body == 5 && (fold >= 2 || d.wts != nullptr) ? lwts + t.group * spt : nullptr;
#pragma unroll 1
    for (int s = 0, r = tidx(), q = 0; s < spt; ++s, r -= rows, at += (uint32_t)d.M, q += body == 4 ? 2 * rows : rows)
#pragma unroll 1
      for (; r < rows; r += ETXB_CONSUMERS) {
        float y = val(q + r);
        if (body == 4) y = __fmul_rn(bfr(silu_f(bfr(y))), bfr(val(q + rows + r)));
        else if (wt) y = __fmul_rn(bfr(y), wt[s]);
        put(at + (uint32_t)r, y);
      }
  }
}

}  // namespace etxb
