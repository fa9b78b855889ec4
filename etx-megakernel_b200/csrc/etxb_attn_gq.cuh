// The attention phase of a decode step, the form for head_dim 128 and 16-position cache blocks: one task per
// (128-position partition, group of gq <= 8 q heads that share a kv head), or one per group that walks the whole context.  Same work
// as the general fused tile (etxb_attn_fused.cuh: q/k RMSNorm + neox rotary, the new position's k / v rows into the paged cache,
// split-KV attention, merge), built around what a decode step makes of it: a few microseconds of latency and a stream of K / V.
//   * K and V come through the weight ring: a cache block of one kv head is 4 KB of K and 4 KB of V in one piece each (a UNIT
//     of 16 positions), three units to a stage.  The producer warp copies them ahead of the task as it does weights -- the rows of earlier
//     positions depend on nothing in this step -- so they lie in shared memory when the q rows arrive.
//   * a warp takes a unit at a time and runs it alone: scores on the tensor cores (mma.sync, 16 positions x 8 heads, K rows by
//     ldmatrix), its own running maximum and sum, the probabilities transposed by movmatrix into the second product's operand, 128
//     output sums per head in its registers.  No barrier between units; the warps' results meet once, at the end.
//   * the probabilities go into the product as a bf16 value, the bf16 of what that rounding lost and that of what the second one lost: the
//     24 bits of their fp32 value, as they were multiplied before.  Plans with a task per whole context: the first two (2^-17 of the value), as before
//     too, but all three for the unit of the new position, whose probability was multiplied in fp32, and where the block asks for it (ETXB_GQ_PRECISE).
//     Sums meet in fp32, so that the partials are no further from 64-bit ones than plain fp32 chains of 32 terms leave them: 1.3e-7 at 1038
//     and 8151 positions against 1.6e-7 (summed up inside the products 1.8e-7).
// Bound by the stream of K / V at long contexts, by the chain q rows -> norm -> scores -> publish -> merge at short ones.
// From the last q row to the last output: one sequence at 8150 positions (64 partitions, 256 tasks) 28.1 us -> 16.5, at 1037 9.3 -> 7.8, a
// small dense model at 601 (one q head a task) 8.4 -> 7.6; 8 sequences at 1033 33.4 -> 22.9, 13 at 333 31.5 -> 24.0; 32 sequences, whole
// contexts of 1045: 53.5 -> 25.0.  The forms before multiplied out of registers on the fp32 pipes, or walked a context with a barrier between
// any two of its steps.
// The new position never comes from the cache: its k / v rows stand in for the stale slot of the staged unit.
//
// It stands where the reference runs dsl_attnprep (etx/ops/attnprep.py:86-211), vLLM's paged attention and its reduce
// kernel (etx/importer/spec.py:243-244; grids examples/vllm_llm/model.py:78-84, 358-362); numerics follow
// examples/llm/ref_numpy.py:113-129 (fp32 scores and sums over bf16 q, k, v; bf16 output).
#pragma once
#include "etxb_attn_fused.cuh"

namespace etxb {

#define ETXB_GQ_PART 128   // positions per task
#define ETXB_GQ_WHOLE (1 << 24)   // part_len bit: one task per (sequence, q group) takes all partitions
#define ETXB_GQ_WORDS (1 << 25)   // part_len bit: qkv names words, the outputs are also written as words (at exp_sums)
#define ETXB_GQ_LIM_SHIFT 26      // part_len bits 26..31: contexts of up to so many partitions are taken whole, by the tasks of the first one
#define ETXB_GQ_PRECISE (1 << 26) // .. in the whole-context form: cached units with all 24 bits of their probabilities, too
#define ETXB_GQ_WHOLE_MAX 157     // .. of partitions x q heads at most (the builder's rule: ops/attn.py)
#define ETXB_GQ_PW 136     // 8-byte (value, flag) pairs a task publishes per q head and partition: 128 outputs, max, sum, padding
#define ETXB_GQ_SHARE 64   // partials (gq x partitions) from which the merge is shared out.  Shared / by one task, us of a phase: 72 partials (8 sequences)
                           // 22.3 / 23.9, 88 (3 sequences) 13.3 / 15.9; 8 x 64 partials are 512 KB for one task.  Few partials: 144 tasks that all wait and poll
                           // made a phase of 2 x 9 partials 9.5, one merging task per group 8.0.  (Between them sharing gains too: 5 x 8 partials 23.6 / 24.5.)
#define ETXB_GQ_UNIT 8192  // a unit in a ring stage: 16 positions' K (4 KB), then their V
#define ETXB_GQ_UPS (ETXB_STAGE_BYTES / ETXB_GQ_UNIT)   // units per stage

// Partial results travel as FLAGGED PAIRS: every fp32 value is stored together with a 32-bit flag derived from the step
// (one aligned 8-byte store: value and flag become visible together), into `tmp_out` viewed as
// [NH][max_parts][ETXB_GQ_PW] pairs.  The merge is run by a task that is known beforehand -- the one of the context's LAST
// partition (the partition of the new position: it has the fewest cached positions, so it is the first to finish and
// polls while the others work) -- which re-reads a pair until its flag is this step's.  No counter, no election, no
// fence: the producers only store, the merger's loads are its wait.  Nothing has to be reset between steps or after an
// abandoned step; a buffer that was zeroed once never shows a current flag by accident (flags are never 0, differ
// from grid to grid within a step and grow with every launch of the process, so sessions may share the buffers, one after the other).  Bounded like every wait: on a give-up the step is abandoned with the timeout status.
// The flag names the launch AND the grid: the layers of a step share the partial buffers, and a merger must not take the
// previous layer's partials of the same step for its own.  The grid's tag travels in the upper half of the block's
// part_len word (the builder puts the layer index there).
__device__ __forceinline__ uint32_t pair_flag(uint32_t serial, int part_len) { return ((serial << 8) | (((uint32_t)part_len >> 16) & 0xffu)) | 0x80000000u; }
__device__ __forceinline__ void st_pair(uint2* p, float v, uint32_t fl) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(fl) : "memory");
}
__device__ __forceinline__ uint2 ld_pair(const uint2* p) {
  uint2 v;
  asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
// value of the pair at `p` once its flag is `fl`; gives up (step abandoned, 0 returned) at the deadline or on an abort
__device__ __forceinline__ float poll_pair(const uint2* p, uint32_t fl, const Smem& sm) {
  uint32_t spins = 0;
  for (;;) {
    const uint2 v = ld_pair(p);
    if (v.y == fl) return __uint_as_float(v.x);
    if ((++spins & 63u) == 0) {
      if (ld_relaxed(sm.ctrl()) != 0) { *(volatile int*)sm.stop = 1; return 0.f; }
      if ((spins & 1023u) == 0 && globaltimer() > *sm.deadline) {
        if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) { sm.ctrl()[1] = sm.cur(); sm.ctrl()[2] = -3; sm.ctrl()[3] = (int32_t)v.y; sm.ctrl()[4] = (int32_t)fl; }
        *(volatile int*)sm.stop = 1;
        return 0.f;
      }
      __nanosleep(32);
    }
  }
}

// Between two rounds of a poll of n pairs (from `p` on, `stride` pairs apart): false when the step is being abandoned (deadline or
// abort, see poll_pair).  The flag that is missing is looked up again for the report, so that the poll need not keep it.
__device__ __forceinline__ bool poll_again(uint32_t& spins, const uint2* p, int n, size_t stride, uint32_t fl, const Smem& sm) {
  if ((++spins & 15u) == 0) {
    if (ld_relaxed(sm.ctrl()) != 0) { *(volatile int*)sm.stop = 1; return false; }
    if ((spins & 255u) == 0 && globaltimer() > *sm.deadline) {
      if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) {
        uint32_t seen = fl;
#pragma unroll 1
        for (int u = 0; u < n && seen == fl; ++u) seen = ld_pair(p + (size_t)u * stride).y;
        sm.ctrl()[1] = sm.cur(); sm.ctrl()[2] = -3; sm.ctrl()[3] = (int32_t)seen; sm.ctrl()[4] = (int32_t)fl;
      }
      *(volatile int*)sm.stop = 1;
      return false;
    }
    __nanosleep(32);
  }
  return true;
}

// What a task covers: worked out alike by the consumer warps and by the producer warp.
struct GqTask {
  int part, hq0, h;          // partition (0 in the whole-context form), first q head of the group, its kv head
  int t0, u0, nu;            // first position; first unit (cache block) and number of units
  int seq;
  long long pos;
  bool whole, owner;         // whole: one task per group takes all of the context; owner: the task's positions hold the one being written
};
__device__ __forceinline__ GqTask gq_task(const etxb_attnf_args& d, int blk, const etxb_stepv& S) {
  GqTask t;
  // the step's own buffers hold what the prologue wrote from the step parameters: take the values from there
  t.pos = (const void*)d.positions == (const void*)S.positions ? (long long)S.pos : __ldcg((const long long*)d.positions);
  t.seq = (const void*)d.seq_lens == (const void*)S.seq_lens ? S.pos + 1 : __ldcg(d.seq_lens);
  const bool form = (d.part_len & ETXB_GQ_WHOLE) != 0;
  const int lg = 31 - __clz(d.gq), NQG = d.NH >> lg;               // (gq: 1, 2, 4 or 8)
  t.part = form ? 0 : udiv_small(blk, NQG);
  t.hq0 = (blk - t.part * NQG) << lg;
  t.h = udiv_small(t.hq0 * d.NKV, d.NH);
  t.t0 = t.part * ETXB_GQ_PART;
  const int np = min((t.seq + ETXB_GQ_PART - 1) / ETXB_GQ_PART, d.max_parts);
  t.whole = form || np <= (int)((uint32_t)d.part_len >> ETXB_GQ_LIM_SHIFT);    // (the tasks of the other partitions have nothing to do then)
  const int tend = t.whole && t.part == 0 ? np * ETXB_GQ_PART : t.t0 + ETXB_GQ_PART;
  t.owner = t.pos >= t.t0 && t.pos < tend && !(t.whole && t.part > 0);
  const int lim = t.owner ? max(t.seq, (int)t.pos + 1) : t.seq;
  t.u0 = t.t0 >> 4;
  t.nu = t.t0 < t.seq && tend > t.t0 && !(t.whole && t.part > 0) ? (min(tend, lim) - t.t0 + 15) >> 4 : 0;
  return t;
}

// Producer warp: the task's units into the ring, three to a stage.  A unit past the context (possible only where positions and
// seq_lens disagree) has no block: its place in the stage stays as it is.
__device__ __forceinline__ bool produce_attn(const etxb_attnf_args& d, int blk, const etxb_stepv& S, uint32_t& n, const Smem& sm, int where) {
  if (blk >= (int)d.nblocks) return true;
  const GqTask t = gq_task(d, blk, S);
  const int lane = tidx() & 31, ns = (t.nu + ETXB_GQ_UPS - 1) / ETXB_GQ_UPS;
  const size_t piece = (size_t)128 * 16 * 2;                        // bytes of one kv head's K (or V) in a cache block
  bool ok = true;
  int tab = 0;
  for (int s = 0; s < ns && ok; ++s) {
    const uint32_t st = n % ETXB_NSTAGE, par = (n / ETXB_NSTAGE) & 1;
    const int i0 = s * ETXB_GQ_UPS;
    if (s % 10 == 0) {                                             // block-table entries of the next ten stages' units, one per lane
      const int u = t.u0 + i0 + lane;
      tab = i0 + lane < t.nu && (u << 4) < t.seq ? __ldg(d.block_tables + u) : 0;
    }
    const int i = i0 + (lane >> 1), u = t.u0 + i;
    const bool live = lane < 2 * ETXB_GQ_UPS && i < t.nu && (u << 4) < t.seq;
    const long long pb = __shfl_sync(0xffffffffu, tab, (i0 % (10 * ETXB_GQ_UPS) + (lane >> 1)) & 31);
    const int pieces = __popc(__ballot_sync(0xffffffffu, live));
    int good = 1;
    if (lane == 0) {
      good = mbar_wait(sm.empty + st, par ^ 1, sm, where) ? 1 : 0;
      if (good) {
        *((volatile uint32_t*)(sm.full + 2 * ETXB_NSTAGE) + st) = n;  // (see wait_use)
        mbar_expect_tx(sm.full + st, (uint32_t)(pieces * piece));
      }
    }
    ok = __shfl_sync(0xffffffffu, good, 0) != 0;
    if (ok && live)
      bulk_g2s(sm.ring + (size_t)st * ETXB_STAGE_BYTES + (lane >> 1) * ETXB_GQ_UNIT + (lane & 1) * piece,
               (const unsigned char*)((lane & 1) ? d.vc : d.kc) + ((size_t)pb * d.NKV + t.h) * piece, (uint32_t)piece, sm.full + st);
    if (ok) ++n;
  }
  return ok;
}

// D += A (16 x 16, row-major) * B (16 x 8, column-major), bf16 operands, fp32 accumulators (the warp-level tensor-core form)
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&a)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ uint32_t movmatrix(uint32_t a) {        // transpose of an 8 x 8 matrix of 16-bit values spread over the warp
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

// Shared memory of the tile in the general region: 47 KB.
struct GqSmem {
  float* raw;                // [10][128] raw rows: q heads, new k (each warp's own, for its norm)
  uint32_t* qb;              // [8][68] words = [8 heads][136] bf16: q rows, normed and rotated (heads past gq: zero)
  __nv_bfloat16* knew;       // [128] new k row
  __nv_bfloat16* vnew;       // [128] new v row
  float* st;                 // [8 slots][8 heads][2] running maximum, sum
  float* po;                 // [8 slots][1152] a warp's output sums: as fragments (handed from warp w + 8 to w), then [head][132]
  float* mg;                 // [16][32] partial sums of the merge
  __device__ explicit GqSmem(float* b) {
    raw = b; qb = (uint32_t*)(raw + 10 * 128); knew = (__nv_bfloat16*)(qb + 8 * 68); vnew = knew + 128;
    st = (float*)(vnew + 128); po = st + 8 * 8 * 2; mg = po + 8 * 1152;
  }
};
static_assert((10 * 128 + 8 * 68 + 128 + 128 + 8 * 1152 + 16 * 32) * 4 <= ETXB_GEN_BYTES, "the layout fits the general region");

// One head row (lane holds elements 4 lane ..): optional RMSNorm with weight nw (mean in numpy's order), then neox rotary.  xh: 128
// floats of the warp's own; o[j]: the bf16-rounded results.  Same arithmetic as head_norm_rope_s<128>, operands in registers.
__device__ __forceinline__ void head_norm_rope_r(uint2 x, float* xh, bool norm, uint2 nw, uint2 cs, uint2 sn, float eps, float (&o)[4]) {
  const int lane = tidx() & 31;
  float v[4] = {bf_lo(x.x), bf_hi(x.x), bf_lo(x.y), bf_hi(x.y)};
  if (norm) {
    const float wf[4] = {bf_lo(nw.x), bf_hi(nw.x), bf_lo(nw.y), bf_hi(nw.y)};
    *(float4*)(xh + 4 * lane) = make_float4(v[0], v[1], v[2], v[3]);
    __syncwarp();
    const float ss = sumsq128_numpy_order_warp(xh);
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(ss, 0.0078125f), eps)));
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = bfr(__fmul_rn(wf[j], bfr(__fmul_rn(v[j], r))));
  }
  const float cf[4] = {bf_lo(cs.x), bf_hi(cs.x), bf_lo(cs.y), bf_hi(cs.y)}, sf[4] = {bf_lo(sn.x), bf_hi(sn.x), bf_lo(sn.y), bf_hi(sn.y)};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float other = __shfl_xor_sync(0xffffffffu, v[j], 16);    // element d +- 64 lives 16 lanes away
    o[j] = bfr(__fadd_rn(bfr(__fmul_rn(v[j], cf[j])), bfr(__fmul_rn(lane < 16 ? -other : other, sf[j]))));
  }
}

template <bool WD>
__device__ __forceinline__ void gq_out(const etxb_attnf_args& d, const Smem& sm, int i, float v) {
  if (WD && (d.part_len & ETXB_GQ_WORDS)) st_word((uint32_t*)d.exp_sums + i, bf_bits(v) | s_vars.flag);
  if (!WD || d.out != nullptr) ((__nv_bfloat16*)d.out)[i] = __float2bfloat16_rn(v);
}
// one row of 128 values of this step's qkv, four per lane
template <bool WD>
__device__ __forceinline__ uint2 gq_row(const etxb_attnf_args& d, const Smem& sm, int row) {
  const int lane = tidx() & 31;
  if (WD && (d.part_len & ETXB_GQ_WORDS)) return words_pack(poll_words4((const uint32_t*)d.qkv + row * 128 + 4 * lane, s_vars.flag));
  return __ldcg((const uint2*)((const __nv_bfloat16*)d.qkv + (size_t)row * 128) + lane);
}

// out[h][:] = bf16(sum_p w_p * tmp[p][:] / sum_p w_p * l_p), w_p = exp(m_p - max m), for the 32-value slices mi, mi + mk, .. of the
// group's gq * 128 output values.  Polls the flagged partials the other CTAs publish (L2).  A warp takes a slice and a share of the
// partitions (its lane: one value); every warp works out its head's weights itself from the partitions' statistics.
// The order of the sums is a matter of gq and np alone (warps per slice, partitions per round): how many tasks share the merge (mk) differs between
// the sequences of a batch and between plans, and equal columns get equal bits.  Past 16 partitions shared merges fetch 32 at a time, four
// warps a slice; below, a warp a slice (all 16 slices of a round at once): against two warps, a phase of 8 sequences at 1033 positions 21.4 us /
// 22.3, of 16 at 1400 48.9 / 50.7, of 3 at 1400 13.3 / 13.4.  (As many warps as the slices of a task left free, 1 to 16: 22.4, 49.2 and 14.1.)
template <bool WD>
__device__ __forceinline__ void attn_gq_merge(const etxb_attnf_args& d, const Smem& sm, float* mg, int hq0, int np, uint32_t fl, int mi, int mk) {
  constexpr int HD = 128, NF = 8;
  const int lane = tidx() & 31, warp = tidx() >> 5;
  const int nsl = (d.gq * 4 - mi + mk - 1) / mk;                   // slices of this task
  const int wps = np > 16 && d.gq * np >= ETXB_GQ_SHARE ? 4 : d.gq > 2 ? 1 : d.gq == 2 ? 2 : 4;   // warps per slice
  const int per = 16 / wps, sub = warp / per;                      // slices per round; the warp's share of the partitions
#pragma unroll 1
  for (int s0 = 0; s0 < nsl; s0 += per) {
    const int si = s0 + (warp & (per - 1));
    const bool on = si < nsl;
    const int sl = mi + min(si, nsl - 1) * mk, g = sl >> 2;
    const uint2* tp = (const uint2*)d.tmp_out + (size_t)(hq0 + g) * d.max_parts * ETXB_GQ_PW;
    const uint2* vp = tp + (sl & 3) * 32 + lane;
    float o = 0.f, L = 0.f, M = -INFINITY;
    if (on) {
      // a round: up to 32 partitions' statistics (a lane each) and this warp's values of them, requested together -- the tail of the
      // phase is one trip to L2 behind the slowest partition.  Between rounds the sums are rescaled to the larger maximum.
      const int ch = min(32, NF * wps);
#pragma unroll 1
      for (int p0 = 0; p0 < np; p0 += ch) {
        const int pe = min(np - p0, ch);
        const uint2* sp = tp + (size_t)p0 * ETXB_GQ_PW + HD;
        uint2 first[NF];
        uint4 v;
        uint32_t spins = 0;
        for (;;) {
          v = ld_volatile16(sp + (size_t)min(lane, pe - 1) * ETXB_GQ_PW);      // (maximum, flag, sum, flag)
#pragma unroll
          for (int u = 0; u < NF; ++u) first[u] = ld_pair(vp + (size_t)(p0 + min(sub + u * wps, pe - 1)) * ETXB_GQ_PW);
          bool ok = v.y == fl && v.w == fl;
#pragma unroll
          for (int u = 0; u < NF; ++u) ok = ok && first[u].y == fl;
          if (ok || !poll_again(spins, sp, pe, ETXB_GQ_PW, fl, sm)) break;
        }
        __syncwarp();
        const float m = lane < pe ? __uint_as_float(v.x) : -INFINITY;
        const float Mn = fmaxf(M, warp_max(m)), Mz = Mn == -INFINITY ? 0.f : Mn;
        const float f = expf(__fsub_rn(M, Mz)), w = expf(__fsub_rn(m, Mz));    // (lanes past the round: 0)
        M = Mn;
        o = __fmul_rn(o, f);
        L = __fmaf_rn(L, f, lane < pe ? __fmul_rn(w, __uint_as_float(v.z)) : 0.f);
#pragma unroll
        for (int u = 0; u < NF; ++u) {
          const float wu = __shfl_sync(0xffffffffu, w, (sub + u * wps) & 31);
          if (sub + u * wps < pe) o = __fmaf_rn(wu, __uint_as_float(first[u].x), o);
        }
      }
      L = warp_sum(L);
    }
    if (wps > 1) {
      mg[warp * 32 + lane] = o;
      csync();
      if (sub == 0)
        for (int q = 1; q < wps; ++q) o = __fadd_rn(o, mg[(warp + q * per) * 32 + lane]);
    }
    if (on && sub == 0) gq_out<WD>(d, sm, hq0 * HD + sl * 32 + lane, __fdiv_rn(o, L));
    if (s0 + per < nsl && wps > 1) csync();
  }
}

// One task.  n: the running stage count of the ring.  mg: how the merge of a context in partitions is shared out -- 0: the task of the
// last partition merges the group (it comes last in the queues, and a task that waits only for tasks of lower index cannot be part of
// a circle); else count << 16 | index + 1: the host has found that the workers' LAST tasks of the grid may wait for all the others (the order of the
// queues and the events leave no circle: waiting_grids), and this is one of `count` such tasks of the group, each of which merges a share; 0xffff: it is not one of them, others are.  Shared out from
// gq * np = ETXB_GQ_SHARE on only: with few partials the last partition's task alone is as quick, and the other tasks are done.
// WD: the kernel's plans may hand the rows over as words.
template <bool WD>
__device__ __forceinline__ void attn_gq_tile(const etxb_attnf_args& d, int blk, const Smem& sm, const etxb_stepv& S, uint32_t& n, uint32_t mg) {
  constexpr int HD = 128, BS = 16;
  const GqTask t = gq_task(d, blk, S);
  const int NKV = d.NKV, gq = d.gq, tid = tidx(), lane = tid & 31, warp = tid >> 5;
  const uint32_t fl = pair_flag(sm.serial(), d.part_len);
  const int np = min((t.seq + ETXB_GQ_PART - 1) / ETXB_GQ_PART, d.max_parts);
  const GqSmem s(sm.xs);
  const uint32_t n0 = n;
  n += (uint32_t)((t.nu + ETXB_GQ_UPS - 1) / ETXB_GQ_UPS);
  if (t.nu > 0) {
    const bool newrow = t.owner || t.whole;
    // ---- this step's rows, a warp each: q heads, the new k row, the new v row
    if (warp < gq || (warp == gq && newrow)) {
      const bool isq = warp < gq;
      const void* nwp = isq ? d.qw : d.kw;
      const uint2 x = gq_row<WD>(d, sm, isq ? t.hq0 + warp : d.NH + t.h);
      const uint2* cs = (const uint2*)((const __nv_bfloat16*)d.cos_sin + (size_t)t.pos * HD);
      const uint2 nw = nwp ? __ldg((const uint2*)nwp + lane) : make_uint2(0u, 0u), c = __ldg(cs + (lane & 15)), sn = __ldg(cs + 16 + (lane & 15));
      float o[4];
      head_norm_rope_r(x, s.raw + warp * HD, nwp != nullptr, nw, c, sn, d.eps, o);
      const uint2 r = make_uint2(pack_bf(o[0], o[1]), pack_bf(o[2], o[3]));
      if (isq) *(uint2*)(s.qb + warp * 68 + 2 * lane) = r;
      else {
        *(uint2*)(s.knew + 4 * lane) = r;
        if (t.hq0 * NKV == t.h * d.NH) {                          // the kv head's first group stores the new k / v rows
          const long long slot = (const void*)d.slot_mapping == (const void*)S.slot_mapping ? (long long)S.pos : __ldcg((const long long*)d.slot_mapping);
          *(uint2*)((__nv_bfloat16*)d.kc + ((((size_t)(slot / BS) * NKV + t.h) * (HD / 8) + (lane >> 1)) * BS + (int)(slot % BS)) * 8 + 4 * (lane & 1)) = r;
        }
      }
    } else if (warp == gq + 1 && newrow) {
      const uint2 x = gq_row<WD>(d, sm, d.NH + NKV + t.h);
      *(uint2*)(s.vnew + 4 * lane) = x;
      if (t.hq0 * NKV == t.h * d.NH) {
        const long long slot = (const void*)d.slot_mapping == (const void*)S.slot_mapping ? (long long)S.pos : __ldcg((const long long*)d.slot_mapping);
        unsigned short* vc = (unsigned short*)d.vc + (((size_t)(slot / BS) * NKV + t.h) * HD + 4 * lane) * BS + (int)(slot % BS);
        vc[0] = (unsigned short)x.x; vc[BS] = (unsigned short)(x.x >> 16); vc[2 * BS] = (unsigned short)x.y; vc[3 * BS] = (unsigned short)(x.y >> 16);
      }
    }
    for (int i = gq * 68 + tid; i < 8 * 68; i += ETXB_CONSUMERS) s.qb[i] = 0u;
    csync();
    mark(sm, 0);
    // ---- the units, warp w: w, w + 16, ..
    const int g8 = lane >> 2, t4 = lane & 3, nwarp = min(t.nu, ETXB_CONSUMER_WARPS), where = sm.cur();
    float acc[8][4];                                               // [dims 16 i + g8, + 8][heads 2 t4, 2 t4 + 1]
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;      // of heads 2 t4, 2 t4 + 1 (l: this lane's positions)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    if (warp < nwarp) {
      const uint32_t* qw = s.qb + g8 * 68 + t4;                     // (read again for every unit: 16 registers fewer)
#pragma unroll 1
      for (int i = warp; i < t.nu; i += ETXB_CONSUMER_WARPS) {
        const int si = i / ETXB_GQ_UPS, ui = i - si * ETXB_GQ_UPS, p0 = (t.u0 + i) << 4;
        const uint32_t k = n0 + (uint32_t)si, st = k % ETXB_NSTAGE;
        // (the parity of a stage tells use k from use k - 1 only, and the use before this one may be another warp's: see wait_use)
        bool ok = wait_use((volatile const uint32_t*)(sm.full + 2 * ETXB_NSTAGE) + st, k, sm, where) && mbar_wait(sm.full + st, (k / ETXB_NSTAGE) & 1, sm, where);
        if (!__all_sync(0xffffffffu, ok)) break;                   // step abandoned: touch nothing
        unsigned char* unit = sm.ring + (size_t)st * ETXB_STAGE_BYTES + ui * ETXB_GQ_UNIT;
        // the unit at the end of the context: the new position's rows over its stale slot; a slot beyond the context may hold anything:
        // it is never multiplied (V: zero, K: the score below)
        const bool ragged = p0 + 16 > t.seq || (t.pos >= p0 && t.pos < p0 + 16);
        if (ragged) {
          const int rn = t.owner && t.pos >= p0 && t.pos < p0 + 16 ? (int)t.pos - p0 : -1;
          if (rn >= 0) *(uint2*)(unit + ((lane >> 1) * 16 + rn) * 16 + 8 * (lane & 1)) = *(const uint2*)(s.knew + 4 * lane);
          const int nv = max(0, min(16, t.seq - p0));              // positions of the context
          // Every 32nd piece of 16 bytes is the lane's: eight positions of one dim, the same eight for all its pieces.  (As 32 words a lane, one read,
          // change and write behind the other, the new position's task came 1.1 us after all others: a phase of a small dense model at
          // 200 positions, one q head a task, 8.0 us -> 7.4.)
          uint32_t keep[4], put[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int p = 8 * (lane & 1) + 2 * q;
            put[q] = (p == rn ? 0xffffu : 0u) | (p + 1 == rn ? 0xffff0000u : 0u);
            keep[q] = ((p < nv ? 0xffffu : 0u) | (p + 1 < nv ? 0xffff0000u : 0u)) & ~put[q];
          }
          uint4* vp = (uint4*)(unit + 4096) + lane;
          const unsigned short* vn = (const unsigned short*)s.vnew + (lane >> 1);
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            uint4 v[2];
            uint32_t x[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) { v[u] = vp[32 * (j + u)]; x[u] = vn[16 * (j + u)]; x[u] |= x[u] << 16; }
#pragma unroll
            for (int u = 0; u < 2; ++u)
              vp[32 * (j + u)] = make_uint4((v[u].x & keep[0]) | (x[u] & put[0]), (v[u].y & keep[1]) | (x[u] & put[1]),
                                            (v[u].z & keep[2]) | (x[u] & put[2]), (v[u].w & keep[3]) | (x[u] & put[3]));
          }
          __syncwarp();
        }
        const uint32_t ks = smem_u32(unit) + lane * 16, vs = smem_u32(unit) + 4096 + ((lane >> 4) << 4) + ((lane & 15) << 5);
        // Four fragments at a time, then their products (a load in front of every product is a chain of their latencies).  A tensor-core sum is
        // cut off, not rounded, where it leaves the 24 bits: every product begins at zero and the eight are added pairwise in fp32.
        float c[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t a[4][4], b[4][2];
          float qs[4][4];
#pragma unroll
          for (int j = 0; j < 16; ++j) qs[j >> 2][j & 3] = 0.f;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            ldmatrix_x4(a[u], ks + (4 * h + u) * 512);             // 16 positions x 16 dims
            b[u][0] = qw[8 * (4 * h + u)]; b[u][1] = qw[8 * (4 * h + u) + 4];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) mma16816(qs[u], a[u], b[u][0], b[u][1]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float v = __fadd_rn(__fadd_rn(qs[0][j], qs[1][j]), __fadd_rn(qs[2][j], qs[3][j]));
            c[j] = h == 0 ? v : __fadd_rn(c[j], v);
          }
        }
        // softmax of the unit: positions g8 (c[0], c[1]) and g8 + 8 (c[2], c[3]), heads 2 t4 and 2 t4 + 1
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = __fmul_rn(c[j], d.scale);
        if (ragged) {
          const int pa = p0 + g8, pb = pa + 8;
          if (pa >= t.seq && !(t.owner && pa == (int)t.pos)) c[0] = c[1] = -INFINITY;
          if (pb >= t.seq && !(t.owner && pb == (int)t.pos)) c[2] = c[3] = -INFINITY;
        }
        float n0m = fmaxf(c[0], c[2]), n1m = fmaxf(c[1], c[3]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) { n0m = fmaxf(n0m, __shfl_xor_sync(0xffffffffu, n0m, o)); n1m = fmaxf(n1m, __shfl_xor_sync(0xffffffffu, n1m, o)); }
        n0m = fmaxf(m0, n0m); n1m = fmaxf(m1, n1m);
        const float b0 = n0m == -INFINITY ? 0.f : n0m, b1 = n1m == -INFINITY ? 0.f : n1m;   // (nothing valid yet: every probability is 0)
        if (i != warp) {
          const float f0 = expf(__fsub_rn(m0, b0)), f1 = expf(__fsub_rn(m1, b1));
          l0 = __fmul_rn(l0, f0); l1 = __fmul_rn(l1, f1);
#pragma unroll
          for (int j = 0; j < 8; ++j) { acc[j][0] *= f0; acc[j][1] *= f1; acc[j][2] *= f0; acc[j][3] *= f1; }
        }
        m0 = n0m; m1 = n1m;
        c[0] = expf(__fsub_rn(c[0], b0)); c[1] = expf(__fsub_rn(c[1], b1)); c[2] = expf(__fsub_rn(c[2], b0)); c[3] = expf(__fsub_rn(c[3], b1));
        l0 = __fadd_rn(l0, __fadd_rn(c[0], c[2])); l1 = __fadd_rn(l1, __fadd_rn(c[1], c[3]));
        float r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = __fsub_rn(c[j], bfr(c[j]));
        const uint32_t h0 = movmatrix(pack_bf(c[0], c[1])), h1 = movmatrix(pack_bf(c[2], c[3]));
        const uint32_t w0 = movmatrix(pack_bf(r[0], r[1])), w1 = movmatrix(pack_bf(r[2], r[3]));
        uint32_t x0 = 0u, x1 = 0u;
        const bool third = ragged || (d.part_len & (ETXB_GQ_WHOLE | ETXB_GQ_PRECISE)) != ETXB_GQ_WHOLE;
        if (third) {                                               // what the second rounding lost
#pragma unroll
          for (int j = 0; j < 4; ++j) r[j] = __fsub_rn(r[j], bfr(r[j]));
          x0 = movmatrix(pack_bf(r[0], r[1])); x1 = movmatrix(pack_bf(r[2], r[3]));
        }
        // (two fragments at a time, four spill; the small parts first, and their sum rounded into the large one's: see the scores)
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          uint32_t a[2][4];
          float lo[2][4], hi[2][4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            ldmatrix_x4(a[u], vs + (j + u) * 512);                 // 16 dims x 16 positions (matrices: dims 0-7, 8-15 of positions 0-7, then of 8-15)
#pragma unroll
            for (int e = 0; e < 4; ++e) lo[u][e] = hi[u][e] = 0.f;
          }
          if (third)
#pragma unroll
            for (int u = 0; u < 2; ++u) mma16816(lo[u], a[u], x0, x1);
#pragma unroll
          for (int u = 0; u < 2; ++u) mma16816(lo[u], a[u], w0, w1);
#pragma unroll
          for (int u = 0; u < 2; ++u) mma16816(hi[u], a[u], h0, h1);
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              // (an infinite V: its product with a small part is NaN where the part is 0 or has another sign than the probability)
              const float v = fabsf(hi[u][e]) < INFINITY ? __fadd_rn(hi[u][e], lo[u][e]) : hi[u][e];
              acc[j + u][e] = __fadd_rn(acc[j + u][e], v);
            }
        }
        if (ragged) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // (this warp's writes, before the next copy into the place)
        __syncwarp();
        const int in_stage = min(t.nu - si * ETXB_GQ_UPS, ETXB_GQ_UPS), share = ETXB_EMPTY_COUNT / ETXB_GQ_UPS;
        if (lane == 0) mbar_arrive_n(sm.empty + st, ui == in_stage - 1 ? ETXB_EMPTY_COUNT - ui * share : share);
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) { l0 += __shfl_xor_sync(0xffffffffu, l0, o); l1 += __shfl_xor_sync(0xffffffffu, l1, o); }
    }
    // ---- the warps' results: warp w + 8 hands its fragments to warp w, then the eight meet in shared memory
    if (nwarp > 8) {
      float4* box = (float4*)(s.po + (warp & 7) * 1152);
      if (warp >= 8 && warp < nwarp) {
#pragma unroll
        for (int j = 0; j < 8; ++j) box[j * 32 + lane] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        box[256 + lane] = make_float4(m0, m1, l0, l1);
      }
      csync();
      if (warp + 8 < nwarp) {
        const float4 o = box[256 + lane];
        const float a0 = fmaxf(m0, o.x), a1 = fmaxf(m1, o.y), z0 = a0 == -INFINITY ? 0.f : a0, z1 = a1 == -INFINITY ? 0.f : a1;
        const float f0 = expf(__fsub_rn(m0, z0)), f1 = expf(__fsub_rn(m1, z1)), e0 = expf(__fsub_rn(o.x, z0)), e1 = expf(__fsub_rn(o.y, z1));
        m0 = a0; m1 = a1;
        l0 = __fmaf_rn(l0, f0, __fmul_rn(o.z, e0)); l1 = __fmaf_rn(l1, f1, __fmul_rn(o.w, e1));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 v = box[j * 32 + lane];
          acc[j][0] = __fmaf_rn(acc[j][0], f0, __fmul_rn(v.x, e0)); acc[j][1] = __fmaf_rn(acc[j][1], f1, __fmul_rn(v.y, e1));
          acc[j][2] = __fmaf_rn(acc[j][2], f0, __fmul_rn(v.z, e0)); acc[j][3] = __fmaf_rn(acc[j][3], f1, __fmul_rn(v.w, e1));
        }
        __syncwarp();
      }
    }
    const int nslot = min(nwarp, 8);
    if (warp < nslot) {
      float* po = s.po + warp * 1152 + (2 * t4) * 132 + g8;
      const bool hA = 2 * t4 < gq, hB = 2 * t4 + 1 < gq;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (hA) { po[16 * j] = acc[j][0]; po[16 * j + 8] = acc[j][2]; }
        if (hB) { po[132 + 16 * j] = acc[j][1]; po[132 + 16 * j + 8] = acc[j][3]; }
      }
      if (g8 == 0) *(float4*)(s.st + (warp * 8 + 2 * t4) * 2) = make_float4(m0, l0, m1, l1);
    }
    csync();
    mark(sm, 1);
    for (int idx = tid; idx < gq * HD; idx += ETXB_CONSUMERS) {
      // a warp's 32 outputs are one head's: lane w works out slot w's factor (one exponential instead of eight), the sums take them by shuffle.
      // (Eight exponentials in every thread: 0.76 us from the barrier to the stores, so 0.51.)
      const int g = idx >> 7, dd = idx & (HD - 1), w0 = lane & 7;
      const float2 ml = w0 < nslot ? *(const float2*)(s.st + (w0 * 8 + g) * 2) : make_float2(-INFINITY, 0.f);
      float M = ml.x;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
      const float f = expf(__fsub_rn(ml.x, M == -INFINITY ? 0.f : M));
      float o = 0.f, L = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float fw = __shfl_sync(0xffffffffu, f, w), lw = __shfl_sync(0xffffffffu, ml.y, w);
        if (w < nslot) {
          L = __fmaf_rn(fw, lw, L);
          o = __fmaf_rn(fw, s.po[w * 1152 + g * 132 + dd], o);
        }
      }
      if (t.whole || np == 1) {
        gq_out<WD>(d, sm, t.hq0 * HD + idx, __fdiv_rn(o, L));
      } else {
        uint2* pw = (uint2*)d.tmp_out + ((size_t)(t.hq0 + g) * d.max_parts + t.part) * ETXB_GQ_PW;
        st_pair(pw + dd, o, fl);
        if (dd == 0) { st_pair(pw + HD, M, fl); st_pair(pw + HD + 1, L, fl); }
      }
    }
  }
  mark(sm, 2);
  // (a merge never looks past the partitions the grid computed, whatever seq_lens says)
  if (gq * np < ETXB_GQ_SHARE) mg = 0u;
  if (!t.whole && np > 1) {
    if (mg == 0u ? t.part == np - 1 : mg != 0xffffu) attn_gq_merge<WD>(d, sm, s.mg, t.hq0, np, fl, mg == 0u ? 0 : (int)(mg & 0xffffu) - 1, mg == 0u ? 1 : (int)(mg >> 16));
  }
  mark(sm, 3);
}

}  // namespace etxb
