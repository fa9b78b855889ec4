// The persistent kernel: one CTA per SM walks its static task queue; per task it waits for the task's events
// (acquire, bounded), runs the tile body, drains its stores and arrives on the out events (release).
//
// Takes over the generated kernel of the reference: worker loop etx/codegen/kernel.py:517-572, the three-phase
// etx_run_task kernel.py:341-468, and the native prologue / argmax tiles examples/vllm_llm/vl_tiles.hip:31-89.
#pragma once
#include "etxb_attn.cuh"
#include "etxb_attn_gq.cuh"
#include "etxb_batch.cuh"
#include "etxb_tc.cuh"
#include "etxb_mla.cuh"
#include "etxb_gemv.cuh"
#include "etxb_prims.cuh"

namespace etxb {

// resid <- embedding row of token_in[t] (nrep copies), positions / seq_lens / slot_mapping <- pos (identity block table)
__device__ __forceinline__ void tile_prologue(const etxb_stepv& S) {
  const int t = S.tok;
  if (tidx() == 0) {
    if (S.token_time) S.token_time[2 * t] = globaltimer();
    S.positions[0] = S.pos; S.seq_lens[0] = S.pos + 1; S.slot_mapping[0] = S.pos;
  }
  const int id = __ldcg(S.token_in + t);
  const uint4* src = (const uint4*)((const __nv_bfloat16*)S.embed + (size_t)id * S.H);
  uint4* dst = (uint4*)S.resid;
  const int n8 = S.H / 8;
  for (int i = tidx(); i < n8 * S.nrep; i += ETXB_CONSUMERS) dst[i] = __ldg(src + i % n8);
}

// greedy sampling: first maximum of the bf16 logits (ties -> lower index, like argmax over float32)
// Sharded lm_head (p.xargmax != 0): the logits are this rank's V of ranks x V, so the rank's (maximum, global index) goes
// into its slot of every rank's argmax block as two 8-byte (payload, step flag) stores -- each atomic, so no fence --
// and the token is the best of all ranks' pairs, ties to the lower index: the same on every rank.
__device__ __forceinline__ void st_volatile8(void* p, uint32_t a, uint32_t b) {
  asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void argmax_exchange(const etxb_params& p, const Smem& sm, float& bv, int& bi) {
  const uint32_t fl = row_flag(p.epoch);
  bi += p.rank * p.step.V;
  const int q_self = p.rank;
  for (int q = 0; q <= p.n_peers; ++q) {                            // peers in xpeer order (ranks without this one), then this rank
    unsigned char* base = q < p.n_peers ? p.xpeer[q] : p.xbase;
    unsigned char* slot = base + p.xargmax + 16 * (size_t)q_self;
    st_volatile8(slot, __float_as_uint(bv), fl);
    st_volatile8(slot + 8, (uint32_t)bi, fl);
  }
  for (int r = 0; r <= p.n_peers; ++r) {
    if (r == p.rank) continue;
    const unsigned char* slot = p.xbase + p.xargmax + 16 * (size_t)r;
    uint2 a, b;
    uint32_t spins = 0;
    for (;;) {
      a = ld_volatile8(slot); b = ld_volatile8(slot + 8);
      if (a.y == fl && b.y == fl) break;
      if ((++spins & 63u) == 0) {
        if (ld_relaxed(sm.ctrl()) != 0) { *(volatile int*)sm.stop = 1; return; }
        if ((spins & 1023u) == 0 && globaltimer() > *sm.deadline) {
          if (atomicOr(sm.ctrl(), ETXB_CTRL_TIMEOUT) == 0) { sm.ctrl()[1] = sm.cur(); sm.ctrl()[2] = -100 - r; sm.ctrl()[3] = (int32_t)(a.y >> 16); sm.ctrl()[4] = (int32_t)(fl >> 16); }
          *(volatile int*)sm.stop = 1;
          return;
        }
        __nanosleep(32);
      }
    }
    const float ov = __uint_as_float(a.x);
    const int oi = (int)b.x;
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
}

// col / ncols: column `col` of a batched step (logits [ncols][V], token_in / token_out [step][ncols]); (0, 1) otherwise.
template <bool XCH>
__device__ __forceinline__ void tile_argmax(const etxb_params& p, const Smem& sm, int col = 0, int ncols = 1) {
  const etxb_stepv& S = p.step;
  float bv = -INFINITY; int bi = 0x7fffffff;
  const uint4* lg4 = (const uint4*)((const __nv_bfloat16*)S.logits + (size_t)col * S.V);
  const int n4 = S.V / 8;
  // One CTA reads the row (300 KB for 151936 logits), so what counts is how much of it is in flight: 12 vectors per thread
  // (96 KB), compared by their largest element (packed maxima); the element itself is looked up in the one vector that
  // won.  4 in flight, every element compared: 8.8 us; now 7.0 (one SM's share of the L2 bandwidth is 2.5).
  // (max of bf16 pairs drops NaN like the comparison does; +0 and -0 compare equal, so the lookup takes the first of them)
  int bj = -1;
  const int B = ETXB_CONSUMERS;
  constexpr int NF = 12;
  for (int j0 = tidx(); j0 < n4; j0 += NF * B) {
    uint4 w[NF];
#pragma unroll
    for (int k = 0; k < NF; ++k) w[k] = ld_act16(lg4 + min(j0 + k * B, n4 - 1));
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      const uint32_t m = max_bf2(max_bf2(w[k].x, w[k].y), max_bf2(w[k].z, w[k].w));
      const float v = fmaxf(bf_lo(m), bf_hi(m));
      if (j0 + k * B < n4 && v > bv) { bv = v; bj = j0 + k * B; }
    }
  }
  if (bj >= 0) {
    const uint4 w = ld_act16(lg4 + bj);
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      if (bf_hi(u[k]) == bv) bi = 8 * bj + 2 * k + 1;
      if (bf_lo(u[k]) == bv) bi = 8 * bj + 2 * k;
    }
  }
  for (int i = 8 * n4 + tidx(); i < S.V; i += B) {
    const float v = ld_bf(lg4, i);
    if (v > bv) { bv = v; bi = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  float* sv = sm.scr; int* si = (int*)(sm.scr + 32);
  if ((tidx() & 31) == 0) { sv[tidx() >> 5] = bv; si[tidx() >> 5] = bi; }
  csync();
  if (tidx() == 0) {
    for (int w = 1; w < ETXB_NWARPS; ++w)
      if (sv[w] > bv || (sv[w] == bv && si[w] < bi)) { bv = sv[w]; bi = si[w]; }
    if constexpr (XCH) { if (p.n_peers > 0 && p.xargmax != 0u) argmax_exchange(p, sm, bv, bi); }
    const int t = S.tok;
    S.token_out[(size_t)t * ncols + col] = bi;
    if (S.write_next) S.token_in[(size_t)(t + 1) * ncols + col] = bi;
    if (S.token_time && col == ncols - 1) S.token_time[2 * t + 1] = globaltimer();
  }
}

// protocol demo (etx/operators/splitk_sum.py:10-33): parts[i][j] = sum of chunk j of row i; out[i] = sum_j parts[i][j]
__device__ __forceinline__ void tile_splitk_part(const unsigned char* a, int i, int j, const Smem& sm) {
  const etxb_splitk_args& d = *(const etxb_splitk_args*)a;
  const int w = d.cols / d.chunks;
  float s = 0.f;
  for (int c = tidx(); c < w; c += ETXB_CONSUMERS) s += __ldcg(d.in + (size_t)i * d.cols + j * w + c);
  s = block_sum(s, sm.scr);
  if (tidx() == 0) d.parts[i * d.chunks + j] = s;
}
__device__ __forceinline__ void tile_splitk_sum(const unsigned char* a, int i) {
  const etxb_splitk_args& d = *(const etxb_splitk_args*)a;
  if (tidx() == 0) {
    float s = 0.f;
    for (int j = 0; j < d.chunks; ++j) s += __ldcg(d.parts + i * d.chunks + j);
    d.out[i] = s;
  }
}

// A task's context in shared memory: its record and a copy of its argument block.  The last consumer warp fetches them
// with asynchronous copies (cp.async) while earlier bodies run -- the record two tasks ahead, the argument block one
// task ahead (its address is in the record) -- and only waits for them at the end of a body, so the chain task ->
// arguments -> data costs the tiles no dependent global round trip and the fetch itself is off the critical path.
struct TaskCtx {
  etxb_rec r;
  unsigned char args[ETXB_CTX_BYTES - 96];
};
static_assert(sizeof(etxb_rec) == 96 && sizeof(TaskCtx) == ETXB_CTX_BYTES, "context slot layout");

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// one warp: lanes 0..5 fetch the record of task `rec_task`, lanes 8..19 the argument block of task `arg_task` (whose
// record must already be in its slot); -1 skips either.  Asynchronous: cp_async_wait_all() completes them.
__device__ __forceinline__ void fetch_ctx(const etxb_params& p, TaskCtx* ctx, int q0, int rec_task, int arg_task) {
  const int lane = tidx() & 31;
  if (rec_task >= 0 && lane < 6) cp_async16((unsigned char*)&ctx[(rec_task - q0) & (ETXB_CTX_SLOTS - 1)].r + 16 * lane,
                                            (const unsigned char*)(p.recs + rec_task) + 16 * lane);
  if (arg_task >= 0 && lane >= 8 && lane < 20) {
    TaskCtx* c = ctx + ((arg_task - q0) & (ETXB_CTX_SLOTS - 1));
    cp_async16(c->args + 16 * (lane - 8), (const unsigned char*)c->r.args + 16 * (lane - 8));
  }
}

__shared__ __align__(8) TcShared s_tc;                             // (used by the kernels of a batched plan only)
__device__ __forceinline__ Smem smem_view() {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem sm;
  sm.ring = smem_raw;
  sm.xs = (float*)(smem_raw + ETXB_RING_BYTES);
  sm.scr = (float*)(smem_raw + ETXB_RING_BYTES + ETXB_GEN_BYTES);
  sm.full = (uint64_t*)(smem_raw + ETXB_RING_BYTES + ETXB_GEN_BYTES + ETXB_SCR_FLOATS * 4);
  sm.empty = sm.full + ETXB_NSTAGE;
  sm.prod = (int32_t*)(sm.empty + ETXB_NSTAGE) + 8;                 // (behind the notes of the stages' uses)
  sm.deadline = &s_deadline; sm.stop = &s_stop; sm.geo = &s_geo; sm.vars = &s_vars;
  return sm;
}
// A tile of the full kernel or of the batched step.  These are calls: each tile gets the registers for itself (inlined side by
// side they spilled into each other's paths).
template <int B>
__device__ __noinline__ void batch_call(const unsigned char* args, int c0, int cur, const etxb_stepv& S) {
  const Smem sm = smem_view();
  if constexpr (B == 18) tile_prologue_nb(args, c0, S);
  else if constexpr (B == 13) tile_norm_col(args, c0, sm);
  else if constexpr (B == 15) tile_route(args, c0, sm);
  else if constexpr (B == 20) tile_gemv_tc(args, c0, sm, s_tc, cur);
  else if constexpr (B == 21) tile_moe_up_tc(args, c0, sm, s_tc, cur);
  else if constexpr (B == 22) tile_moe_down_tc(args, c0, sm, s_tc, cur);
  else if constexpr (B == 7) tile_attnprep(args, c0, sm, S);
  else if constexpr (B == 8) tile_attn(args, c0, sm, S);
  else if constexpr (B == 9) tile_attn_reduce(args, c0, sm, S);
  else if constexpr (B == 12) attn_fused_impl<0, 0>(*(const etxb_attnf_args*)args, c0, sm, S);
  else attn_fused_impl<128, 16>(*(const etxb_attnf_args*)args, c0, sm, S);
}
__device__ __noinline__ void argmax_col_call(const etxb_params& p, const unsigned char* args, int c0) {
  const int nb = ((const etxb_batch_args*)args)->nb;
  if (c0 < nb) tile_argmax<false>(p, smem_view(), c0, nb);
}
// Attention out of a kernel that holds all its forms, a call each: the grouped form (gq > 0 in the argument block; head_dim 128,
// cache blocks of 16) and, in the full kernel, the general tile and latent attention.  They return the running stage count of the ring.
template <bool WD>
__device__ __noinline__ uint32_t attn_call(const etxb_attnf_args& d, int blk, const etxb_stepv& S, uint32_t n, uint32_t mg) {
  attn_gq_tile<WD>(d, blk, smem_view(), S, n, mg);
  return n;
}
__device__ __noinline__ uint32_t narrow_call(const unsigned char* args, int blk, uint32_t n) {
  tile_gemv_narrow(args, blk, smem_view(), n);
  return n;
}
__device__ __noinline__ uint32_t mla_call(const unsigned char* args, int blk, const etxb_stepv& S, uint32_t n) {
  tile_mla_attn(args, blk, smem_view(), S, n);
  return n;
}
// (in the full kernel: inlined there, its code spilled into the other tiles' paths)
template <bool XCH>
__device__ __noinline__ uint32_t gemv_call(int body, const unsigned char* args, int blk, uint32_t n, int cur) {
  tile_gemv_family<false, XCH, true>(body, args, blk, smem_view(), n, cur);
  return n;
}
template <bool GENERAL>
__device__ __forceinline__ void tile_attn_any(const unsigned char* a, int blk, int cur, const etxb_stepv& S, uint32_t& n, uint32_t mg) {
  const etxb_attnf_args& d = *(const etxb_attnf_args*)a;
  if (blk >= (int)d.nblocks || d.gq < 0) return;
  if (d.gq == 0) {
    if constexpr (GENERAL) { if (attn_fused_128(d)) batch_call<12 + 128>(a, blk, cur, S); else batch_call<12>(a, blk, cur, S); }
    return;
  }
  n = attn_call<GENERAL>(d, blk, S, n, mg);
}

// Run the body of the task whose context is `c` on the consumer warps.
// KV: the kernel variant.  0 = every tile.  ETXB_VARIANT_LEAN = the lean decode kernel: only the tiles of a fused decode step
// (prologue, argmax, the GEMV family with norm folds of at most one row and top-k folds over at most 128 experts, the
// grouped attention tile); ETXB_VARIANT_MLA = the lean kernel of a latent-attention model (the
// same GEMV family with the latent-attention tile in place of the grouped one); ETXB_VARIANT_BATCH = the tiles of a batched step
// on the tensor cores.  The host picks it from the plan (select_variant): the full
// kernel is 1020 KB of code, of which a decode step uses a fraction scattered through it, and its tiles are calls.  From the
// 142 KB kernel (same bits): 12 layers of a 128-expert model 794 -> 693 us, of a dense one 1393 -> 1253; 9 layers of a
// latent-attention model 794 -> 689 from its 170 KB; the batched kernel (610 KB) gives 1 to 5 % (batched_plan).  (Sizes as measured
// then; since the attention tile is one for all group sizes 721, 150, 160 and 315 KB.)
// XCH: the variants a sharded session launches -- the same bodies plus the exchange code (flagged-row folds of R = ranks
// rows, row publishing after the body, the argmax exchange); compiled out of the others.
#define ETXB_VARIANT_LEAN 1
#define ETXB_VARIANT_MLA 16
#define ETXB_VARIANT_BATCH 32         // the batched step on the tensor cores: its tiles and the attention tiles, nothing else
template <int KV, bool XCH>
__device__ __forceinline__ void run_body(const etxb_params& p, const TaskCtx* c, int cur, const Smem& sm, uint32_t& n) {
  const unsigned char* args = c->args;
  const int c0 = c->r.c0, c1 = c->r.c1;
  constexpr bool LEAN = KV != 0;
  constexpr bool SH = KV == 0 || KV == ETXB_VARIANT_MLA;         // always-on (shared) experts: the full kernel and the latent-attention variant
  constexpr bool FULL = KV == 0, BATCHED = KV == ETXB_VARIANT_BATCH;
  // (a body this variant does not hold: the host picks the variant from the plan's bodies, so this is a corrupted record)
#define ETXB_TILE(cond, call) if constexpr (cond) { call; } else { if (tidx() == 0) atomicOr(p.ctrl, ETXB_CTRL_BADTASK); } break
  if constexpr (LEAN && !BATCHED) {                                // (four of five phases; a jump table first is a trip for its entry)
    if ((unsigned)(c->r.body - 3) < 3u) { tile_gemv_family<LEAN, XCH, SH>(c->r.body, args, c0, sm, n, cur); return; }
  }
  switch (c->r.body) {
    case 0: break;
    case 1: ETXB_TILE(!BATCHED, tile_prologue(p.step));
    case 2: ETXB_TILE(!BATCHED, tile_argmax<XCH>(p, sm));
    case 3: case 4: case 5: ETXB_TILE(FULL, n = gemv_call<XCH>(c->r.body, args, c0, n, cur));
    case 12:
      if constexpr (KV == ETXB_VARIANT_MLA) { if (tidx() == 0) atomicOr(p.ctrl, ETXB_CTRL_BADTASK); }      // (the latent-attention variant has no GQA tile)
      else if constexpr (KV == ETXB_VARIANT_LEAN) {
        const etxb_attnf_args& d = *(const etxb_attnf_args*)args;
        if (c0 < (int)d.nblocks && d.gq > 0) attn_gq_tile<!XCH>(d, c0, sm, p.step, n, c->r.mirror);
      } else tile_attn_any<FULL>(args, c0, cur, p.step, n, c->r.mirror);
      break;
    case 6: ETXB_TILE(!LEAN, tile_topk(args, c0, sm));
    case 7: ETXB_TILE(!LEAN, batch_call<7>(args, c0, cur, p.step));
    case 8: ETXB_TILE(!LEAN, batch_call<8>(args, c0, cur, p.step));
    case 9: ETXB_TILE(!LEAN, batch_call<9>(args, c0, cur, p.step));
    case 10: ETXB_TILE(!LEAN, tile_splitk_part(args, c0, c1, sm));
    case 11: ETXB_TILE(!LEAN, tile_splitk_sum(args, c0));
    // batched decode (several columns per step).  The mma.sync tiles (14, 16, 17) are inlined: their loops want every register, and
    // a call saves the caller's on the stack first.  3 layers of 64 experts: 8 sequences at 1000 positions 818 us with calls, 661
    // inlined; 32 at 300 positions 1416, 1199.
    case 13: ETXB_TILE(FULL || BATCHED, batch_call<13>(args, c0, cur, p.step));
    case 14: ETXB_TILE(!LEAN, tile_gemv_nb(args, c0, sm));
    case 15: ETXB_TILE(FULL || BATCHED, batch_call<15>(args, c0, cur, p.step));
    case 16: ETXB_TILE(!LEAN, tile_moe_up_g(args, c0, sm));
    case 17: ETXB_TILE(!LEAN, tile_moe_down_g(args, c0, sm));
    case 18: ETXB_TILE(FULL || BATCHED, batch_call<18>(args, c0, cur, p.step));
    case 19: ETXB_TILE(FULL || BATCHED, argmax_col_call(p, args, c0));
    case 20:
      if constexpr ((FULL || BATCHED) && !XCH) {
        if (((const etxb_gemv_args*)args)->tpe > 1) n = narrow_call(args, c0, n);
        else batch_call<20>(args, c0, cur, p.step);
      } else if (tidx() == 0) atomicOr(p.ctrl, ETXB_CTRL_BADTASK);
      break;
    case 21: ETXB_TILE((FULL || BATCHED) && !XCH, batch_call<21>(args, c0, cur, p.step));
    case 22: ETXB_TILE((FULL || BATCHED) && !XCH, batch_call<22>(args, c0, cur, p.step));
    case 23:
      if constexpr (KV == ETXB_VARIANT_MLA) tile_mla_attn(args, c0, sm, p.step, n);
      else { ETXB_TILE(FULL, n = mla_call(args, c0, p.step, n)); }
      break;
    default:
      if (tidx() == 0) atomicOr(p.ctrl, ETXB_CTRL_BADTASK);
      break;
  }
#undef ETXB_TILE
}

// Producer warp: waits for what the addresses of a task's stream depend on; false when the step is being abandoned.
__device__ __forceinline__ bool producer_wait(const etxb_params& p, const Smem& sm, const etxb_rec* t, int cur) {
  const int sw = t->stream_word;
  if (sw == -1) return true;                                       // (an abandoned step ends at a stage that nobody gives back; a look at the word here is a trip to L2 per task)
  int good = 1;
  if ((tidx() & 31) == 0) {
    if (sw >= 0) good = wait_event(p, sw, (int32_t)(p.epoch * (uint32_t)p.evcount[sw]), cur, *sm.deadline) ? 1 : 0;
    else
      for (int i = 0; good && i < (t->in_n & (ETXB_IN_ROUTED - 1)); ++i) {
        const int word = i < 4 ? t->in_word[i] : p.inwords[t->in_off + i];
        good = wait_event(p, word, (int32_t)(p.epoch * (uint32_t)p.evcount[word]), cur, *sm.deadline) ? 1 : 0;
      }
  }
  return __shfl_sync(0xffffffffu, good, 0) != 0;
}

// .. until every task of the queue before `cur` is over; false when the step is being abandoned.
__device__ __forceinline__ bool queue_done(const Smem& sm, int cur) {
  int good = 1;
  if ((tidx() & 31) == 0) good = wait_done(sm, cur) ? 1 : 0;
  return __shfl_sync(0xffffffffu, good, 0) != 0;
}

// The producer warp: walks the same queue ahead of the consumers and streams the weight rows of every GEMV-family
// task into the ring.  It waits only for what the weight ADDRESSES depend on (nothing for static weights, the router's
// event for expert weights), never for the task's activations.
// Attention tasks: the K / V units of their positions (GQ: grouped), W_UK and the cached rows (MLA: latent attention).  In a kernel whose
// other tiles use the ring's memory as their own (TC: the tensor-core tiles) the copies wait until every task before this one is over;
// they still run ahead of the task's events.  The same for weights in a plan that has such tiles (none of the bundled ones mixes them).
template <bool LEAN, bool SH, bool GEMV, bool GQ, bool MLA, bool TC>
__device__ __forceinline__ void producer_loop(const etxb_params& p, const Smem& sm, int q0, int q1) {
  uint32_t n = 0;
  const int lane = tidx() & 31;
  bool ok = true;
  for (int cur = q0; cur < q1 && ok; ++cur) {
    const etxb_rec* t = p.recs + cur;
    const int body = t->body;
    if constexpr (GQ || MLA) {
      if ((GQ && body == 12) || (MLA && body == 23) || (TC && body == 20)) {
        etxb_attnf_args* aa = (etxb_attnf_args*)(sm.prod + 32);
        __syncwarp();
        if (lane < (int)(sizeof(etxb_attnf_args) / 8)) ((uint64_t*)aa)[lane] = __ldg((const uint64_t*)t->args + lane);   // (at least as long as the other block)
        __syncwarp();
        if (body == 12 && aa->gq <= 0) continue;
        if (TC && body == 20 && ((const etxb_gemv_args*)aa)->tpe <= 1) continue;
        if constexpr (TC) { if (!queue_done(sm, cur)) break; }
        if constexpr (TC) {
          if (body == 20) {                                        // (static weights)
            if (ld_relaxed(p.ctrl) != 0) break;
            ok = produce_narrow(*(const etxb_gemv_args*)aa, t->c0, n, sm, cur);
            continue;
          }
        }
        if (!producer_wait(p, sm, t, cur)) break;
        if constexpr (GQ && MLA) ok = body == 12 ? produce_attn(*aa, t->c0, p.step, n, sm, cur) : produce_mla(*(const etxb_mla_args*)aa, t->c0, p.step, n, sm, cur);
        else if constexpr (GQ) ok = produce_attn(*aa, t->c0, p.step, n, sm, cur);
        else ok = produce_mla(*(const etxb_mla_args*)aa, t->c0, p.step, n, sm, cur);
        continue;
      }
    }
    if (!GEMV || body < 3 || body > 5) continue;
    // the argument block through shared memory, fetched BEFORE the wait below (it depends on no event)
    etxb_gemv_args* pa = (etxb_gemv_args*)(sm.prod + 32);
    if (lane < 20) ((uint64_t*)pa)[lane] = __ldg((const uint64_t*)t->args + lane);
    __syncwarp();
    GemvGeom gg;                                                   // (nor does the task's geometry)
    gg.t = gemv_task(body, *pa, t->c0);
    gemv_stages(body, pa->mode, gg);
    const GemvTask gt = gg.t;
    if constexpr (TC) { if (p.tc_on != 0u && !queue_done(sm, cur)) break; }
    // (a down grid behind its gate+up grid: the ids are there.  With the event waited for and the top-k done again, 2 us, its stream began
    // when the gate+up rows in the ring were used up)
    if (!(t->in_n & ETXB_IN_ROUTED)) {
      if (!producer_wait(p, sm, t, cur)) break;
      if (gt.n > 0 && body != 3) gemv_routing<LEAN, SH>(*pa, sm.prod, nullptr);  // (the ids alone: the stream waits for them)
    }
    ok = produce_task<SH>(body, *pa, gt, gg.rps, gg.spr != 0, sm.prod, n, sm, cur, p.trace ? p.trace + 8 * (size_t)t->id : nullptr);
  }
  // Nothing is left in flight on a normal exit (the consumers waited for every stage).  When the step was abandoned,
  // wait (bounded) for the copies already issued before the CTA's shared memory goes away.
  if (ld_relaxed(p.ctrl) != 0 && lane == 0) {
    const uint32_t issued = n < ETXB_NSTAGE ? n : ETXB_NSTAGE;
    for (uint32_t k = 0; k < issued; ++k) {
      const uint32_t m = n - 1 - k, st = m % ETXB_NSTAGE, par = (m / ETXB_NSTAGE) & 1;
      for (int spin = 0; spin < 2000000 && !mbar_try_wait(sm.full + st, par); ++spin) {}
    }
  }
}

template <int KV, bool XCH = false>
__global__ void __launch_bounds__(ETXB_THREADS, 1) etxb_megakernel(const __grid_constant__ etxb_params p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr bool TC = (KV == 0 || KV == ETXB_VARIANT_BATCH) && !XCH;
  const Smem sm = smem_view();
  if (threadIdx.x == 0) {
    s_stop = 0;
    s_vars.ctrl = p.ctrl; s_vars.tr = nullptr; s_vars.serial = p.serial; s_vars.flag = row_flag(p.epoch); s_vars.cur = 0; s_vars.halt = 0; s_vars.hold = 0; s_vars.done = -1;
    s_deadline = globaltimer() + p.timeout_ns;
    for (int i = 0; i < ETXB_NSTAGE; ++i) { mbar_init(sm.full + i, 1); mbar_init(sm.empty + i, ETXB_EMPTY_COUNT); ((uint32_t*)(sm.empty + ETXB_NSTAGE))[i] = 0xffffffffu; }
    if constexpr (TC) {
      for (int i = 0; i < ETXB_TC_MAXSTAGE; ++i) { mbar_init(s_tc.full + i, 1); mbar_init(s_tc.empty + i, 1); s_tc.lu[i] = 0; s_tc.mu[i] = 0; }
      for (int i = 0; i < 2; ++i) { mbar_init(s_tc.acc_full + i, 1); mbar_init(s_tc.acc_free + i, 4); s_tc.nfull[i] = 0; s_tc.nfree[i] = 0; }
      s_tc.tmem = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if ((int)blockIdx.x >= p.n_workers) return;
  {
  const int q0 = p.qbegin[blockIdx.x], q1 = p.qbegin[blockIdx.x + 1];
  if (threadIdx.x >= ETXB_CONSUMERS) {
    producer_loop<KV != 0, KV == 0 || KV == ETXB_VARIANT_MLA, KV != ETXB_VARIANT_BATCH, KV != ETXB_VARIANT_MLA, KV == 0 || KV == ETXB_VARIANT_MLA, TC>(p, sm, q0, q1);
    return;
  }
  TaskCtx* const ctx = (TaskCtx*)(smem_raw + ETXB_RING_BYTES + ETXB_GEN_BYTES + ETXB_SCR_FLOATS * 4 + 512);
  if constexpr (TC) {
    // tensor memory for the tensor-core tiles of a batched plan: allocated once per launch by warp 0 (one CTA per SM, so
    // the columns are always there), freed by the same warp after the last task on every path out of the loop below
    if (p.tc_on != 0u && threadIdx.x < 32) tc_alloc(&s_tc.tmem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  if (threadIdx.x == 0) { s_vars.q0 = q0; s_vars.q1 = q1; s_vars.cur = q0; *(volatile int*)&s_vars.done = q0; }
  if (threadIdx.x >= ETXB_CONSUMERS - 32 && q0 < q1) {
    fetch_ctx(p, ctx, q0, q0, -1);
    fetch_ctx(p, ctx, q0, q0 + 1 < q1 ? q0 + 1 : -1, -1);
    cp_async_wait_all();
    __syncwarp();
    fetch_ctx(p, ctx, q0, -1, q0);
    cp_async_wait_all();
  }
  }
  csync();
  // What the loop needs after a body it reads again from shared memory: held in registers across the calls (or the widest tiles) it
  // would go to the stack, and a stack access that follows an event's acquire is a trip to L2 (the acquire empties the
  // L1) -- the hand-off between two tiles of the batched step took 1 us more.
  volatile CtaVars* const vars = &s_vars;
  TaskCtx* const ctx = (TaskCtx*)(smem_raw + ETXB_RING_BYTES + ETXB_GEN_BYTES + ETXB_SCR_FLOATS * 4 + 512);
  uint32_t n = 0;                                                  // stages consumed so far (same count the producer keeps)
  for (int cur = vars->q0; cur < vars->q1; ++cur) {
    const TaskCtx* c = ctx + ((cur - vars->q0) & (ETXB_CTX_SLOTS - 1));
    if (tidx() == 0) {
      const int in_n = c->r.in_n & (ETXB_IN_ROUTED - 1);
      if (p.trace) p.trace[8 * (size_t)c->r.id] = globaltimer();
      // Everybody must leave the loop at the same task, or a barrier waits for warps that have left.  s_stop may be set at any
      // time (by the producer warp, by a warp whose wait in a body gives up), so only this thread looks at it, before the barrier.
      const bool stopped = *(volatile int*)&s_stop != 0;
      bool ok = true;                                              // wait_event polls the abort word itself
      for (int i = 0; ok && i < in_n; ++i) {
        int word, cnt;
        if (i < 4) { word = c->r.in_word[i]; cnt = c->r.in_cnt[i]; }
        else { word = p.inwords[c->r.in_off + i]; cnt = p.evcount[word]; }
        ok = wait_event(p, word, (int32_t)(p.epoch * (uint32_t)cnt), cur, s_deadline);
      }
      if (!ok) s_stop = 1;
      s_vars.halt = stopped || !ok;
      s_vars.tr = p.trace ? p.trace + 8 * (size_t)c->r.id : nullptr;
      s_vars.cur = cur;
      if (p.trace) p.trace[8 * (size_t)c->r.id + 1] = globaltimer();
    } else if (KV != ETXB_VARIANT_BATCH && tidx() == 32) {   // meanwhile: what the task multiplies and how the warps share it
      const int body = c->r.body;
      if (body >= 3 && body <= 5) {
        GemvGeom g;
        g.t = gemv_task(body, *(const etxb_gemv_args*)c->args, c->r.c0);
        gemv_geom(body, ((const etxb_gemv_args*)c->args)->mode, g);
        s_geo = g;
      }
    }
    else if (KV != ETXB_VARIANT_BATCH && !XCH && (tidx() >> 5) == 2) {   // .. and the routing of a down task, where it is known already
      const etxb_gemv_args& d = *(const etxb_gemv_args*)c->args;
      const int body = c->r.body;
      if (body == 5 && gemv_routed_early(body, d)) {
        const GemvTask t = gemv_task(body, d, c->r.c0);
        if (t.n > 0) gemv_route_words(d, *(const etxb_gemv_words*)(c->args + sizeof d), t, smem_view().scr);
      }
    } else if (tidx() >= ETXB_CONSUMERS - 32) {                    // the last consumer warp keeps the contexts coming (asynchronously)
      const int q1 = vars->q1;
      fetch_ctx(p, ctx, vars->q0, cur + 2 < q1 ? cur + 2 : -1, cur + 1 < q1 ? cur + 1 : -1);
    }
    csync();
    if (vars->halt) {                                              // the context copies of this task are waited for at its end otherwise
      if (tidx() >= ETXB_CONSUMERS - 32) cp_async_wait_all();
      break;
    }
    run_body<KV, XCH>(p, c, cur, smem_view(), n);
    cur = vars->cur;                                               // (before the barrier: thread 0 moves it on behind it)
    c = ctx + ((cur - vars->q0) & (ETXB_CTX_SLOTS - 1));
    if (tidx() >= ETXB_CONSUMERS - 32) cp_async_wait_all();
    csync();                                                       // every consumer thread's stores are issued, the next contexts landed
    // Sharded model: warp 1 publishes the bf16 rows this task wrote as flagged words (value | this step's flag) into the
    // grid's block of every rank's exchange region, its own included -- plain 4-byte stores, over NVLink for the peers.
    // Value and flag travel in one word, so nothing has to be ordered: no fence, no barrier, no remote counter; the
    // arrival below only tells this rank's consumers that the local phase is over, the folds then poll the flags.
    const uint32_t mirror = XCH && c->r.body != 12 ? c->r.mirror : 0u;   // 0 unless the grid is exchanged
    if (XCH && mirror != 0u && s_stop == 0 && (threadIdx.x >> 5) == 1) {   // (an abandoned body publishes nothing)
      const etxb_gemv_args& d = *(const etxb_gemv_args*)c->args;
      const int r0 = (c->r.body == 3 ? c->r.c0 : c->r.c0 % d.tpe) * d.rpt;
      const unsigned short* src = (const unsigned short*)d.out + r0;
      const uint32_t off = mirror & 0x3fffffu, len = mirror >> 22, fl = row_flag(p.epoch);
      for (uint32_t i = threadIdx.x & 31; i < len; i += 32) {
        const uint32_t v = (uint32_t)__ldcg(src + i) | fl;
        for (int q = 0; q < p.n_peers; ++q) st_flagged((uint32_t*)p.xpeer[q] + off + i, v);
        st_flagged((uint32_t*)p.xbase + off + i, v);
      }
    }
    if (tidx() == 0) {
      const int out_n = c->r.out_n & (ETXB_OUT_RELAXED - 1), id = c->r.id;
      const bool relaxed = KV != ETXB_VARIANT_BATCH && (c->r.out_n & ETXB_OUT_RELAXED) != 0;   // (the readers look at the words themselves; batched plans have none)
      if (s_stop == 0)                                             // (set when a stage wait gave up inside the body: no arrivals then)
#pragma unroll 1
        for (int i = 0; i < out_n; ++i) {                          // release: orders the CTA's stores (seen through the barrier) before the count
          const int word = i < 4 ? c->r.out_word[i] : p.outwords[c->r.out_off + i];
          if (relaxed) red_relaxed_add(p.events + (size_t)word * ETXB_EV_STRIDE, 1);
          else red_release_add(p.events + (size_t)word * ETXB_EV_STRIDE, 1);
        }
      vars->hold = 0;
      if constexpr (TC) vars->done = cur + 1;
      if (p.trace) { p.trace[8 * (size_t)id + 2] = globaltimer(); p.trace[8 * (size_t)id + 3] = blockIdx.x; }
      if (p.exec_count) atomicAdd(p.exec_count + id, 1);
    }
  }
  if constexpr (TC) {
    if (p.tc_on != 0u) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      csync();                                                     // nobody reads an accumulator any more
      if (threadIdx.x < 32) {
        // an abandoned step may have loaded stages that no MMA took, and MMAs that nobody waited for may still be reading theirs
        // and writing tensor memory: wait (bounded) for the copies, and for the commit behind each stage's last MMAs
        if (__any_sync(0xffffffffu, ld_relaxed(p.ctrl) != 0)) {
          for (int i = 0; i < ETXB_TC_MAXSTAGE; ++i) {
            const uint32_t lu = s_tc.lu[i], mu = s_tc.mu[i];
            if (lu != mu)
              for (int spin = 0; spin < 2000000 && !mbar_try_wait(s_tc.full + i, (lu - 1) & 1); ++spin) {}
            if (mu != 0)
              for (int spin = 0; spin < 2000000 && !mbar_try_wait(s_tc.empty + i, (mu - 1) & 1); ++spin) {}
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          __syncwarp();
        }
        tc_dealloc(s_tc.tmem);
      }
    }
  }
}

}  // namespace etxb
