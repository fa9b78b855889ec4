// Absorbed multi-head latent attention (DeepSeek-V2 family), one decode step, one task per head.
//
// The latent cache holds ONE row per position, shared by all heads: c (kv_lora values, RMS-normed) | k_pe (qk_rope
// values, rotated).  W_UK is folded into the query and W_UV into the output:
//   q_c[h] = q_nope[h] W_UK[h];   s[h][t] = scale (q_c[h] . c[t] + q_pe[h] . k_pe[t]);   p = softmax_t(s);
//   o_c[h] = sum_t p[t] c[t];     out[h] = W_UV[h] o_c[h]
// It stands where the reference's DeepSeek-V2-Lite graph runs the tasks q_absorb, attention (16 heads x 16 KV chunks),
// merge_uv (examples/dsv2lite/graph.py:98-209); the arithmetic follows the archived NumPy reference of that model,
// attention_absorbed (examples/dsv2lite/results/2026-10-14-k1/b_alld4r0l1kvs_stamps/fleet_src/host/reference_decode.py:207-253):
// bf16 q / kv_a rows, RMSNorm rounded twice on the latent, interleave-then-rotate rope with fp32 YaRN tables rounded to
// bf16 after the rotation, fp32 scores / softmax / sums, bf16 output.
//
// A task is (head h, partition of 128 positions): 16 heads x 9 partitions fill the SMs at a 1K context (one task per head
// over the whole context took 73 us per layer; this form takes a quarter of that).  Every task computes the new
// position's latent row from the kv_a row (576 values: cheaper than a phase of its own) and uses it from shared
// memory -- the task (head 0, last partition) also stores it into the cache --, folds W_UK into its head's query, and
// produces its partition's softmax statistics and weighted latent.  The partials travel as flagged (value, step) pairs
// like those of the grouped GQA tile (etxb_attn_gq.cuh); four finishing tasks per head, placed after the partition tasks
// in the grid, poll them, merge them in ascending partition order and apply a quarter of W_UV's rows each.
//
// W_UK's rows and the cached rows come through the weight ring (the producer warp copies them ahead of the task, as it does
// weights; all heads read the same cached rows, from L2): a partition task is 128 KB of W_UK and 147 KB of cache, and with loads
// into registers, eight in flight per thread, it spent its time waiting for them.
// A phase of 16 heads at 1043 positions: 19.5 us -> 16.5.  (Two positions at a time per warp: 72 bytes of spills, 18.)
#pragma once
#include "etxb_attn_gq.cuh"

namespace etxb {

#define ETXB_MLA_MAXCTX 8192   // longest context (64 partitions)
#define ETXB_MLA_PART 128      // positions per task
#define ETXB_MLA_FIN 4         // finishing tasks per head: each merges the head's partials and applies a quarter of W_UV's rows

struct etxb_mla_args {
  const void* qkv;             // 0   bf16 [NH * (DN + DR) + C + DR]: the q heads (nope | rope part each), then the kv_a row (c | k_pe)
  const void* kvln;            // 8   bf16 [C]: weight of the latent's RMSNorm
  const void* cos_sin;         // 16  fp32 [maxlen][2 * DR]: cos | sin rows of the rotary table (YaRN: already scaled)
  const void* wkvb;            // 24  bf16 [NH * (DN + DV)][C]: per head DN rows of W_UK, then DV rows of W_UV
  void* cache;                 // 32  bf16 [maxlen][C + DR]: the layer's latent cache
  const int64_t* positions;    // 40
  void* out;                   // 48  bf16 [NH * DV]
  int32_t NH, C, DN, DR, DV, maxlen;   // 56..79
  float scale, eps;            // 80..87
  void* tmp;                   // 88  (value, flag) pairs [NH][max_parts][C + 8]: weighted latent, then max logit and exp sum
  int32_t max_parts, tag;      // 96, 100: partitions the grid covers (tasks = (max_parts + 4) * NH: partitions, then finishing tasks); tag tells the layers that share tmp apart
  uint32_t* words;             // 104  hand-off as words: qkv names words, the outputs are also written as words here; null: bf16 vectors
  uint32_t grid[3], nblocks;   // 112..127
};

__device__ __forceinline__ void mla_out(const etxb_mla_args& d, int i, float v) {
  if (d.words != nullptr) st_word(d.words + i, bf_bits(v) | s_vars.flag);
  if (d.out != nullptr) ((__nv_bfloat16*)d.out)[i] = __float2bfloat16_rn(v);
}
// A finishing task of head h: waits (bounded) for the head's np partials, merges them -- weights exp(m_p - max m),
// partitions in ascending order -- and applies rows [f * DV / FIN, ..) of W_UV.  The finishing tasks come after the
// partition tasks in the grid, so whatever they wait for runs on another worker or ran before them on their own; the
// partition tasks never wait.  Four tasks per head instead of one cut the tail of the phase (merge + all of W_UV by the
// last partition's task: 15 us) to a third.
__device__ __forceinline__ void mla_finish(const etxb_mla_args& d, const Smem& sm, int h, int f, int np) {
  const int C = d.C, DN = d.DN, DV = d.DV, PW = C + 8;
  const int tid = tidx(), lane = tid & 31, warp = tid >> 5;
  const uint32_t fl = pair_flag(sm.serial(), d.tag << 16);
  float* oc = sm.xs;                                               // [C] merged, normalised latent
  const __nv_bfloat16* wuv = (const __nv_bfloat16*)d.wkvb + ((size_t)h * (DN + DV) + DN) * C;
  const int v_lo = f * ((DV + ETXB_MLA_FIN - 1) / ETXB_MLA_FIN), v_hi = min(DV, v_lo + (DV + ETXB_MLA_FIN - 1) / ETXB_MLA_FIN);
  // this task's rows of W_UV (the first 32 of them) travel to shared memory while it waits for the partials
  unsigned char* const wsm = (unsigned char*)sm.xs + 16384;        // [32][C] bf16
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int v = v_lo + warp + r * ETXB_CONSUMER_WARPS;
    if (v < v_hi)
      for (int j = 8 * lane; j < C; j += 256) cp_async16(wsm + ((warp + r * ETXB_CONSUMER_WARPS) * C + j) * 2, wuv + (size_t)v * C + j, true);
  }
  cp_async_commit();
  const uint2* ph = (const uint2*)d.tmp + (size_t)h * d.max_parts * PW;
  // A round: up to NF partitions' statistics (a lane each, every warp for itself) and this thread's values of them, requested together: behind the
  // slowest partition comes one trip to L2.  Between rounds (contexts of more than 1280 positions) the sums are rescaled to the larger maximum:
  // rms error of the weighted means at 4080 / 8150 positions 1.39e-7 / 1.72e-7, with all maxima waited for first 1.35e-7 / 1.70e-7, and 4 layers at 4080 in 440 us
  // instead of 428; the same scheme over the former sums of the warps 1.36e-7 / 1.69e-7 (and 6.3e-8 for the sum of the weights, so 4.1e-8).
  // (Statistics, then weights by one warp, then values, a barrier between any two, and bf16 vectors instead of words: 18.1 us a phase at 1043 positions, so 15.6.)
  constexpr int NF = 10;
  const uint2* vp = ph + min(tid, C - 1);
  float o = 0.f, L = 0.f, M = -INFINITY;
#pragma unroll 1
  for (int p0 = 0; p0 < np; p0 += NF) {
    const int pe = min(np - p0, NF);
    const uint2* sp = ph + (size_t)p0 * PW + C;
    uint2 first[NF];
    uint4 v;
    uint32_t spins = 0;
    for (;;) {
      v = ld_volatile16(sp + (size_t)min(lane, pe - 1) * PW);      // (maximum, flag, sum, flag)
#pragma unroll
      for (int u = 0; u < NF; ++u) first[u] = ld_pair(vp + (size_t)(p0 + min(u, pe - 1)) * PW);
      bool ok = v.y == fl && v.w == fl;
#pragma unroll
      for (int u = 0; u < NF; ++u) ok = ok && first[u].y == fl;
      if (ok || !poll_again(spins, sp, pe, PW, fl, sm)) break;
    }
    __syncwarp();
    const float m = lane < pe ? __uint_as_float(v.x) : -INFINITY;
    const float Mn = fmaxf(M, warp_max(m)), Mz = Mn == -INFINITY ? 0.f : Mn;
    const float f = expf(__fsub_rn(M, Mz)), wq = expf(__fsub_rn(m, Mz));       // (lanes past the round: 0)
    M = Mn;
    o = __fmul_rn(o, f);
    L = __fmaf_rn(L, f, lane < pe ? __fmul_rn(wq, __uint_as_float(v.z)) : 0.f);
#pragma unroll
    for (int u = 0; u < NF; ++u) {
      const float wu = __shfl_sync(0xffffffffu, wq, u);
      if (u < pe) o = __fmaf_rn(wu, __uint_as_float(first[u].x), o);
    }
  }
  L = warp_sum(L);
  if (tid < C) oc[tid] = __fdiv_rn(o, L);
  cp_async_wait0();
  csync();
  // ---- out[v] = W_UV[h][v] . o_c: a warp per output row, lanes over the columns
  for (int r = 0; r < 2; ++r) {
    const int v = v_lo + warp + r * ETXB_CONSUMER_WARPS;
    float acc = 0.f;
    if (v < v_hi)
#pragma unroll 2
      for (int j = 8 * lane; j < C; j += 256) {
        const uint4 x = *(const uint4*)(wsm + ((warp + r * ETXB_CONSUMER_WARPS) * C + j) * 2);
        const float wf[8] = {bf_lo(x.x), bf_hi(x.x), bf_lo(x.y), bf_hi(x.y), bf_lo(x.z), bf_hi(x.z), bf_lo(x.w), bf_hi(x.w)};
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = __fmaf_rn(wf[u], oc[j + u], acc);
      }
    acc = warp_sum(acc);
    if (lane == 0 && v < v_hi) mla_out(d, h * DV + v, acc);
  }
  for (int v0 = v_lo + 2 * ETXB_CONSUMER_WARPS; v0 < v_hi; v0 += ETXB_CONSUMER_WARPS) {   // (more than 32 rows per finishing task: DV > 128)
    const int v = v0 + warp;
    float acc = 0.f;
    if (v < v_hi)
      for (int j = 8 * lane; j < C; j += 256) {
        const uint4 x = __ldg((const uint4*)(wuv + (size_t)v * C + j));
        const float wf[8] = {bf_lo(x.x), bf_hi(x.x), bf_lo(x.y), bf_hi(x.y), bf_lo(x.z), bf_hi(x.z), bf_lo(x.w), bf_hi(x.w)};
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = __fmaf_rn(wf[u], oc[j + u], acc);
      }
    acc = warp_sum(acc);
    if (lane == 0 && v < v_hi) mla_out(d, h * DV + v, acc);
  }
  csync();
}

// What a partition task covers and streams, worked out alike by the consumer warps and by the producer warp: first the head's W_UK
// (DN rows of C), then the partition's cached rows (C + DR each), as many whole rows to a ring stage as fit.
struct MlaTask {
  int part, h, np;           // np: partitions of the context;  part >= max_parts: a finishing task
  int tbase, ncached;        // first position; rows that come from the cache (the new one, last of its partition, does not)
  bool owner, work;          // owner: the new position falls into the partition
  int ra, rb, na, nb;        // rows per stage and stages, of W_UK and of the cache
  long long pos;
};
__device__ __forceinline__ MlaTask mla_task(const etxb_mla_args& d, int blk, const etxb_stepv& S) {
  MlaTask t;
  t.part = udiv_small(blk, d.NH); t.h = blk - t.part * d.NH;
  t.pos = (const void*)d.positions == (const void*)S.positions ? (long long)S.pos : __ldcg((const long long*)d.positions);
  t.work = t.pos >= 0 && t.pos < d.maxlen && t.pos < ETXB_MLA_MAXCTX;
  const int seq = t.work ? (int)t.pos + 1 : 0;
  t.np = min((seq + ETXB_MLA_PART - 1) / ETXB_MLA_PART, d.max_parts);
  t.tbase = t.part * ETXB_MLA_PART;
  t.owner = t.work && (int)t.pos >= t.tbase && (int)t.pos < t.tbase + ETXB_MLA_PART;
  t.ncached = t.owner ? (int)t.pos - t.tbase : min(seq - t.tbase, ETXB_MLA_PART);
  t.ra = udiv_small(ETXB_STAGE_BYTES, d.C * 2); t.rb = udiv_small(ETXB_STAGE_BYTES, (d.C + d.DR) * 2);
  const bool streams = t.work && t.part < d.max_parts && t.part < t.np;
  t.na = streams ? udiv_small(d.DN + t.ra - 1, t.ra) : 0; t.nb = streams ? udiv_small(t.ncached + t.rb - 1, t.rb) : 0;
  return t;
}
__device__ __forceinline__ bool produce_mla(const etxb_mla_args& d, int blk, const etxb_stepv& S, uint32_t& n, const Smem& sm, int where) {
  if (blk >= (int)d.nblocks) return true;
  const MlaTask t = mla_task(d, blk, S);
  bool ok = true;
  if ((tidx() & 31) == 0) {
    const unsigned char* wa = (const unsigned char*)d.wkvb + (size_t)t.h * (d.DN + d.DV) * d.C * 2;
    const unsigned char* wb = (const unsigned char*)d.cache + (size_t)t.tbase * (d.C + d.DR) * 2;
    for (int s = 0; s < t.na + t.nb && ok; ++s) {
      const uint32_t st = n % ETXB_NSTAGE, par = (n / ETXB_NSTAGE) & 1;
      ok = mbar_wait(sm.empty + st, par ^ 1, sm, where);
      if (!ok) break;
      const bool A = s < t.na;
      const int r0 = A ? s * t.ra : (s - t.na) * t.rb, nr = A ? min(t.ra, d.DN - r0) : min(t.rb, t.ncached - r0), rbytes = A ? d.C * 2 : (d.C + d.DR) * 2;
      *((volatile uint32_t*)(sm.full + 2 * ETXB_NSTAGE) + st) = n;
      mbar_expect_tx(sm.full + st, (uint32_t)(nr * rbytes));
      bulk_g2s(sm.ring + (size_t)st * ETXB_STAGE_BYTES, (A ? wa : wb) + (size_t)r0 * rbytes, (uint32_t)(nr * rbytes), sm.full + st);
      ++n;
    }
  }
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  n = __shfl_sync(0xffffffffu, n, 0);
  return ok;
}

__device__ __forceinline__ void unpack16(const uint4 a, const uint4 b, float (&f)[16]) { unpack8(a, f); unpack8(b, f + 8); }

__device__ __forceinline__ void tile_mla_attn(const unsigned char* a, int blk, const Smem& sm, const etxb_stepv& S, uint32_t& n) {
  const etxb_mla_args& d = *(const etxb_mla_args*)a;
  if (blk >= (int)d.nblocks || blk >= d.NH * (d.max_parts + ETXB_MLA_FIN)) return;
  const MlaTask tk = mla_task(d, blk, S);
  if (!tk.work) return;
  if (tk.part >= d.max_parts) { mla_finish(d, sm, tk.h, tk.part - d.max_parts, tk.np); return; }
  if (tk.part >= tk.np) return;
  const int h = tk.h, C = d.C, DN = d.DN, DR = d.DR, QH = DN + DR, ROW = C + DR, PW = C + 8;
  const bool owner = tk.owner;
  const uint32_t fl = pair_flag(sm.serial(), d.tag << 16);
  const int tid = tidx(), lane = tid & 31, warp = tid >> 5, where = sm.cur();
  float* qf = sm.xs;            // [QH <= 256] this head's q row
  float* kvf = qf + 256;        // [ROW <= 640] the raw kv_a row
  float* cn = kvf + 640;        // [C <= 512] the new position's latent (bf16 values)
  float* kpn = cn + 512;        // [DR <= 64] its rotated k_pe (bf16 values)
  float* qpe = kpn + 64;        // [DR] this head's rotated q_pe (bf16 values)
  float* cs = qpe + 64;         // [2 DR] cos | sin of the position
  float* qc = cs + 128;         // [C] q_nope W_UK
  float* part = qc + 512;       // [16][512] the warps' partial sums (q_c, then o_c)
  float* red = part + 16 * 512; // [64]
  float* st = red + 64;         // [16][2] the warps' maximum and sum
  auto ldq = [&](int i) { return d.words != nullptr ? bf_lo(poll_word((const uint32_t*)d.qkv + i, s_vars.flag)) : ld_bf(d.qkv, i); };
  for (int i = tid; i < QH + 2 * DR + (owner ? ROW : 0); i += ETXB_CONSUMERS) {
    if (i < QH) qf[i] = ldq(h * QH + i);
    else if (i < QH + 2 * DR) cs[i - QH] = __ldg((const float*)d.cos_sin + (size_t)tk.pos * 2 * DR + (i - QH));
    else kvf[i - QH - 2 * DR] = ldq(d.NH * QH + (i - QH - 2 * DR));
  }
  csync();
  mark(sm, 0);
  // ---- q_c[j] = sum_i q_nope[i] W_UK[h][i][j]: a warp takes rows w, w + 16, .. (they lie in the ring), its lanes the columns
  //      8 lane .. and 256 + 8 lane ..; the warps' sums are added in warp order
  const bool c0 = 8 * lane < C, c1 = 256 + 8 * lane < C;
  const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
  float acc[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) acc[u] = 0.f;
  // (every warp walks every stage and gives back its sixteenth, so a stage's parity says which use it is)
  uint32_t k = n;
  n += (uint32_t)(tk.na + tk.nb);
  bool ok = true;
  int i0 = 0;
#pragma unroll 1
  for (int s = 0; s < tk.na && ok; ++s, i0 += tk.ra, ++k) {
    const uint32_t sx = k % ETXB_NSTAGE;
    ok = mbar_wait(sm.full + sx, (k / ETXB_NSTAGE) & 1, sm, where);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const int ie = min(DN, i0 + tk.ra);
    for (int i = i0 + ((warp - i0) & 15); i < ie; i += 16) {
      const uint4* row = (const uint4*)(sm.ring + (size_t)sx * ETXB_STAGE_BYTES + (size_t)(i - i0) * C * 2);
      float f[16];
      unpack16(c0 ? row[lane] : z4, c1 ? row[32 + lane] : z4, f);
      const float q = qf[i];
#pragma unroll
      for (int u = 0; u < 16; ++u) acc[u] = __fmaf_rn(q, f[u], acc[u]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_n(sm.empty + sx, ETXB_EMPTY_COUNT / ETXB_CONSUMER_WARPS);
  }
#pragma unroll
  for (int u = 0; u < 16; u += 4) *(float4*)(part + warp * 512 + (u >> 3) * 256 + 8 * lane + (u & 7)) = make_float4(acc[u], acc[u + 1], acc[u + 2], acc[u + 3]);
  // ---- meanwhile: the rotated q_pe, and, for the new position, its cache row: latent = rmsnorm(kv_a[:C]) (rounded twice), k_pe = rope(kv_a[C:])
  if (tid < 2 * DR && (owner || tid >= DR)) {
    // de-interleave (even elements first, then odd), then the half rotation: y cos + rot(y) sin
    const int i = tid < DR ? tid : tid - DR, half = DR >> 1;
    const float* x = tid < DR ? kvf + C : qf + DN;
    const float y = i < half ? x[2 * i] : x[2 * (i - half) + 1];
    const float rot = i < half ? -x[2 * i + 1] : x[2 * (i - half)];
    const float v = bfr(__fadd_rn(__fmul_rn(y, cs[i]), __fmul_rn(rot, cs[DR + i])));
    (tid < DR ? kpn : qpe)[i] = v;
  }
  if (owner) {
    const float ss = sumsq_numpy_order(kvf, C, red);               // (with barriers; owner is the same for all threads)
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)C), d.eps)));
    for (int i = tid; i < C; i += ETXB_CONSUMERS)
      cn[i] = bfr(__fmul_rn(bfr(__fmul_rn(kvf[i], r)), __bfloat162float(__ldg((const __nv_bfloat16*)d.kvln + i))));
  }
  csync();
  if (tid < C) {
    float v = part[tid];
#pragma unroll
    for (int w = 1; w < 16; ++w) v = __fadd_rn(v, part[w * 512 + tid]);
    qc[tid] = v;
  }
  if (h == 0 && owner) {
    __nv_bfloat16* row = (__nv_bfloat16*)d.cache + (size_t)tk.pos * ROW;
    for (int i = tid; i < ROW; i += ETXB_CONSUMERS) row[i] = __float2bfloat16_rn(i < C ? cn[i] : kpn[i - C]);
  }
  csync();
  mark(sm, 1);
  // ---- the positions, one at a time per warp (rows w, w + 16, ..; the new one after them): score, running maximum and sum, and the
  //      weighted latent in the lanes' registers -- a row is read once
  float q[16], qp[2];
#pragma unroll
  for (int u = 0; u < 8; ++u) { q[u] = c0 ? qc[8 * lane + u] : 0.f; q[8 + u] = c1 ? qc[256 + 8 * lane + u] : 0.f; }
  qp[0] = 2 * lane < DR ? qpe[2 * lane] : 0.f; qp[1] = 2 * lane < DR ? qpe[2 * lane + 1] : 0.f;
#pragma unroll
  for (int u = 0; u < 16; ++u) acc[u] = 0.f;
  float m = -INFINITY, l = 0.f;
  auto take = [&](const float (&f)[16], float p0, float p1) {
    float sa = 0.f, sb = 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u) { sa = __fmaf_rn(f[u], q[u], sa); sb = __fmaf_rn(f[8 + u], q[8 + u], sb); }
    sa = __fmaf_rn(p0, qp[0], sa); sb = __fmaf_rn(p1, qp[1], sb);
    const float sc = __fmul_rn(warp_sum(__fadd_rn(sa, sb)), d.scale);
    if (sc > m) {                                                  // (the same in every lane)
      const float g = expf(__fsub_rn(m, sc));
      m = sc; l = __fmul_rn(l, g);
#pragma unroll
      for (int u = 0; u < 16; ++u) acc[u] = __fmul_rn(acc[u], g);
    }
    const float e = expf(__fsub_rn(sc, m == -INFINITY ? 0.f : m)); // (a first row of score -inf: probability 0)
    l = __fadd_rn(l, e);
#pragma unroll
    for (int u = 0; u < 16; ++u) acc[u] = __fmaf_rn(e, f[u], acc[u]);
  };
  i0 = 0;
#pragma unroll 1
  for (int s = 0; s < tk.nb && ok; ++s, i0 += tk.rb, ++k) {
    const uint32_t sx = k % ETXB_NSTAGE;
    ok = mbar_wait(sm.full + sx, (k / ETXB_NSTAGE) & 1, sm, where);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const int ie = min(tk.ncached, i0 + tk.rb);
#pragma unroll 1
    for (int i = i0 + ((warp - i0) & 15); i < ie; i += 16) {
      const unsigned char* base = sm.ring + (size_t)sx * ETXB_STAGE_BYTES + (size_t)(i - i0) * ROW * 2;
      const uint4* row = (const uint4*)base;
      float f[16];
      unpack16(c0 ? row[lane] : z4, c1 ? row[32 + lane] : z4, f);
      const uint32_t pe = 2 * lane < DR ? *(const uint32_t*)(base + 2 * C + 4 * lane) : 0u;
      take(f, bf_lo(pe), bf_hi(pe));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_n(sm.empty + sx, ETXB_EMPTY_COUNT / ETXB_CONSUMER_WARPS);
  }
  if (owner && warp == (tk.ncached & 15)) {
    float f[16];
#pragma unroll
    for (int u = 0; u < 8; ++u) { f[u] = c0 ? cn[8 * lane + u] : 0.f; f[8 + u] = c1 ? cn[256 + 8 * lane + u] : 0.f; }
    take(f, 2 * lane < DR ? kpn[2 * lane] : 0.f, 2 * lane < DR ? kpn[2 * lane + 1] : 0.f);
  }
#pragma unroll
  for (int u = 0; u < 16; u += 4) *(float4*)(part + warp * 512 + (u >> 3) * 256 + 8 * lane + (u & 7)) = make_float4(acc[u], acc[u + 1], acc[u + 2], acc[u + 3]);
  if (lane == 0) { st[2 * warp] = m; st[2 * warp + 1] = l; }
  csync();
  mark(sm, 2);
  // ---- publish the partition's partial as flagged pairs: weighted latent [C], then max and sum (the warps' in warp order)
  uint2* pw = (uint2*)d.tmp + ((size_t)h * d.max_parts + tk.part) * PW;
  {
    // lane w works out warp w's factor (one exponential instead of sixteen), the sums take them by shuffle
    const float2 ml = *(const float2*)(st + 2 * (lane & 15));
    float M = ml.x;
#pragma unroll
    for (int x = 1; x < 16; x <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, x));
    const float g = expf(__fsub_rn(ml.x, M == -INFINITY ? 0.f : M));           // (a warp without a position: maximum -inf, weight 0)
    float L = __fmul_rn(g, ml.y), v = 0.f;
#pragma unroll
    for (int x = 1; x < 16; x <<= 1) L = __fadd_rn(L, __shfl_xor_sync(0xffffffffu, L, x));
#pragma unroll
    for (int w = 0; w < 16; ++w) v = __fmaf_rn(__shfl_sync(0xffffffffu, g, w), part[w * 512 + min(tid, C - 1)], v);
    if (tid < C) {
      st_pair(pw + tid, v, fl);
      if (tid == 0) { st_pair(pw + C, M, fl); st_pair(pw + C + 1, L, fl); }
    }
  }
  mark(sm, 3);
}

}  // namespace etxb
