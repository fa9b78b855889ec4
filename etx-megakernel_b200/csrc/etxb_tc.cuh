// Batched decode on the Blackwell tensor cores: tcgen05.mma with the tokens as the M side (A operand, shared memory,
// SWIZZLE_128B K-major), 64 .. 256 weight rows as the N side (B operand, loaded by TMA tensor copies --
// cp.async.bulk.tensor.2d with SWIZZLE_128B, one tensor map per weight tensor, boxes of 64 k x 64 rows, up to four per
// instruction) and fp32 accumulators in tensor memory, read back with tcgen05.ld for the epilogue.
//
// These tiles serve the same grids as the mma.sync tiles of etxb_batch.cuh (column-batched GEMV, expert-grouped gate+up
// and down: etx/ops/gemv.py:40-73, 176-289 and examples/vllm_llm/model.py:194-211 of the reference) and are what the
// batched step uses.  Sizing, measured on B200: one tcgen05.mma (cta_group::1, kind::f16) takes 156 clocks whatever its
// M, N (8 .. 256) or the number of accumulators in flight, so its cost is per instruction: with N = 256 weight rows per
// instruction (8 KB of weights per k16 step) the pipe moves 52 bytes of weights per clock and SM, twice what the HBM
// delivers (22.5), and all of a batch's tokens (up to 32 here) ride along for free -- mma.sync m16n8k16, the legacy
// path, managed about a sixth of that with 8 tokens per pass.
//
// A task = a few tiles of 64 .. 256 weight rows (neighbouring rows of a matrix, or up to 128 of an expert's gate rows and
// as many up rows) x all of K x up to 32 tokens.  Roles inside the CTA's consumer warps: one
// warp issues the TMA loads of the weight tiles (a lane per box of 64 rows), k-chunk by k-chunk, through a ring of 32 KB stages
// (as many as fit beside the tokens: 2 with 32 tokens of 2048 columns, 5 with up to 8), and starts before the tokens are there;
// the other threads stage the tokens' vectors into the swizzled layout, once per task; one thread issues the MMAs (four k16 steps per 64-wide chunk) and commits each stage back to the loader; when the last
// MMA of a tile has completed, four warps read its accumulators (one token per TMEM lane) and run the epilogue while
// the next tile's MMAs fill the other accumulator buffer.  The weight ring's memory and the general region form one area for
// tokens and stages here: the producer warp copies into the ring (units of attention, rows of the narrow tiles, streamed
// weights) only when every task before the one it copies for is over.  Every wait is bounded by the step's deadline; tensor memory is allocated once per
// launch by the kernel and freed on every exit path.
#pragma once
#include <cuda.h>

#include "etxb_gemv.cuh"

namespace etxb {

#define ETXB_TC_ROWS 128               // weight rows a block of the grids' geometry has; an instruction takes up to two (N <= 256)
#define ETXB_TC_BOXROWS 64             // weight rows per TMA box: the unit by which the expert grids are shared out
#define ETXB_TC_BOX 8192               // one box: 64 rows x 64 k x 2 bytes
#define ETXB_TC_STAGE (4 * ETXB_TC_BOX)   // one k-chunk of a tile: up to 256 rows
#define ETXB_TC_MAXSTAGE 6
#define ETXB_TC_TAIL 8192              // end of the area: the routing tables of the expert tiles
#define ETXB_TC_AREA (ETXB_RING_BYTES + ETXB_GEN_BYTES - 1024 - ETXB_TC_TAIL)   // the weight ring and the general region, 1024-byte aligned inside
#define ETXB_TC_XBYTES 131072          // at most this much of it holds tokens (32 tokens x 2048 columns); the rest are weight stages
#define ETXB_TC_MAXTOK 32              // tokens per job (M = 64 up to 8 tokens, 128 above)
#define ETXB_TC_COLS 512               // tensor-memory columns the kernel allocates: two accumulator buffers of 256

struct TcShared {                      // per-CTA state of the tensor-core tiles (static shared memory of the kernel)
  uint64_t full[ETXB_TC_MAXSTAGE], empty[ETXB_TC_MAXSTAGE];
  uint64_t acc_full[2], acc_free[2];   // accumulator buffer b: MMAs complete / epilogue done with it
  uint32_t lu[ETXB_TC_MAXSTAGE], mu[ETXB_TC_MAXSTAGE];   // how often the loader / the MMA issuer has used each stage (its barriers' phase)
  uint32_t nfull[2], nfree[2];         // completions of acc_full / acc_free so far
  uint32_t tmem;                       // base address of the allocation
  uint32_t pad;
};

__device__ __forceinline__ void tma_load_2d(void* dst, const void* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
// K-major SWIZZLE_128B shared-memory matrix descriptor: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
  d |= (uint64_t)1 << 16;                        // leading byte offset: unused for swizzled K-major layouts
  d |= (uint64_t)(1024 >> 4) << 32;              // stride between 8-row groups
  d |= (uint64_t)1 << 46;                        // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                        // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_alloc(uint32_t* slot) {        // one warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ETXB_TC_COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t base) {       // the same warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ETXB_TC_COLS) : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// 8 consecutive bf16 results of one token: one 16-byte store when all of them are inside [.., r1), else one by one
__device__ __forceinline__ void tc_store8(__nv_bfloat16* o, int r, int r1, const float (&y)[8]) {
  if (r + 8 <= r1 && (((uintptr_t)(o + r)) & 15) == 0) {
    uint4 pk;
    pk.x = pack_bf(y[0], y[1]); pk.y = pack_bf(y[2], y[3]); pk.z = pack_bf(y[4], y[5]); pk.w = pack_bf(y[6], y[7]);
    *(uint4*)(o + r) = pk;
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) if (r + u < r1) o[r + u] = __float2bfloat16_rn(y[u]);
  }
}

// The weight rows of a task, in tiles of tmax rows (a multiple of 64, up to 256) and one lower one at the end: rows y0 .. y0 + nrow;
// or, where a task takes two runs (an expert's gate rows and up rows, tmax <= 128), rows y1 .. y1 + nrow as well.
struct TcSeg {
  int y0, y1, nrow, tmax;                                          // nrow: a multiple of 64
  __device__ __forceinline__ int tiles() const { return (nrow + tmax - 1) / tmax; }
  __device__ __forceinline__ int height(int i) const { return min(tmax, nrow - i * tmax); }
};
// k-chunks of the tokens that fit at once / weight stages beside them
__device__ __forceinline__ int tc_window(int K, int ntok) { return min(K >> 6, ETXB_TC_XBYTES / (((ntok + 7) >> 3) * 1024)); }
__device__ __forceinline__ int tc_stages(int K, int ntok) {
  return min(ETXB_TC_MAXSTAGE, (ETXB_TC_AREA - tc_window(K, ntok) * ((ntok + 7) >> 3) * 1024) / ETXB_TC_STAGE);
}

// One task: for every tile i of the segment, h = height(i) rows, D_i[tok][j] = sum_k x_tok[k] * W[y0 + i tmax + j][k] for j < h, then
// epi(i, tok, j, v0, v1) for every tok < ntok and j = 0, 8, .. h - 8 with v0[u] = D_i[tok][j + u]; TWO: v1[u] = the same of the second run
// (one instruction multiplies both, N = 2 h).  K: a multiple of 64.  xsrc(n): the bf16 row of token n;
// map: the tensor map of the weight tensor (rows x all columns, box 64 x 64).  All consumer threads call; ends with a barrier.
// nx, nx_tok: the segment that the same caller runs next with the same map and K, and its tokens (0: none).
// pre: in, how many stages an earlier call has already filled for this segment; out, for the next one.
//
// The tokens are staged ONCE per task (the tiles of a task share them) whenever all of K fits the token area; the tiles
// then stream back to back through the stage ring, their accumulators alternating between two buffers of tensor
// memory, so that the epilogue of tile i overlaps the MMAs of tile i + 1.  When K does not fit (4096 columns x 32
// tokens) the tokens go in windows of K and a task handles its tiles one by one, accumulating across the windows.
// The weights depend on nothing a task waits for, so the loader fills the stage ring before the tokens are staged, and as its
// stages fall free at the end of a segment it fills them for the next one (the stages lie at the end of the area, the same
// place whatever the number of tokens): the step from one expert to the next, which a third of the workers take, does not
// drain the stream.
template <bool TWO, typename XSrc, typename Epi>
__device__ __forceinline__ void tc_task(const Smem& sm, TcShared& tc, const void* map, const TcSeg seg, const TcSeg nx, int nx_tok, int& pre, int K, int ntok,
                                        int where, XSrc xsrc, Epi epi) {
  const int tid = tidx(), warp = tid >> 5, lane = tid & 31;
  unsigned char* area = (unsigned char*)(((uintptr_t)sm.ring + 1023) & ~(uintptr_t)1023);
  const int M = ntok <= 8 ? 64 : 128, groups = (ntok + 7) >> 3, nchunk = K >> 6;
  // (an instruction reads M / 8 row groups of its k-chunk: the ones past the tokens' groups are the next chunks' rows or,
  // at the end, the first stage's -- whatever they hold only reaches accumulator rows that nobody reads)
  const int wc = tc_window(K, ntok), ntiles = seg.tiles();
  const int nwin = (nchunk + wc - 1) / wc;
  unsigned char* const ws = area + ETXB_TC_AREA - ETXB_TC_STAGE;   // stage s lies at ws - s * ETXB_TC_STAGE
  const int nst = tc_stages(K, ntok);
  const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(M >> 4) << 24);   // fp32 D, bf16 A / B, K-major; N goes in per tile
  const bool alive0 = *(volatile int*)sm.stop == 0;
  const uint32_t f0[2] = {tc.nfull[0], tc.nfull[1]}, r0[2] = {tc.nfree[0], tc.nfree[1]};     // (the previous task ended with a barrier)
  // one pass = one staging of tokens + the tiles that use it: all tiles x all of K, or (K in windows) one tile x one window
  const int npass = nwin == 1 ? 1 : ntiles * nwin;
  uint32_t tile_seq = 0;                                           // tiles finished before this pass (their buffer = tile_seq & 1)
  for (int pass = 0; pass < npass; ++pass) {
    const int i0 = nwin == 1 ? 0 : pass / nwin, i1 = nwin == 1 ? ntiles : i0 + 1, win = nwin == 1 ? 0 : pass - i0 * nwin;
    const int w0 = win * wc, nc = min(wc, nchunk - w0);
    const bool first_win = win == 0, last_win = win == nwin - 1;
    // loader: every tile of the pass, chunk by chunk (warp 1: a lane per box, their issue is what limits one thread)
    const bool loader = warp == 1 && alive0;
    auto load = [&](const TcSeg& g, int i, int c, int st) -> bool {
      const uint32_t uu = tc.lu[st];
      if (!__all_sync(0xffffffffu, mbar_wait(tc.empty + st, (uu & 1) ^ 1, sm, where))) return false;
      const int per = g.height(i) / ETXB_TC_BOXROWS, nb = TWO ? 2 * per : per;
      if (lane == 0) { tc.lu[st] = uu + 1; mbar_expect_tx(tc.full + st, (uint32_t)nb * ETXB_TC_BOX); }
      __syncwarp();
      if (lane < nb) {
        const bool second = TWO && lane >= per;
        tma_load_2d(ws - (size_t)st * ETXB_TC_STAGE + lane * ETXB_TC_BOX, map, (w0 + c) * 64,
                    (second ? g.y1 - per * ETXB_TC_BOXROWS : g.y0) + i * g.tmax + lane * ETXB_TC_BOXROWS, tc.full + st);
      }
      return true;
    };
    int li = i0, lc = 0, lst = 0;
    bool lok = true;
    auto load_next = [&]() {
      lok = load(seg, li, lc, lst);
      lst = lst + 1 == nst ? 0 : lst + 1;
      if (++lc == nc) { lc = 0; ++li; }
    };
    if (loader) {
      if (pass == 0)
        for (int q = 0; q < pre; ++q) {                            // (already on their way)
          lst = lst + 1 == nst ? 0 : lst + 1;
          if (++lc == nc) { lc = 0; ++li; }
        }
      for (int q = pass == 0 ? pre : 0; q < nst && li < i1 && lok; ++q) load_next();
    }
    // the tokens' slice [64 w0, 64 (w0 + nc)) -> swizzled rows: token n is row n % 8 of group n / 8 of its k-chunk
    if (!loader) {
    const int first = warp == 0 ? lane : tid - 32, step = alive0 ? ETXB_CONSUMERS - 32 : ETXB_CONSUMERS;   // (an abandoned step: whatever)
    for (int i = first; i < ntok * nc * 8; i += step) {
      const int n = i / (nc * 8), v = i - n * (nc * 8), c = v >> 3, j = v & 7, r = n & 7;
      const uint4 val = ld_act16((const __nv_bfloat16*)xsrc(n) + (size_t)(w0 * 64 + v * 8));
      *(uint4*)(area + (size_t)(c * groups + (n >> 3)) * 1024 + r * 128 + ((j ^ r) << 4)) = val;
    }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the tensor core's reads
    csync();
    if (sm.tr() != nullptr && tid == 0 && pass == 0) sm.tr()[4] = globaltimer();
    if (loader) {
      while (li < i1 && lok) load_next();
      const int nfill = nx_tok > 0 && nwin == 1 ? min(min(nst, tc_stages(K, nx_tok)), nx.tiles() * nchunk) : 0;
      for (int q = 0, i = 0, c = 0; q < nfill && lok; ++q) {
        lok = load(nx, i, c, q);
        if (++c == nchunk) { c = 0; ++i; }
      }
    } else if (warp == 2 && lane == 0 && alive0) {                 // MMA issuer
      bool ok = true;
      int st = 0;
      for (int i = i0; i < i1 && ok; ++i) {
        const uint32_t seq = tile_seq + (uint32_t)(i - i0), bsel = seq & 1;
        const uint32_t idesc = idesc0 | ((uint32_t)((TWO ? 2 : 1) * seg.height(i) >> 3) << 17);
        if (first_win) {                                           // a fresh accumulator buffer: the epilogue of the tile two back must be done with it
          const uint32_t nth = r0[bsel] + (seq >> 1);              // acc_free[bsel] completions expected before this use
          if (nth > 0) ok = mbar_wait(tc.acc_free + bsel, (nth - 1) & 1, sm, where);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t dcol = tc.tmem + bsel * 2 * ETXB_TC_ROWS;
        for (int c = 0; c < nc && ok; ++c) {
          const uint32_t uu = tc.mu[st];
          ok = mbar_wait(tc.full + st, uu & 1, sm, where);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t aaddr = smem_u32(area + (size_t)c * groups * 1024), baddr = smem_u32(ws - (size_t)st * ETXB_TC_STAGE);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma(dcol, tc_desc(aaddr + 32 * k), tc_desc(baddr + 32 * k), idesc, (w0 + c + k) > 0 ? 1u : 0u);
          tc_commit(tc.empty + st);                                // the stage is free once these MMAs have read it
          tc.mu[st] = uu + 1;
          st = st + 1 == nst ? 0 : st + 1;
        }
        if (ok) tc_commit(tc.acc_full + bsel);                     // the tile's MMAs (of this window) are complete
      }
      if (sm.tr() != nullptr && pass == npass - 1) sm.tr()[5] = globaltimer();
    }
    __syncwarp();                                                  // the role threads' warp-mates wait here, not in a spin beside them
    // epilogue: warps 0, 4, 8, 12 own TMEM lanes 0..31 (one token per lane), a quarter of a run's columns each.  Only
    // they wait for the accumulators: the issuer runs at most one tile ahead of the slowest of them (it needs their four
    // arrivals to reuse a buffer), so none of them can miss a phase; the other warps go on to the barrier below.
    if ((warp & 3) == 0) {
      for (int i = i0; i < i1; ++i) {
        const uint32_t seq = tile_seq + (uint32_t)(i - i0), bsel = seq & 1;
        // completions of acc_full[bsel] before this one: one per tile on that buffer (per window, when K goes in windows)
        const uint32_t done = f0[bsel] + (nwin == 1 ? (seq >> 1) : (seq >> 1) * (uint32_t)nwin + (uint32_t)win);
        bool alive = alive0;
        if (alive) alive = mbar_wait(tc.acc_full + bsel, done & 1, sm, where);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        alive = __all_sync(0xffffffffu, alive);
        if (!last_win) continue;
        if (alive) {
          const int h = seg.height(i), c0 = (warp >> 2) * (h >> 2), c1 = c0 + (h >> 2);
#pragma unroll 1
          for (int col = c0; col < c1; col += 8) {
            float v0[8], v1[8];
            tc_ld8(tc.tmem + bsel * 2 * ETXB_TC_ROWS + (uint32_t)col, v0);
            if (TWO) tc_ld8(tc.tmem + bsel * 2 * ETXB_TC_ROWS + (uint32_t)(h + col), v1);
            if (lane < ntok) epi(i, lane, col, v0, v1);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(tc.acc_free + bsel);            // four arrivals per tile: the buffer may be overwritten
      }
    }
    if (last_win) tile_seq += (uint32_t)(i1 - i0);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    csync();                                                       // the tokens may be restaged
  }
  pre = nx_tok > 0 && nwin == 1 ? min(min(nst, tc_stages(K, nx_tok)), nx.tiles() * nchunk) : 0;
  if (tid == 0) {
    const uint32_t nt = (uint32_t)ntiles;
    for (int b = 0; b < 2; ++b) {
      const uint32_t tiles_b = (nt + (b == 0 ? 1u : 0u)) >> 1;     // tiles that used buffer b
      tc.nfull[b] = f0[b] + tiles_b * (uint32_t)nwin;
      tc.nfree[b] = r0[b] + tiles_b;
    }
  }
  csync();
}

// ---------------------------------------------------------------------------------------------- batched dense GEMV
// out[b * sout + r] = bf16(W[r,:] . x[b] (+ bias[r])) for the nb columns b.  The GEMV block of gemv_nb; `ln` = the tensor
// map of W (rows M, box 64 x 64), put there by the host library when the plan is bound.
//
// tpe = 1: task blk covers rows [blk * rpt, ...) through the tcgen05 engine above.
__device__ __forceinline__ void tile_gemv_tc(const unsigned char* a, int blk, const Smem& sm, TcShared& tc, int where) {
  const etxb_gemv_args& d = *(const etxb_gemv_args*)a;
  if (blk >= (int)d.nblocks) return;
  const int r0 = blk * d.rpt, r1 = min(d.M, r0 + d.rpt);
  if (r0 >= r1) return;
  const __nv_bfloat16* bias = (d.mode & ETXB_MODE_BIAS) ? (const __nv_bfloat16*)d.wts : nullptr;
  __nv_bfloat16* out = (__nv_bfloat16*)d.out;
  const TcSeg seg = {r0, 0, (r1 - r0 + ETXB_TC_BOXROWS - 1) & -ETXB_TC_BOXROWS, 2 * ETXB_TC_ROWS};
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // what other tiles left in this memory: ordered before the copies
  csync();
  for (int b0 = 0; b0 < d.nb; b0 += ETXB_TC_MAXTOK) {
    const int nt = min(ETXB_TC_MAXTOK, d.nb - b0);
    int pre = 0;
    tc_task<false>(sm, tc, d.ln, seg, seg, 0, pre, d.K, nt, where,
            [&](int n) { return (const __nv_bfloat16*)d.x + (size_t)(b0 + n) * d.sx; },
            [&](int i, int tok, int j, const float (&v)[8], const float (&)[8]) {
              const int rr = r0 + 2 * i * ETXB_TC_ROWS + j;
              float y[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) y[u] = (bias && rr + u < r1) ? __fadd_rn(v[u], __bfloat162float(bias[rr + u])) : v[u];
              tc_store8(out + (size_t)(b0 + tok) * d.sout, rr, r1, y);
            });
  }
}

// ---------------------------------------------------------------------------------------------- narrow dense GEMV
// The same grid with tpe = S > 1: a matrix of a few thousand rows (qkv, o_proj, the router), S tasks per block of rpt rows.  Task blk
// takes the rows [(blk / S) * rpt + (blk % S) * R, + R), R = rpt / S rounded up to 16, over ALL of K: no partial sums leave the SM.
// With so few rows a tcgen05.mma (the same time for 16 rows as for 256) would take K / 16 times its 156 clocks, so these tiles run on
// mma.sync: sub-blocks of up to 128 rows as m16 tiles, the tokens as n8 tiles, K shared out between the warps.
//   weights  boxes of (rows of a sub-block) x 64 k through the ring, issued by the producer warp as soon as the task before is over
//            (they depend on no event): up to 144 KB lie in shared memory when the activations arrive
//   tokens   staged by all threads in rows of 64 k (pieces XOR-ed with the row, as the boxes: no bank conflicts for ldmatrix), all of K
//            at once where it fits 64 KB, else in two alternating windows of 32 KB with asynchronous copies
//   warps    16 = (16-row tiles of a sub-block) x (K groups): chunk c of 64 k belongs to K group c % KG; the groups' sums meet in
//            shared memory and are added in group order
// Against cutting K between the tasks (fp32 partial sums through L2, the last task to arrive adds them), us: qkv (5120 x 2048) 18.5 -> 12.5
// with 8 tokens and 23 -> 16.5 with 32, o_proj (2048 x 4096) 15 -> 9 and 20 -> 15, the router (128 x 2048) 9.5 -> 5 and 11 -> 8.5.  What is
// left is the staging of the tokens (2 .. 4) behind the event and the release.
struct NarrowGeo {
  int r0, r1, R, nsub;       // rows [r0, r1) of the task; rows of a sub-block (16, 32, 64, 128); sub-blocks
  int nmt, KG, cps, cnt;     // m16 tiles of a sub-block, K groups, 64-k chunks per ring stage, arrivals per warp and chunk
  int nchunk, ns;            // chunks of K; stages of one sub-block and pass
};
// rows of a task, a multiple of 16, and of its sub-blocks (the box of the grid's tensor map)
__host__ __device__ __forceinline__ int narrow_rows(int rpt, int S) { return ((rpt + S - 1) / S + 15) & -16; }
__host__ __device__ __forceinline__ int narrow_box(int rpt, int S) {
  const int per = narrow_rows(rpt, S);
  return per <= 16 ? 16 : per <= 32 ? 32 : per <= 64 ? 64 : 128;
}
__device__ __forceinline__ NarrowGeo narrow_geo(const etxb_gemv_args& d, int blk) {
  NarrowGeo g;
  const int S = d.tpe, rb = udiv_small(blk, S), ksl = blk - rb * S, per = narrow_rows(d.rpt, S);
  const int e = min(d.M, rb * d.rpt + d.rpt);
  g.r0 = min(e, rb * d.rpt + ksl * per); g.r1 = blk < (int)d.nblocks ? min(e, g.r0 + per) : g.r0;
  g.R = narrow_box(d.rpt, S);
  g.nmt = g.R >> 4; g.KG = ETXB_CONSUMER_WARPS / g.nmt;
  g.nsub = (g.r1 - g.r0 + g.R - 1) / g.R;
  g.cps = ETXB_STAGE_BYTES / (g.R * 128);                          // 12, 6, 3, 1
  g.cnt = ETXB_EMPTY_COUNT / (g.cps * g.nmt);                      // 4, 4, 4, 6
  g.nchunk = d.K >> 6;
  g.ns = udiv_small(g.nchunk + g.cps - 1, g.cps);
  return g;
}
__device__ __forceinline__ bool produce_narrow(const etxb_gemv_args& d, int blk, uint32_t& n, const Smem& sm, int where) {
  const NarrowGeo g = narrow_geo(d, blk);
  const int lane = tidx() & 31, npass = (d.nb + ETXB_TC_MAXTOK - 1) / ETXB_TC_MAXTOK;
  bool ok = true;
  for (int p = 0; p < npass && ok; ++p)
    for (int b = 0; b < g.nsub && ok; ++b)
      for (int s = 0; s < g.ns && ok; ++s) {
        const uint32_t st = n % ETXB_NSTAGE, par = (n / ETXB_NSTAGE) & 1;
        const int c0 = s * g.cps, nc = min(g.cps, g.nchunk - c0);
        int good = 1;
        if (lane == 0) {
          good = mbar_wait(sm.empty + st, par ^ 1, sm, where) ? 1 : 0;
          if (good) {
            *((volatile uint32_t*)(sm.full + 2 * ETXB_NSTAGE) + st) = n;  // (see wait_use)
            mbar_expect_tx(sm.full + st, (uint32_t)(nc * g.R * 128));
          }
        }
        ok = __shfl_sync(0xffffffffu, good, 0) != 0;
        if (ok && lane < nc)
          tma_load_2d(sm.ring + (size_t)st * ETXB_STAGE_BYTES + lane * g.R * 128, d.ln, (c0 + lane) * 64, g.r0 + b * g.R, sm.full + st);
        if (ok) ++n;
      }
  return ok;
}
__device__ __forceinline__ void tile_gemv_narrow(const unsigned char* a, int blk, const Smem& sm, uint32_t& n) {
  const etxb_gemv_args& d = *(const etxb_gemv_args*)a;
  const NarrowGeo g = narrow_geo(d, blk);
  if (g.nsub <= 0) return;
  const int tid = tidx(), warp = tid >> 5, lane = tid & 31, where = sm.cur();
  const int mt = warp & (g.nmt - 1), kg = warp / g.nmt, g8 = lane >> 2, t4 = lane & 3;
  const __nv_bfloat16* bias = (d.mode & ETXB_MODE_BIAS) ? (const __nv_bfloat16*)d.wts : nullptr;
  __nv_bfloat16* out = (__nv_bfloat16*)d.out;
  unsigned char* xs = (unsigned char*)sm.xs;                       // tokens; then the K groups' sums
  volatile const uint32_t* use = (volatile const uint32_t*)(sm.full + 2 * ETXB_NSTAGE);
  for (int b0 = 0; b0 < d.nb; b0 += ETXB_TC_MAXTOK) {
    const int nt = min(ETXB_TC_MAXTOK, d.nb - b0);
    const int n8 = nt <= 8 ? 1 : nt <= 16 ? 2 : 4, tp = 8 * n8;    // n8 tiles the products take; token rows in a chunk
    const int lw = n8 == 1 ? 5 : n8 == 2 ? 4 : 3;                  // log2 of the chunks of a 32 KB window
    const bool whole = g.nchunk <= 2 << lw;                        // all of K fits both windows
    const int nwin = whole ? 1 : (g.nchunk + (1 << lw) - 1) >> lw, wlen = whole ? g.nchunk : 1 << lw;
    auto stage = [&](int w) {                                      // window w of the tokens -> its buffer, asynchronously (tokens past nt: zero)
      const int c0 = w * wlen, nc = min(wlen, g.nchunk - c0);
      unsigned char* dst = xs + (whole ? 0 : (w & 1) * 32768);
      for (int i = tid; i < nc * 8 * tp; i += ETXB_CONSUMERS) {
        const int j = i & 7, q = i >> 3, c = n8 == 1 ? q >> 3 : n8 == 2 ? q >> 4 : q >> 5, r = q & (tp - 1);   // piece, then token, then chunk
        const bool live = r < nt;
        cp_async16(dst + (size_t)(c * tp + r) * 128 + ((j ^ (r & 7)) << 4),
                   (const __nv_bfloat16*)d.x + (size_t)(b0 + (live ? r : 0)) * d.sx + (c0 + c) * 64 + 8 * j, live);
      }
      cp_async_commit();
    };
    for (int b = 0; b < g.nsub; ++b) {
      const uint32_t n0 = n;
      n += (uint32_t)g.ns;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      stage(0);
      bool ok = true;
      for (int w = 0; w < nwin; ++w) {
        cp_async_wait0();
        csync();                                                   // everybody's copies of window w; everybody is done with window w - 1
        if (w + 1 < nwin) stage(w + 1);
        if (w == 0 && b == 0 && b0 == 0) mark(sm, 0);
        const int c0 = w * wlen, ce = min(g.nchunk, c0 + wlen);
        const uint32_t xw = smem_u32(xs + (whole ? 0 : (w & 1) * 32768));
        for (int c = c0 + ((kg - c0) & (g.KG - 1)); c < ce && ok; c += g.KG) {
          const int s = g.cps == 1 ? c : udiv_small(c, g.cps), ci = c - s * g.cps;
          const uint32_t k = n0 + (uint32_t)s, st = k % ETXB_NSTAGE;
          ok = wait_use(use + st, k, sm, where) && mbar_wait(sm.full + st, (k / ETXB_NSTAGE) & 1, sm, where);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const int br = lane & 7;
          const uint32_t aw = smem_u32(sm.ring) + st * ETXB_STAGE_BYTES + ci * g.R * 128 + (16 * mt + (lane & 15)) * 128;
          const uint32_t bw = xw + ((c - c0) * tp + br) * 128, ap = (aw >> 7) & 7;   // (the copies' swizzle goes by the address)
#pragma unroll
          for (int h = 0; h < 2; ++h) {                            // 32 k: two k16 steps
            uint32_t a0[4], a1[4], x[4][4];                        // (all fragments, then their products: the loads' latencies overlap)
            ldmatrix_x4(a0, aw + (((4 * h + (lane >> 4)) ^ ap) << 4));
            ldmatrix_x4(a1, aw + (((4 * h + 2 + (lane >> 4)) ^ ap) << 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) if (i < n8) ldmatrix_x4(x[i], bw + i * 1024 + (((4 * h + (lane >> 3)) ^ br) << 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) if (i < n8) mma16816(acc[i], a0, x[i][0], x[i][1]);
#pragma unroll
            for (int i = 0; i < 4; ++i) if (i < n8) mma16816(acc[i], a1, x[i][2], x[i][3]);
          }
          __syncwarp();
          // (the last chunk of a stage that is not full gives back the missing ones' arrivals too)
          const int in_stage = min(g.cps, g.nchunk - s * g.cps);
          if (lane == 0) mbar_arrive_n(sm.empty + st, (uint32_t)(g.cnt * (ci == in_stage - 1 ? g.cps - ci : 1)));
        }
      }
      csync();                                                     // (the sums lie where the tokens were)
      if (b == 0 && b0 == 0) mark(sm, 1);
      // the K groups' sums: [group][token][R + 4] floats
      float* red = (float*)xs;
      const int ld = g.R + 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < n8) {
          float* q = red + (size_t)(kg * tp + 8 * i + 2 * t4) * ld + 16 * mt + g8;
          q[0] = acc[i][0]; q[ld] = acc[i][1]; q[8] = acc[i][2]; q[ld + 8] = acc[i][3];
        }
      csync();
      const int rows = min(g.R, g.r1 - g.r0 - b * g.R);
      for (int i = tid; i < nt * g.R; i += ETXB_CONSUMERS) {
        const int tok = i >> (31 - __clz(g.R)), r = i & (g.R - 1), row = g.r0 + b * g.R + r;
        float v = red[tok * ld + r];
        for (int q = 1; q < g.KG; ++q) v = __fadd_rn(v, red[(size_t)(q * tp + tok) * ld + r]);
        if (r < rows) out[(size_t)(b0 + tok) * d.sout + row] = __float2bfloat16_rn(bias ? __fadd_rn(v, __bfloat162float(bias[row])) : v);
      }
      if (b + 1 < g.nsub || b0 + ETXB_TC_MAXTOK < d.nb) csync();   // the tokens of the next sub-block or pass may come
    }
  }
  mark(sm, 2);
}

// ---------------------------------------------------------------------------------------------- expert-grouped gate+up / down
// The expert phases of a batched step, scheduled by SHARE: the grid has one task per worker, and task blk of S takes
// tiles [blk * total / S, (blk + 1) * total / S) of the step's active experts (total = active experts x tiles per expert,
// experts in ascending id, an expert's tiles in row order) -- every worker streams the same number of weight rows (+-1
// tile) however the routing falls, where a grid of (expert, row chunk) tasks leaves the workers of unselected experts idle
// and gives others three chunks.  Every task derives the routing tables itself from the step's top-k ids (nb x R int32,
// one L2 read): per-expert counts, the active list, and per expert the (column << 8 | slot) pairs that selected it in
// ascending (column, slot) order.
//
// The GEMV block, read this way: W / estride / M / K / E as in the one-token MoE tiles (gate+up: M gate rows then M up
// rows per expert; down: M rows), ids = the routing ids [nb][R], nb columns, R = top-k, nblocks = S;
// gate+up: x[b * sx ..] the columns' normed vectors, out = act [nb][R][M], resid_out = optional int32 counter that
// share 0 increases by the number of active experts; down: x = act [nb][R][K], wts [nb][R] routing weights, out = y [nb][R][M].
// `ln` = the tensor map of the expert tensor seen as one [E * rows][K] matrix.
struct TcRoute {
  int32_t* sids;     // [nb * R] expert ids of the step
  int32_t* scnt;     // [E] entries per expert
  int32_t* ent;      // [<= nb] entries of the current expert
  float* wt;         // [<= nb] their routing weights (down)
  uint16_t* alist;   // [nact] active experts, ascending
  int32_t* nact;
};
__device__ __forceinline__ TcRoute tc_route_tables(const Smem& sm) {
  unsigned char* tail = (unsigned char*)(((uintptr_t)sm.ring + 1023) & ~(uintptr_t)1023) + ETXB_TC_AREA;
  TcRoute r;
  r.sids = (int32_t*)tail; r.scnt = r.sids + 1024; r.ent = r.scnt + 256; r.wt = (float*)(r.ent + 64); r.alist = (uint16_t*)(r.wt + 64);
  r.nact = (int32_t*)(r.alist + 256);
  return r;
}
// counts and the active list (all consumer threads; ends with a barrier)
__device__ __forceinline__ void tc_route_build(const etxb_gemv_args& d, const TcRoute& rt) {
  const int tid = tidx(), n = d.nb * d.R;
  for (int i = tid; i < n; i += ETXB_CONSUMERS) { const int e = __ldcg(d.ids + i); rt.sids[i] = (unsigned)e < (unsigned)d.E ? e : 0; }
  for (int e = tid; e < d.E; e += ETXB_CONSUMERS) rt.scnt[e] = 0;
  csync();
  for (int i = tid; i < n; i += ETXB_CONSUMERS) atomicAdd(rt.scnt + rt.sids[i], 1);
  csync();
  if (tid < 32) {
    int na = 0;
    for (int e0 = 0; e0 < d.E; e0 += 32) {
      const bool on = e0 + tid < d.E && rt.scnt[e0 + tid] > 0;
      const uint32_t m = __ballot_sync(0xffffffffu, on);
      if (on) rt.alist[na + __popc(m & ((1u << tid) - 1u))] = (uint16_t)(e0 + tid);
      na += __popc(m);
    }
    if (tid == 0) *rt.nact = na;
  }
  csync();
}
// the entries of expert e, in (column, slot) order (warp 0; the caller syncs)
__device__ __forceinline__ void tc_route_entries(const etxb_gemv_args& d, const TcRoute& rt, int e, const float* wts) {
  const int tid = tidx(), n = d.nb * d.R;
  if (tid >= 32) return;
  int cnt = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + tid;
    const bool hit = i < n && rt.sids[i] == e;
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    const int at = cnt + __popc(m & ((1u << tid) - 1u));
    if (hit && at < 64) {
      rt.ent[at] = ((i / d.R) << 8) | (i % d.R);
      if (wts != nullptr) rt.wt[at] = __ldcg(wts + i);
    }
    cnt += __popc(m);
  }
}

template <bool UP>
__device__ __forceinline__ void tile_moe_tc(const unsigned char* a, int blk, const Smem& sm, TcShared& tc, int where) {
  const etxb_gemv_args& d = *(const etxb_gemv_args*)a;
  if (blk >= (int)d.nblocks) return;
  const TcRoute rt = tc_route_tables(sm);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // what other tiles left in this memory: ordered before the copies
  tc_route_build(d, rt);                                           // (with barriers)
  const int nact = *rt.nact;
  // Shares are cut in units of 64 rows of M (gate+up: with their up rows); a task's run of units of one expert goes through in
  // tiles as high as an instruction takes and one lower one at its end.  (In whole tiles the step of 8 sequences had 348 for
  // 148 workers: a third of them took three, the rest two, and the phase lasted 74 us where its mean share took 58.)
  constexpr int TROWS = ETXB_TC_BOXROWS, TMAX = UP ? ETXB_TC_ROWS : 2 * ETXB_TC_ROWS;
  const int T = (d.M + TROWS - 1) / TROWS;
  const uint32_t total = (uint32_t)nact * (uint32_t)T;
  const bool small = total < (1u << 20) && d.nblocks < (1u << 12);   // (a 64-bit division is a microsecond)
  int t = small ? (int)(total * (uint32_t)blk / d.nblocks) : (int)((unsigned long long)total * blk / d.nblocks);
  const int hi = small ? (int)(total * (uint32_t)(blk + 1) / d.nblocks) : (int)((unsigned long long)total * (blk + 1) / d.nblocks);
  if (UP && blk == 0 && tidx() == 0 && d.resid_out != nullptr) atomicAdd((int32_t*)d.resid_out, nact);
  const int erows = (int)(d.estride / d.K);
  auto segment = [&](int at, int& t1) {                             // the run of units of one expert that begins at `at`
    const int ai = at / T, t0 = at - ai * T;
    t1 = min(T, t0 + (hi - at));
    const int erow = rt.alist[ai] * erows;                          // first row of the expert in the [E * rows][K] view
    return TcSeg{erow + t0 * TROWS, erow + d.M + t0 * TROWS, (t1 - t0) * TROWS, TMAX};   // (up rows follow the M gate rows)
  };
  auto entries = [&](int at) { return min(min(rt.scnt[rt.alist[at / T]], d.nb), 64); };
  int pre = 0;
  while (t < hi) {
    const int ai = t / T, t0 = t - ai * T;
    int t1, nt1 = 0;
    const TcSeg seg = segment(t, t1);
    const int cnt = entries(t), tn = t + t1 - t0;
    const TcSeg nseg = tn < hi ? segment(tn, nt1) : seg;
    const int ntn = tn < hi ? min(ETXB_TC_MAXTOK, entries(tn)) : 0;
    tc_route_entries(d, rt, rt.alist[ai], UP ? nullptr : d.wts);
    csync();
    const int r0 = t0 * TROWS, r1 = min(d.M, t1 * TROWS);
    for (int p0 = 0; p0 < cnt; p0 += ETXB_TC_MAXTOK) {
      const int nt = min(ETXB_TC_MAXTOK, cnt - p0), nxt = p0 + nt < cnt ? 0 : ntn;
      const int32_t* ent = rt.ent + p0;
      if constexpr (UP) {
        tc_task<true>(sm, tc, d.ln, seg, nseg, nxt, pre, d.K, nt, where,
                [&](int n) { return (const __nv_bfloat16*)d.x + (size_t)(ent[n] >> 8) * d.sx; },
                [&](int i, int tok, int j, const float (&g)[8], const float (&up)[8]) {
                  const int r = r0 + i * TMAX + j, en = ent[tok];
                  float y[8];
#pragma unroll
                  for (int u = 0; u < 8; ++u) y[u] = __fmul_rn(bfr(silu_f(bfr(g[u]))), bfr(up[u]));
                  tc_store8((__nv_bfloat16*)d.out + ((size_t)(en >> 8) * d.R + (en & 0xff)) * d.M, r, r1, y);
                });
      } else {
        const float* wt = rt.wt + p0;
        tc_task<false>(sm, tc, d.ln, seg, nseg, nxt, pre, d.K, nt, where,
                [&](int n) { return (const __nv_bfloat16*)d.x + ((size_t)(ent[n] >> 8) * d.R + (ent[n] & 0xff)) * d.K; },
                [&](int i, int tok, int j, const float (&v)[8], const float (&)[8]) {
                  const int r = r0 + i * TMAX + j, en = ent[tok];
                  float y[8];
#pragma unroll
                  for (int u = 0; u < 8; ++u) { const float q = bfr(v[u]); y[u] = d.wts ? bfr(__fmul_rn(q, wt[tok])) : q; }
                  tc_store8((__nv_bfloat16*)d.out + ((size_t)(en >> 8) * d.R + (en & 0xff)) * d.M, r, r1, y);
                });
      }
    }
    t = tn;
  }
}
__device__ __forceinline__ void tile_moe_up_tc(const unsigned char* a, int blk, const Smem& sm, TcShared& tc, int where) { tile_moe_tc<true>(a, blk, sm, tc, where); }
__device__ __forceinline__ void tile_moe_down_tc(const unsigned char* a, int blk, const Smem& sm, TcShared& tc, int where) { tile_moe_tc<false>(a, blk, sm, tc, where); }

}  // namespace etxb
