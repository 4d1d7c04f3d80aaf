// Causal grouped-query attention of prompt steps over the paged bfloat16 cache on the
// fifth-generation tensor cores: head size 64, full (unwindowed) attention.
//
// A block owns 128 query rows of one (sequence, KV head): rows are (token, head-in-group) pairs,
// GP heads of the group packed beside each other (the reference orders the queries of a KV head the
// same way, src/model.zig:1352-1366), and walks the keys in tiles of 64 that lie inside one cache
// page.  Roles:
//   * warp 4 (one lane) is the producer: one 3-D TMA load brings the 128 x 64 query tile, then per
//     key tile two 2-D TMA loads bring K and V ([64 keys, 64] each, 128-byte swizzle) into a ring of
//     four stages, so that the loads run three tiles ahead of the MMAs;
//   * warp 5 (one lane) issues tcgen05.mma: S = Q K^T (M 128, N 64 keys, four k steps; K is the
//     K-major B operand) into one of two score buffers in tensor memory, and O += P V (N 64 columns,
//     four k steps over the 64 keys; P is the A operand and lies in tensor memory, V as it lies in the
//     cache is the MN-major B operand);
//   * warps 0..3 are the softmax, a thread per row: it reads its 64 scores with tcgen05.ld, applies the
//     causal mask, keeps the running maximum and the sum of the online softmax (src/attention.zig:478-517, no
//     tile skipped) and writes its row of P as bfloat16 into one of two buffers in tensor memory, each with barriers of
//     its own (see NP below).  Only where a maximum moved does a warp wait for P V of the tile before and rescale O, and it does
//     so behind the exponentials.  (A reference that stays until a score passes it by 2^8 is faster still, 209 us against
//     230, but then the largest P is no longer 1 and is rounded: errors against 64 bits 1.77e-3 -> 2.16e-3
//     with scores of a wide spread.)
// Q K^T of tile t + 1 is issued before the MMA warp waits for P of tile t, so it runs while the softmax
// warps work on tile t, and P V of tile t runs while they work on tile t + 1.  One block needs 256
// columns of tensor memory (two score buffers, O, two of P) and 82 KB of shared memory: two blocks share an SM.
// What bounds it: the special-function unit (64 x 128 exponentials are 512 cycles of an SM, the MMAs of the
// tile 256), whose pipe is busy for 58 % of the cycles (8,192 tokens; the clock is 1.69 GHz under this load); the rest is a
// warp's chain from scores to P with two warps per scheduler.
// Measured on a B200, microseconds a layer with flushed caches, against two threads per row that exchanged their maxima
// every tile, P in shared memory and the blocks head after head: 8,192 tokens, 16 heads on 8 332 -> 240 (573 TFLOP/s),
// 32 heads on 8 554 -> 453; 2,048 tokens 46 -> 38 and 70 -> 51; with a distance table 461 -> 330 (8,192 tokens, 16 heads).  With O
// rescaled before the exponentials it took 261 where this form took 230; with one score buffer that P replaces (four blocks an
// SM, the scores read twice for the registers) a fifth longer.  Scores stay unscaled in registers; the
// scale is folded into the exponent (2^((s - m) * scale * log2 e), ex2.approx), tiles below the
// diagonal skip the mask.
//
// Options (the EXT form of the kernel): a table of numbers per (head, distance) added to the scaled scores, a mask in
// stretches of positions (a query sees its own stretch only; the walk starts at the tile of the first query's stretch), and a
// gate per (token, head) on the output.  The rows and keys of a tile span 128/GP tokens by 64 keys, so a tile needs 128/GP + 63
// consecutive distances of each of its GP heads: the producer brings that slice of the table with the tile's keys and values
// (one bulk copy per head, rounded out to 16 bytes, into the same stage and on the same barrier), in rows of dist_ld(GP)
// floats, which puts a warp's 32 lookups in 32 banks.  The table lies padded in memory (DIST_FRONT entries ahead of distance
// 0, which only masked keys meet, and DIST_BACK copies of the last number behind it), so no lookup clamps.  (A first form, in
// which every warp fetched its own slice with ordinary loads ahead of the scores, took 77 us where this kernel without a table
// takes 45.)
//
// Rows of V beyond the last visible key are set to zero in shared memory before P V (their
// probabilities are zero, but zero times a stale NaN would not be); scores of masked keys are
// replaced, never used.  Every wait on an mbarrier is bounded: after about two seconds the block
// records a code in *status, stops issuing work, frees its tensor memory and returns.
#include "tcgen05.cuh"
#include <math.h>
#include <stdint.h>

namespace {

using namespace tc5;

constexpr int HD = 64;            // head size
constexpr int ROWS = 128;         // query rows per block = accumulator lanes
constexpr int TK = 64;            // keys per tile
constexpr int SM_THREADS = ROWS;  // four softmax warps: a thread per row
constexpr int THREADS = SM_THREADS + 64;   // then the producer warp and the MMA warp
constexpr int PRODUCER_WARP = SM_THREADS / 32, MMA_WARP = PRODUCER_WARP + 1;
constexpr int Q_BYTES = ROWS * HD * 2, KV_BYTES = TK * HD * 2;
constexpr int NSTG = 4;           // K/V tiles in shared memory: the loads run three tiles ahead of the MMAs
constexpr size_t SMEM_BYTES = Q_BYTES + 2 * NSTG * KV_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
// EXT: a stage's slice of the distance table
constexpr int DIST_FRONT = 192, DIST_BACK = 256;
__host__ __device__ constexpr int dist_len_of(int gp) { return (ROWS / gp + TK - 1 + 3 + 3) / 4 * 4; }       // floats copied per head
__host__ __device__ constexpr int dist_ld(int gp) {      // floats between heads: at least that, and 32/gp modulo 32 for gp 2, 4, 8
  return gp == 1 ? dist_len_of(1) : gp == 2 ? 144 : gp == 4 ? 104 : 100;
}
static_assert(dist_ld(2) >= dist_len_of(2) && dist_ld(4) >= dist_len_of(4) && dist_ld(8) >= dist_len_of(8), "slices fit their rows");
constexpr size_t DIST_BYTES = (size_t)NSTG * 8 * dist_ld(8) * sizeof(float);      // slices of all stages with the most heads
static_assert(dist_ld(1) <= 8 * dist_ld(8) && 2 * dist_ld(2) <= 8 * dist_ld(8) && 4 * dist_ld(4) <= 8 * dist_ld(8), "8 heads need the most");
constexpr unsigned TMEM_COLS = 256;   // two blocks fit an SM
constexpr unsigned T_S = 0, T_O = 128, T_P = 192;   // score buffers at columns 0 and 64, O, P at 192 and 224
// Buffers of P, and for each a barrier "P is written" and a barrier "P V is complete".  A warp whose maxima stay does not wait for
// P V of the tile before, so it may be a tile ahead of another warp; the scores of tile t + 1 are there before P of tile t is
// complete.  So the arrivals for t and t + 1 must not meet on one barrier: those of the fast warp for t + 1 would stand for
// the slow warp's for t, and P V of t would run on rows of P and of O that the slow warp is still at.  With a barrier per buffer they
// cannot: a warp that arrives for t + 2 has waited for P V of t or of t + 1, and neither begins before every warp arrived for t.
constexpr int NP = 2;

struct Params {
  bf16* out;
  const int* tile_seq;
  const int* tile_q0;
  const int* cu_q;
  const int* seq_start;
  const int* seq_slot;
  const int* page_table;
  int* status;
  int pt_stride, H, Hkv, page_size, gp;   // gp: heads of a KV group packed into one block
  float scale;
  // cross mode (both or neither): blockIdx.z names the key/value head whose VALUES a block reads in place of its
  // own key/value head's, and the block's normalised rows go, as float32, to part_o [tokens * H * Hkv, HD] with
  // (maximum 0, denominator 1) in part_ml [tokens * H * Hkv, 2], rows ordered (token, head, value head): what
  // the kernel that mixes the heads' weights after the softmax reads.
  float* part_o;
  float* part_ml;
  // EXT form: dist float32 (null: none), rows of dist_row floats, one per head: entry DIST_FRONT + n of row h is added to the
  // scaled score of a query and a key n positions before it; the last DIST_BACK entries of a row are equal and stand for every
  // larger distance too; mask_chunk > 0: a query sees only keys of its own stretch of mask_chunk positions, counted from position 0; gate
  // (null: none): logits, a token's rows ld_gate apart, head h's output is multiplied by sigmoid(gate[t, h]).
  const float* dist;
  int dist_row, mask_chunk;
  const bf16* gate;
  int ld_gate;
};

// 2^x on the special-function unit (relative error about 2^-22; 2^-inf = 0).
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to this block's shared memory, counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar))
               : "memory");
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&t);
}

// two float32 operations in one instruction; the results are those of the single ones
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
      "fma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

template <bool EXT>
__global__ void __launch_bounds__(THREADS, 2)
    attn_prefill_tc5_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, const Params p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* q_sm = base;
  unsigned char* kv_sm = base + Q_BYTES;          // stage s: K at kv_sm + 2 s KV_BYTES, V behind it
  auto k_sm = [&](int s) { return kv_sm + 2 * s * KV_BYTES; };
  auto v_sm = [&](int s) { return kv_sm + (2 * s + 1) * KV_BYTES; };
  unsigned char* bar_sm = base + Q_BYTES + 2 * NSTG * KV_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(bar_sm);
  unsigned long long* q_full = bars;            // 1
  unsigned long long* kv_full = bars + 1;               // [NSTG]
  unsigned long long* kv_empty = bars + 1 + NSTG;       // [NSTG]
  unsigned long long* s_full = bars + 1 + 2 * NSTG;     // [2]: one per score buffer
  unsigned long long* p_ready = bars + 3 + 2 * NSTG;    // [NP]: one per P buffer, an arrival per softmax thread
  unsigned long long* pv_done = p_ready + NP;           // [NP]: one per P buffer
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(pv_done + NP);
  static_assert((3 + 2 * NP + 2 * NSTG) * 8 + 16 <= 256, "the barriers fit their 256 bytes");
  volatile int* aborted = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* dist_sm = reinterpret_cast<float*>(bar_sm + 256);     // EXT: [NSTG][GP][dist_ld(GP)]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int GP = p.gp, G = p.H / p.Hkv, chunks = G / GP;
  const int BQ = ROWS / GP;                   // tokens per block
  const int packs = p.Hkv * chunks, pack = blockIdx.x % packs, kvh = pack / chunks, chunk = pack % chunks;
  const bool cross = p.part_o != nullptr;
  const int vh = cross ? blockIdx.z : kvh;
  // Tiles are taken from the last (a sequence's late tokens see the most keys) to the first, all heads of a tile before the
  // next, so that what is left for the end is short.  Head after head, the last head's longest tiles began when 7 of 8 of the
  // work was done, and SMs were busy for 80 % of the time (16 heads on 8, 8,192 tokens).
  const int tile = (gridDim.x - 1 - blockIdx.x) / packs;
  const int b = p.tile_seq[tile], q0 = p.tile_q0[tile];
  const int t_base = p.cu_q[b], Tq = p.cu_q[b + 1] - t_base;
  const int start = p.seq_start[b];
  const int last_tq = min(q0 + BQ, Tq) - 1;
  const int k_end = start + last_tq + 1;      // keys [k_begin, k_end)
  const int k_begin = EXT && p.mask_chunk > 0 ? (start + q0) / p.mask_chunk * p.mask_chunk / TK * TK : 0;
  const int n_tiles = (k_end - k_begin + TK - 1) / TK;
  // EXT: where in a row of the table the slice of the tile at key kb begins (its first entry is the distance of the block's first
  // token from the tile's last key); behind the last distinct number every place is as good as any other
  auto dist_at = [&](int kb) { return min(start + q0 - kb - (TK - 1) + DIST_FRONT, p.dist_row - dist_len_of(GP)); };

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < NSTG; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    for (int i = 0; i < NP; ++i) {
      mbar_init(&p_ready[i], SM_THREADS);
      mbar_init(&pv_done[i], 1);
    }
    *aborted = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == MMA_WARP) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = *tmem_slot;
  const unsigned tmem_o = tmem_base + T_O;
  // Barriers and tensor memory are set up while the kernel before this one ends; q and the cache
  // are its results.  (The batch's index arrays read above were uploaded before the step began.)
  zk_let_next_start();
  zk_wait_prior();

  if (warp == PRODUCER_WARP && lane == 0) {
    // ---------------------------------------------------------------- producer
    const int* pt = p.page_table + (size_t)p.seq_slot[b] * p.pt_stride;
    mbar_expect_tx(q_full, Q_BYTES);
    tma_load_3d(q_sm, &map_q, 0, kvh * G + chunk * GP, t_base + q0, q_full);
    for (int t = 0; t < n_tiles; ++t) {
      const int s = t % NSTG;
      if (!mbar_wait(&kv_empty[s], ((t / NSTG) & 1) ^ 1)) {
        atomicExch(p.status, 14);
        *aborted = 1;
        break;
      }
      if (*aborted) break;
      const int kb = k_begin + t * TK;
      const int page = pt[kb / p.page_size];
      if (page < 0) {               // a visible position without a page: the step's inputs are wrong
        atomicExch(p.status, 2);
        *aborted = 1;
        break;
      }
      const int row = (page * p.Hkv + kvh) * p.page_size + kb % p.page_size;
      if (EXT && p.dist) {
        const int len = dist_len_of(GP), ld = dist_ld(GP), at = dist_at(kb) & ~3;
        mbar_expect_tx(&kv_full[s], 2 * KV_BYTES + GP * len * 4);
        for (int g = 0; g < GP; ++g)
          bulk_load(dist_sm + (s * GP + g) * ld, p.dist + (size_t)(kvh * G + chunk * GP + g) * p.dist_row + at, len * 4, &kv_full[s]);
      } else {
        mbar_expect_tx(&kv_full[s], 2 * KV_BYTES);
      }
      tma_load_2d(k_sm(s), &map_k, 0, row, &kv_full[s]);
      tma_load_2d(v_sm(s), &map_v, 0, row + (vh - kvh) * p.page_size, &kv_full[s]);
    }
  } else if (warp == MMA_WARP && lane == 0) {
    // ---------------------------------------------------------------- MMA issuer
    const unsigned idesc_s = instr_desc(ROWS, TK);                    // Q [128 x 64] . K^T: both K-major
    const unsigned idesc_o = instr_desc(ROWS, HD) | (1u << 16);       // P [128 x 64 keys] . V: V is MN-major
    bool ok = mbar_wait(q_full, 0);
    if (!ok) atomicExch(p.status, 15);
    auto issue_s = [&](int t) {
      const int s = t % NSTG, sb = t & 1;   // the K/V stage; the score buffer
      if (!mbar_wait(&kv_full[s], (t / NSTG) & 1)) {
        atomicExch(p.status, 15);
        return false;
      }
      tc_fence_after();
      const unsigned long long dq = smem_desc(q_sm), dk = smem_desc(k_sm(s));
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)   // 32 bytes further along the swizzled rows per k step
        umma_bf16(tmem_base + T_S + 64u * (unsigned)sb, dq + (unsigned long long)(2 * k), dk + (unsigned long long)(2 * k),
                  idesc_s, k > 0 ? 1u : 0u);
      umma_commit(&s_full[sb]);
      return true;
    };
    if (ok && n_tiles > 0) ok = issue_s(0);
    for (int t = 0; t < n_tiles && ok && !*aborted; ++t) {
      // The scores of the next tile are computed while the softmax warps work on this one: they go to the
      // other score buffer, whose last scores (tile t - 1) were read before P of that tile was announced.
      if (t + 1 < n_tiles) {
        ok = issue_s(t + 1);
        if (!ok) break;
      }
      // the scores are read, P of tile t is in tensor memory, O is rescaled, in every warp
      if (!mbar_wait(&p_ready[t % NP], (t / NP) & 1)) {
        atomicExch(p.status, 16);
        ok = false;
        break;
      }
      tc_fence_after();
      const unsigned long long dv = smem_desc(v_sm(t % NSTG));
#pragma unroll
      for (int k = 0; k < TK / 16; ++k)   // P: 8 columns (16 keys) further; V: 16 key rows of 128 bytes further
        umma_bf16_ta(tmem_o, tmem_base + T_P + 32u * (unsigned)(t % NP) + 8u * (unsigned)k, dv + (unsigned long long)(128 * k),
                     idesc_o, (t > 0 || k > 0) ? 1u : 0u);
      umma_commit(&kv_empty[t % NSTG]);
      umma_commit(&pv_done[t % NP]);
    }
    if (!ok) *aborted = 1;
  } else if (warp < PRODUCER_WARP) {
    // ---------------------------------------------------------------- softmax and epilogue
    const int r = threadIdx.x;                      // row of the tile = accumulator lane
    const int tq = r / GP, hl = r % GP;
    const bool row_ok = q0 + tq < Tq;
    const int row_hi = start + q0 + tq + 1;          // this row sees keys [0, row_hi)
    const unsigned lane_sel = (unsigned)(warp * 32) << 16;
    // scores are kept raw; the scale goes into the exponent: p = 2^((s - m) * scale * log2(e))
    // (with a distance table the scores are scaled as they are read, and only log2(e) is left)
    const float c2 = (EXT && p.dist ? 1.0f : p.scale) * 1.4426950408889634f;
    const int all_visible = start + q0 + 1;          // keys below this are visible to every row of the tile
    // EXT: this row sees keys from row_lo on, every row of the tile keys from lo_last on
    const int row_lo = EXT && p.mask_chunk > 0 ? (row_hi - 1) / p.mask_chunk * p.mask_chunk : 0;
    const int lo_last = EXT && p.mask_chunk > 0 ? (k_end - 1) / p.mask_chunk * p.mask_chunk : 0;
    const float* row_dist = dist_sm + hl * dist_ld(GP) + tq + TK - 1;    // [-j]: key j of a tile
    float m_run = -INFINITY, l_run = 0.f;            // the running maximum; the sum of the exponentials
    bool ok = true;
    // P V of tile t (0 or later) has finished
    auto pv_wait = [&](int t) {
      ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[t % NP], (t / NP) & 1));
      if (!ok) {
        atomicExch(p.status, 18);
        *aborted = 1;
      }
      tc_fence_after();
      return ok;
    };
    for (int t = 0; t < n_tiles; ++t) {
      const int s = t & 1, kb = k_begin + t * TK;
      // (a warp decides as one: the tensor-memory loads and stores below are warp-collective)
      // the scores are there, so the tile has landed; its own barrier makes the slice that came with it visible to this thread
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[s], (t >> 1) & 1) &&
                                       (!EXT || !p.dist || mbar_wait(&kv_full[t % NSTG], (t / NSTG) & 1)));
      if (!ok) {
        atomicExch(p.status, 17);
        *aborted = 1;
        break;
      }
      tc_fence_after();
      float sc[TK];
      tmem_ld64(tmem_base + T_S + 64u * (unsigned)s + lane_sel, sc);
      if (EXT) {
        if (p.dist) {
          const float* d = row_dist + (t % NSTG) * GP * dist_ld(GP) + (dist_at(kb) & 3);
#pragma unroll
          for (int j = 0; j < TK; ++j) sc[j] = fmaf(sc[j], p.scale, d[-j]);
        }
        if (kb < lo_last) {
#pragma unroll
          for (int j = 0; j < TK; ++j) sc[j] = kb + j >= row_lo ? sc[j] : -INFINITY;
        }
      }
      if (kb + TK > all_visible || !row_ok) {          // a tile on the diagonal (or a row that does not exist): mask
        const int lim = row_ok ? row_hi - kb : 0;      // keys of the tile that this row sees
#pragma unroll
        for (int j = 0; j < TK; ++j) sc[j] = j < lim ? sc[j] : -INFINITY;
      }
      float m4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
      for (int j = 4; j < TK; j += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) m4[e] = j + 4 + e < TK ? fmaxf(fmaxf(m4[e], sc[j + e]), sc[j + 4 + e]) : fmaxf(m4[e], sc[j + e]);
      const float m_tile = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      const bool move = m_tile > m_run;
      // both maxima scaled and rounded as the exponents below have them, so that what was summed relative to the old one is
      // brought to the new one exactly, however large the scores are
      const float mc_old = m_run == -INFINITY ? -INFINITY : m_run * c2;
      if (move) m_run = m_tile;
      const float mc = m_run == -INFINITY ? 0.f : m_run * c2;
      const float alpha = move ? ex2(mc_old - mc) : 1.0f;
      l_run *= alpha;
      const float2 c22 = make_float2(c2, c2), mc2 = make_float2(-mc, -mc);
      float2 sum0 = make_float2(0.f, 0.f), sum1 = sum0;
      unsigned pk[TK / 2];
#pragma unroll
      for (int j = 0; j < TK; j += 4) {
        float2 a = fma2(make_float2(sc[j], sc[j + 1]), c22, mc2), b = fma2(make_float2(sc[j + 2], sc[j + 3]), c22, mc2);
        a.x = ex2(a.x);
        a.y = ex2(a.y);
        b.x = ex2(b.x);
        b.y = ex2(b.y);
        sum0 = add2(sum0, a);
        sum1 = add2(sum1, b);
        pk[j / 2] = pack_bf16(a.x, a.y);
        pk[j / 2 + 1] = pack_bf16(b.x, b.y);
      }
      l_run += (sum0.x + sum0.y) + (sum1.x + sum1.y);
      if (t > 0 && __any_sync(0xffffffffu, move)) {    // O follows the new maximum once P V of the tile before is complete
        if (!pv_wait(t - 1)) break;
#pragma unroll
        for (int c0 = 0; c0 < HD; c0 += 32) {
          float o[32];
          tmem_ld32(tmem_o + lane_sel + (unsigned)c0, o);
          unsigned w[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) w[j] = __float_as_uint(o[j] * alpha);
          tmem_st32(tmem_o + lane_sel + (unsigned)c0, w);
        }
      } else if (t >= NP) {                            // its P buffer may be overwritten
        if (!pv_wait(t - NP)) break;
      }
      tmem_st32(tmem_base + T_P + 32u * (unsigned)(t % NP) + lane_sel, pk);
      // rows of V beyond the last key of the sequence's step hold stale cache contents
      if (kb + TK > k_end) {
        const int first = k_end - kb;   // 1 .. 63
        for (int i = threadIdx.x; i < (TK - first) * 8; i += SM_THREADS)
          *reinterpret_cast<uint4*>(v_sm(t % NSTG) + (first + i / 8) * 128 + (i % 8) * 16) = make_uint4(0, 0, 0, 0);
        fence_async_smem();
      }
      tc_fence_before();
      mbar_arrive(&p_ready[t % NP]);
    }
    if (ok) pv_wait(n_tiles - 1);
    if (ok) {   // uniform in the warp: every lane reads its row of O, the rows that exist store it
      float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      if (EXT && p.gate)
        inv /= 1.0f + expf(-to_f32(p.gate[(size_t)(t_base + min(q0 + tq, Tq - 1)) * p.ld_gate + kvh * G + chunk * GP + hl]));
      bf16* dst = p.out + (size_t)(t_base + min(q0 + tq, Tq - 1)) * p.H * HD + (size_t)(kvh * G + chunk * GP + hl) * HD;
      const size_t xrow = ((size_t)(t_base + min(q0 + tq, Tq - 1)) * p.H + (kvh * G + chunk * GP + hl)) * p.Hkv + vh;
      if (cross && row_ok) *reinterpret_cast<float2*>(p.part_ml + xrow * 2) = make_float2(0.f, 1.f);
#pragma unroll
      for (int c0 = 0; c0 < HD; c0 += 16) {
        float o[16];
        tmem_ld16(tmem_o + lane_sel + (unsigned)c0, o);
        if (cross) {
          if (row_ok) {
            float* xdst = p.part_o + xrow * HD + c0;
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              *reinterpret_cast<float4*>(xdst + i) = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
          }
          continue;
        }
        uint4 w0, w1;
        w0.x = pack_bf16(o[0] * inv, o[1] * inv);   w0.y = pack_bf16(o[2] * inv, o[3] * inv);
        w0.z = pack_bf16(o[4] * inv, o[5] * inv);   w0.w = pack_bf16(o[6] * inv, o[7] * inv);
        w1.x = pack_bf16(o[8] * inv, o[9] * inv);   w1.y = pack_bf16(o[10] * inv, o[11] * inv);
        w1.z = pack_bf16(o[12] * inv, o[13] * inv); w1.w = pack_bf16(o[14] * inv, o[15] * inv);
        if (row_ok) {
          *reinterpret_cast<uint4*>(dst + c0) = w0;
          *reinterpret_cast<uint4*>(dst + c0 + 8) = w1;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

int packed_heads(int G) {
  for (int gp = 8; gp >= 1; gp >>= 1)
    if (G % gp == 0) return gp;
  return 1;
}

}  // namespace

extern "C" {

// Whether the kernel takes these sizes, and how many tokens one of its query tiles holds (the host
// builds the tile table with that many tokens per tile).
int zk_attn_prefill_tc5_takes(int H, int Hkv, int hd, int page_size, int window) {
  if (Hkv <= 0 || H % Hkv) return 0;
  return hd == HD && page_size % TK == 0 && window <= 0;
}
// Entries of a padded distance table ahead of distance 0, and equal ones behind its last number.
int zk_attn_prefill_tc5_dist_front() { return DIST_FRONT; }
int zk_attn_prefill_tc5_dist_back() { return DIST_BACK; }
int zk_attn_prefill_tc5_tile_tokens(int H, int Hkv) { return ROWS / packed_heads(H / Hkv); }

// q, out [n_tokens, H*64] bfloat16; k_cache, v_cache [num_pages, Hkv, page_size, 64] bfloat16;
// tiles of zk_attn_prefill_tc5_tile_tokens tokens.  part_o, part_ml (both or neither): the cross mode, see Params;
// `out` is then not written.  dist [H, dist_row] (padded as Params says), mask_chunk, gate, ld_gate: the options of the EXT form, each absent as null or 0;
// none goes with the cross mode.
int zk_attn_prefill_tc5(const void* q, const void* k_cache, const void* v_cache, void* out, const int* tile_seq,
                        const int* tile_q0, const int* cu_q, const int* seq_start, const int* seq_slot,
                        const int* page_table, int pt_stride, int n_tiles, int n_tokens, long long num_pages, int H,
                        int Hkv, int hd, int page_size, float scale, int* status, float* part_o, float* part_ml,
                        const float* dist, int dist_row, int mask_chunk, const void* gate, int ld_gate, cudaStream_t stream) {
  if (n_tiles <= 0 || n_tokens <= 0) return 0;
  const bool ext = dist || mask_chunk > 0 || gate;
  if ((dist && (dist_row % 4 || dist_row < DIST_FRONT + DIST_BACK || (uintptr_t)dist % 16)) || mask_chunk < 0 || (gate && ld_gate < H) || (ext && part_o)) return ZK_EINVAL;
  if ((part_o == nullptr) != (part_ml == nullptr) || ((uintptr_t)part_o % 16) || (part_o && Hkv > 65535)) return ZK_EINVAL;
  if (!zk_attn_prefill_tc5_takes(H, Hkv, hd, page_size, 0) || !status || num_pages <= 0) return ZK_EINVAL;
  if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) % 16) return ZK_EINVAL;
  EncodeTiledFn fn = encode_fn();
  if (!fn) return ZK_EINVAL;
  const int G = H / Hkv, gp = packed_heads(G);
  CUtensorMap mq, mk, mv;
  {
    const cuuint64_t dims[3] = {(cuuint64_t)HD, (cuuint64_t)H, (cuuint64_t)n_tokens};
    const cuuint64_t strides[2] = {(cuuint64_t)HD * 2, (cuuint64_t)H * HD * 2};
    const cuuint32_t box[3] = {(cuuint32_t)HD, (cuuint32_t)gp, (cuuint32_t)(ROWS / gp)};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (fn(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return ZK_EINVAL;
  }
  for (int which = 0; which < 2; ++which) {
    const cuuint64_t dims[2] = {(cuuint64_t)HD, (cuuint64_t)num_pages * Hkv * page_size};
    const cuuint64_t strides[1] = {(cuuint64_t)HD * 2};
    const cuuint32_t box[2] = {(cuuint32_t)HD, (cuuint32_t)TK};
    const cuuint32_t estr[2] = {1, 1};
    if (fn(which ? &mv : &mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(which ? v_cache : k_cache), dims,
           strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return ZK_EINVAL;
  }
  Params p{};
  p.out = (bf16*)out; p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.cu_q = cu_q; p.seq_start = seq_start;
  p.seq_slot = seq_slot; p.page_table = page_table; p.status = status;
  p.pt_stride = pt_stride; p.H = H; p.Hkv = Hkv; p.page_size = page_size; p.gp = gp; p.scale = scale;
  p.part_o = part_o; p.part_ml = part_ml;
  p.dist = dist; p.dist_row = dist_row; p.mask_chunk = mask_chunk; p.gate = (const bf16*)gate; p.ld_gate = ld_gate;
  auto kern = ext ? attn_prefill_tc5_kernel<true> : attn_prefill_tc5_kernel<false>;
  const size_t smem = SMEM_BYTES + (dist ? (size_t)NSTG * gp * dist_ld(gp) * sizeof(float) : 0);
  // The limit belongs to the kernel and is shared by all threads of the process: every call sets it to the most that any call
  // needs, so that none lowers it between another's setting and launch.
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(SMEM_BYTES + (ext ? DIST_BYTES : 0)));
  if (e != cudaSuccess) return (int)e;
  if ((long long)n_tiles * Hkv * (G / gp) > 0x7fffffffLL) return ZK_EINVAL;
  dim3 grid(n_tiles * Hkv * (G / gp), 1, part_o ? Hkv : 1);
  return zk_launch_dependent(kern, grid, dim3(THREADS), smem, stream, mq, mk, mv, p);
}

}  // extern "C"
