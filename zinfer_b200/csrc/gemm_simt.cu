// C[M, N] (+)= A[M, K] . W[N, K]^T (+ bias[N]) on the CUDA cores with float32 FMA.
//
// This is the contraction of the true 32-bit path and the fallback of the bfloat16 path for
// shapes the tensor-core kernels refuse.  Each output element is one float32 accumulator that
// walks k = 0 .. K-1 in order, or, where N and K ask for it (`split_k`), the sum in order of the
// accumulators of four stretches of k, so a row's result does not depend on M, on the row's place in
// the batch or on the tile it falls in (reference: one dot product per output row,
// src/model.zig:923-1026; float32 dot src/quant.zig:424-431; `accumulate` = residual add,
// src/model.zig:918-920).  All kernels here keep that order, so they give the same bits and the
// launcher may pick among them by size.
#include "common.cuh"

namespace {

// ------------------------------------------------------------------------------ stretches of k
// A contraction with few outputs leaves SMs idle, and its blocks walk a long chain of dependent FMAs.  There the sum over k is that
// of SEGMENTS stretches, in order; N and K alone decide, not M: the sums of a row are the same in any batch.  How the
// stretches are run depends on how many blocks the rows give:
//  * BY_CLUSTER: a block of a cluster each.  A block leaves its sums in shared memory, and the blocks then share the outputs out
//    among themselves and add the stretches;
//  * IN_TURN: one block all of them, where there are blocks enough.
// Float32, microseconds with one accumulator per output and now: N = 1024, K = 4608, 1 / 8 / 64 / 256 / 450 rows 27 / 28 / 82 / 120 / 169 ->
// 13 / 18 / 47 / 74 / 138; K = 1024, 16 / 450 rows 14 / 44 -> 12 / 41.  The error against 64 bits is smaller (four shorter sums): a model's
// logits 6.1e-6 -> 4.4e-6.  What it costs: from 500 rows on, where blocks are no longer few, IN_TURN is 1 to 5 % slower than one accumulator
// (2,000 rows, N = 1024, K = 1024, bfloat16 120 -> 125 us), and some sizes of 7 to 48 rows are 3 to 7 % slower.
constexpr int SEGMENTS = 4;
enum { WHOLE = 0, BY_CLUSTER = 1, IN_TURN = 2 };

// Where stretch i of K begins: the 512-byte blocks of a row that gemm_few_kernel walks, shared out whole (K of 1,024 and more has at least
// four of them).
template <typename T>
__host__ __device__ inline int stretch_at(int K, int i) {
  constexpr int KC = 512 / (int)sizeof(T);
  const int at = (K + KC - 1) / KC * i / SEGMENTS * KC;
  return at < K ? at : K;
}

__device__ __forceinline__ float ld_cluster(const float* local, unsigned rank) {
  unsigned remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// ------------------------------------------------------------------------------ tiles
// A block owns BM x BN outputs, a thread TM x TN of them in groups of 4 adjacent rows and 4 adjacent columns.  The
// operands lie in shared memory as [k][row], so that a group is one 16-byte load; two buffers, PF k blocks further on being
// fetched into registers while this one is multiplied (one barrier per k block).
//
// What bounds it: 128 FMAs a cycle and SM (74 TFLOP/s) against 128 bytes a cycle from shared memory into registers, which
// 8 x 8 outputs per thread just balance (8 x 4 need 1.5 times, 4 x 4 twice the time of their FMAs for their loads); packed
// FMAs (fma.rn.f32x2) leave the issue slots to the loads, 7 to 10 % over single ones.  8 x 16 outputs (one block of 128 threads
// in place of two of 256 per SM) were no faster.  Float32, [450, K] rows, microseconds before (64 x 64 tiles, 4 x 4 outputs, one
// buffer) and now: N = 9216, K = 1024 320 -> 192 (44 TFLOP/s); N = 65536 1962 -> 1230 (49 TFLOP/s); N = 1024, K = 4608
// 334 -> 169; N = 1024, K = 1024 72 -> 42.
constexpr int BK = 16, PAD = 4;

// Four adjacent values of a row, as they are stored until they are put into shared memory: widened at the load, bfloat16 values
// were waited for there, and no k block was under way beside the FMAs.  PACKED: bfloat16 rows that allow 8-byte loads, two values
// to a register.  [450, 1024] x 9216 with bfloat16 operands, microseconds with values widened at the load and now: 260 -> 197
// (305 with 64 x 64 tiles, 4 x 4 outputs, one buffer); K = 1022, whose rows allow no 8-byte loads, 277 -> 231 (391);
// [16, 1024] x 9216 104 -> 35 (96); [128, 1022] x 4736 182 -> 57 (119).
template <typename T, bool PACKED> struct Four { T v[4]; };
template <> struct Four<bf16, true> { uint2 v; };

template <typename T, bool PACKED>
__device__ __forceinline__ float nth(const Four<T, PACKED>& f, int j) {
  if constexpr (PACKED) {
    const unsigned w = j < 2 ? f.v.x : f.v.y;
    return __uint_as_float((j & 1) ? w & 0xffff0000u : w << 16);
  } else {
    return to_f32(f.v[j]);
  }
}

// Values beyond K, and those of a row that does not exist, are zeros.
template <typename T, bool PACKED>
__device__ __forceinline__ void load4(const T* __restrict__ p, bool vec_ok, int k0, int K, bool row_ok, Four<T, PACKED>& out) {
  if constexpr (PACKED) {
    if (row_ok && k0 + 3 < K) {
      out.v = *reinterpret_cast<const uint2*>(p + k0);
      return;
    }
    unsigned h[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) h[j] = row_ok && k0 + j < K ? __bfloat16_as_ushort(p[k0 + j]) : 0;
    out.v = make_uint2(h[0] | h[1] << 16, h[2]);
  } else if constexpr (sizeof(T) == 4) {
    if (!row_ok) {
      out.v[0] = out.v[1] = out.v[2] = out.v[3] = 0.f;
      return;
    }
    if (vec_ok && k0 + 3 < K) {
      const float4 v = *reinterpret_cast<const float4*>(p + k0);
      out.v[0] = v.x; out.v[1] = v.y; out.v[2] = v.z; out.v[3] = v.w;
      return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) out.v[j] = (k0 + j < K) ? p[k0 + j] : 0.f;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) out.v[j] = row_ok && k0 + j < K ? p[k0 + j] : from_f32<T>(0.f);
  }
}

// Two float32 FMAs in one instruction, each rounded as fmaf rounds.
__device__ __forceinline__ void fma2(float2& d, float a, float2 b) {
  unsigned long long dd, aa, bb;
  asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(dd) : "f"(d.x), "f"(d.y));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(dd) : "l"(aa), "l"(bb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(dd));
}

// vecA, vecW: rows that allow loads of four float32 values (PACKED: both operands' rows allow loads of four bfloat16 values).
// BY_CLUSTER and IN_TURN keep the tile's sums in dynamic shared memory [BM][BN].
template <int BM, int BN, int TM, int TN, int PF, bool PACKED, int MODE, typename T, typename TC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN >= 64 ? 2 : 3)
    gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, TC* __restrict__ C, const float* __restrict__ bias,
                     int M, int N, int K_all, int lda, int ldw, int ldc, int accumulate, int vecA, int vecW) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  constexpr int GM = TM / 4, GN = TN / 4;                   // groups of 4 rows / columns per thread
  constexpr int LA = BM * BK / 4 / THREADS, LW = BN * BK / 4 / THREADS;   // 4-value pieces a thread fetches per k block
  static_assert(LA * THREADS * 4 == BM * BK && LW * THREADS * 4 == BN * BK, "whole pieces per thread");
  __shared__ __align__(16) float As[2][BK][BM + PAD];
  __shared__ __align__(16) float Ws[2][BK][BN + PAD];
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  constexpr bool RUN_ON = MODE == IN_TURN && TM * TN < 64 && PACKED;  // the k blocks under way run on from stretch to stretch
  int K = MODE == IN_TURN && !RUN_ON ? stretch_at<T>(K_all, 1) : K_all;
  if constexpr (MODE == BY_CLUSTER) {
    const int k0 = stretch_at<T>(K_all, (int)cluster_rank());
    K = stretch_at<T>(K_all, (int)cluster_rank() + 1) - k0;
    A += k0;
    W += k0;
  }
  extern __shared__ __align__(16) float tile[];
  auto in_tile = [&](int i, int j) {                        // where the 4 sums of row i, group j lie
    return reinterpret_cast<float4*>(tile + ((i / 4) * (BM / GM) + ty * 4 + (i & 3)) * BN + j * (BN / GN) + tx * 4);
  };

  float2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);

  Four<T, PACKED> av[PF][LA], wv[PF][LW];
  auto fetch = [&](int kb, int f) {
#pragma unroll
    for (int l = 0; l < LA; ++l) {
      const int p = tid + l * THREADS, r = p >> 2, k = (p & 3) * 4;
      const bool ok = m0 + r < M;
      load4<T, PACKED>(A + (size_t)(ok ? m0 + r : 0) * lda, vecA, kb + k, K, ok, av[f][l]);
    }
#pragma unroll
    for (int l = 0; l < LW; ++l) {
      const int p = tid + l * THREADS, r = p >> 2, k = (p & 3) * 4;
      const bool ok = n0 + r < N;
      load4<T, PACKED>(W + (size_t)(ok ? n0 + r : 0) * ldw, vecW, kb + k, K, ok, wv[f][l]);
    }
  };
  auto put = [&](int buf, int f) {
#pragma unroll
    for (int l = 0; l < LA; ++l) {
      const int p = tid + l * THREADS, r = p >> 2, k = (p & 3) * 4;
#pragma unroll
      for (int j = 0; j < 4; ++j) As[buf][k + j][r] = nth(av[f][l], j);
    }
#pragma unroll
    for (int l = 0; l < LW; ++l) {
      const int p = tid + l * THREADS, r = p >> 2, k = (p & 3) * 4;
#pragma unroll
      for (int j = 0; j < 4; ++j) Ws[buf][k + j][r] = nth(wv[f][l], j);
    }
  };

  // PF k blocks are under way in registers; the body of PF rounds is unrolled so that each has registers of its own.  With small
  // tiles they run on from one stretch to the next.  A thread with 64 sums has no registers left for them while it adds those up (2,000
  // rows, N = 2304, K = 4608, float32: 930 us, 842 with every stretch begun anew).
  int buf = 0, k_from = 0, k_to = RUN_ON ? stretch_at<T>(K_all, 1) : K;
  for (int turn = 0; turn < (MODE == IN_TURN ? SEGMENTS : 1); ++turn) {
    if (MODE == IN_TURN && turn > 0) {                      // the stretch before goes to what is there
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < GN; ++j) {
          float4 v = make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
          if (turn > 1) {
            const float4 o = *in_tile(i, j);
            v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w;
          }
          *in_tile(i, j) = v;
          acc[i][2 * j] = acc[i][2 * j + 1] = make_float2(0.f, 0.f);
        }
      if (RUN_ON) {
        k_from = k_to;
        k_to = stretch_at<T>(K_all, turn + 1);
      } else {
        A += K;
        W += K;
        k_to = K = stretch_at<T>(K_all, turn + 1) - stretch_at<T>(K_all, turn);
        __syncthreads();                                    // the buffers are free
        buf = 0;
      }
    }
    if (!RUN_ON || turn == 0) {
#pragma unroll
      for (int f = 0; f < PF; ++f) fetch(f * BK, f);        // beyond K: zeros
      put(0, 0);
      __syncthreads();
    }
    for (int kb0 = k_from; kb0 < k_to; kb0 += PF * BK) {
#pragma unroll
      for (int f = 0; f < PF; ++f) {
        const int kb = kb0 + f * BK;
        if (kb >= k_to) break;
        fetch(kb + PF * BK, f);                               // this block's values are in shared memory since the round before
#pragma unroll
        for (int k = 0; k < BK; ++k) {
          float a[TM];
          float2 b[TN / 2];
#pragma unroll
          for (int i = 0; i < GM; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(&As[buf][k][i * (BM / GM) + ty * 4]);
            a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
          }
#pragma unroll
          for (int j = 0; j < GN; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(&Ws[buf][k][j * (BN / GN) + tx * 4]);
            b[2 * j] = make_float2(v.x, v.y);
            b[2 * j + 1] = make_float2(v.z, v.w);
          }
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], a[i], b[j]);
        }
        if (kb + BK < K) {
          put(buf ^ 1, (f + 1) % PF);
          __syncthreads();
          buf ^= 1;
        }
      }
    }
  }

  if constexpr (MODE == BY_CLUSTER) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < GN; ++j)
        *in_tile(i, j) = make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
    cluster_barrier();
    constexpr int PER = BM * BN / SEGMENTS / THREADS;       // outputs of this block per thread
    const int first = (int)cluster_rank() * (BM * BN / SEGMENTS) + tid;
#pragma unroll 4
    for (int e = 0; e < PER; ++e) {
      const int at = first + e * THREADS, m = m0 + at / BN, n = n0 + at % BN;
      float v = ld_cluster(tile + at, 0);
#pragma unroll
      for (int r = 1; r < SEGMENTS; ++r) v += ld_cluster(tile + at, r);
      if (m >= M || n >= N) continue;
      if (bias) v += bias[n];
      TC* c = C + (size_t)m * ldc + n;
      if (accumulate) v += to_f32(*c);
      *c = from_f32<TC>(v);
    }
    cluster_barrier();                                      // nobody leaves while its sums may still be read
    return;
  }
  const bool vecC = sizeof(TC) == 4 && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i / 4) * (BM / GM) + ty * 4 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < GN; ++j) {
      const int n = n0 + j * (BN / GN) + tx * 4;
      float v[4] = {acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y};
      if constexpr (MODE == IN_TURN) {
        const float4 o = *in_tile(i, j);
        v[0] = o.x + v[0]; v[1] = o.y + v[1]; v[2] = o.z + v[2]; v[3] = o.w + v[3];
      }
      TC* c = C + (size_t)m * ldc + n;
      if (vecC && n + 3 < N) {
        if constexpr (sizeof(TC) == 4) {
          if (bias) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] += bias[n + e];
          }
          if (accumulate) {
            const float4 o = *reinterpret_cast<const float4*>(c);
            v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
          }
          *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (n + e >= N) continue;
          float t = v[e];
          if (bias) t += bias[n + e];
          if (accumulate) t += to_f32(c[e]);
          c[e] = from_f32<TC>(t);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------ few rows
// Up to 64 rows of A (single-token steps, short prompts): what counts is that the weights stream and that the chain of K
// dependent FMAs runs at its 4 cycles each.  A block owns 16 weight rows; its threads keep a ring of k blocks of W and
// A under way with 16-byte asynchronous copies, and thread (row, group) adds the products of its weight row with the
// rows group, group + GROUPS, ... of A in k order, the operands of the next 16 k in registers before they are needed.
// A row of the ring is 16 bytes longer than its values, so that the 16-byte loads of 8 adjacent rows fall into different
// banks.  Two float32 rows, microseconds before (the tiled form: 64 x 64, one buffer) and now: N = 1024, K = 4608 385 -> 23
// (K dependent FMAs alone are 9.4); N = 9216, K = 1024 86 -> 17; N = 65536 278 -> 74 (3.6 TB/s).
constexpr int FEW_ROWS = 16, FEW_MAX_M = 64;

__device__ __forceinline__ void cp16(void* dst, const void* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = in ? 16 : 0;                                 // fewer source bytes than 16: the rest is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <typename T>
__device__ __forceinline__ float4 four(const T* p) {
  if constexpr (sizeof(T) == 4) {
    return *reinterpret_cast<const float4*>(p);
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&v.x);
    const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
    return make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
  }
}

// GROUPS: threads per weight row; NT: rows of A per thread (GROUPS * NT >= M); STAGES of the ring.  A block takes the stretches of
// 16 weight rows blockIdx.x, blockIdx.x + gridDim.x, ...; its ring runs on from one to the next.  BY_CLUSTER: the sums meet in shared
// memory behind the ring, [M][16].
template <int GROUPS, int NT, int STAGES, int MODE, typename T, typename TC>
__global__ void __launch_bounds__(FEW_ROWS * GROUPS)
    gemm_few_kernel(const T* __restrict__ A, const T* __restrict__ W, TC* __restrict__ C, const float* __restrict__ bias,
                    int M, int N, int K_all, int lda, int ldw, int ldc, int accumulate) {
  constexpr int THREADS = FEW_ROWS * GROUPS;
  constexpr bool WALKS = MODE == BY_CLUSTER || (MODE == WHOLE && GROUPS <= 2);      // else a block has one task
  constexpr int PIECE = 16 / (int)sizeof(T), KC = 512 / (int)sizeof(T), LD = KC + PIECE;   // 512 bytes of a row per k block
  extern __shared__ __align__(16) unsigned char few_smem[];
  T* ring = reinterpret_cast<T*>(few_smem);
  const int rows = FEW_ROWS + M;                             // W's rows, then A's
  const int tid = threadIdx.x;
  const int tasks = (N + FEW_ROWS - 1) / FEW_ROWS;
  const int first_task = blockIdx.x, task_step = gridDim.x;
  int K = K_all;
  if constexpr (MODE == BY_CLUSTER) {
    const int k0 = stretch_at<T>(K_all, (int)cluster_rank());
    K = stretch_at<T>(K_all, (int)cluster_rank() + 1) - k0;
    A += k0;
    W += k0;
  }
  const int n_kb = (K + KC - 1) / KC;                        // k blocks of a task
  // a warp copies whole rows (32 pieces of 16 bytes): lane = piece, warps take rows in turn
  const int e = (tid & 31) * PIECE;
  auto request = [&](int task, int kb, int stage) {
    T* dst = ring + (size_t)stage * rows * LD + e;
    const int n0 = task * FEW_ROWS, k = kb * KC + e;
    const bool k_in = k < K;                                 // K is a whole number of pieces
    const T* wk = W + (k_in ? k : 0);
    const T* ak = A + (k_in ? k : 0);
#pragma unroll
    for (int r = tid >> 5; r < FEW_ROWS; r += THREADS / 32) {
      const bool in = k_in && n0 + r < N;
      cp16(dst + r * LD, wk + (size_t)(in ? n0 + r : 0) * ldw, in);
    }
    for (int r = tid >> 5; r < M; r += THREADS / 32) cp16(dst + (FEW_ROWS + r) * LD, ak + (size_t)r * lda, k_in);
  };
  // Requests the k block that follows those under way: of a block that walks, the next of this task or of the one after it; else kb.
  int r_task = first_task, r_kb = 0, r_stage = 0;
  auto request_next = [&](int kb) {
    if constexpr (WALKS) {
      if (r_task < tasks) request(r_task, r_kb, r_stage);
      if (++r_kb == n_kb) {
        r_kb = 0;
        r_task += task_step;
      }
      if (++r_stage == STAGES) r_stage = 0;
    } else {
      if (kb < n_kb) request(first_task, kb, kb % STAGES);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // More than two rows: the next kernel's blocks, let in early, fell unevenly onto the SMs beside this one's ([8, 1024] x 3072 twenty
  // times in a row: 12.8 us, 10.9 without).  The weights are requested behind the wait too: nothing says that no kernel wrote them.
  if (GROUPS <= 2) zk_let_next_start();
  zk_wait_prior();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) request_next(s);
  const int row = tid % FEW_ROWS, group = tid / FEW_ROWS;
  float acc[NT], total[MODE == IN_TURN ? NT : 1];
  int at[NT];                                                // where the rows of A lie in a stage
#pragma unroll
  for (int t = 0; t < NT; ++t) at[t] = (FEW_ROWS + (group + t * GROUPS < M ? group + t * GROUPS : 0)) * LD;   // no such row: another's, not stored
  int stage = 0;
  for (int task = first_task; task < tasks; task += WALKS ? task_step : tasks) {
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0.f;
    for (int turn = 0, kb = 0; turn < (MODE == IN_TURN ? SEGMENTS : 1); ++turn) {
      const int stretch_end = MODE == IN_TURN ? n_kb * (turn + 1) / SEGMENTS : n_kb;
      for (; kb < stretch_end; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                     // the k block is here, and nobody reads the one before it
        const T* st = ring + (size_t)(WALKS ? stage : kb % STAGES) * rows * LD;
        float4 x[2][4], y[2][NT][4];
        auto read = [&](int k, int b) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[b][i] = four(st + row * LD + k + 4 * i);
#pragma unroll
            for (int t = 0; t < NT; ++t) y[b][t][i] = four(st + at[t] + k + 4 * i);
          }
        };
        read(0, 0);
        request_next(kb + STAGES - 1);
#pragma unroll
        for (int k = 0; k < KC; k += 16) {
          const int b = (k >> 4) & 1;
          if (k + 16 < KC) read(k + 16, b ^ 1);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = fmaf(y[b][t][i].x, x[b][i].x, acc[t]);
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = fmaf(y[b][t][i].y, x[b][i].y, acc[t]);
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = fmaf(y[b][t][i].z, x[b][i].z, acc[t]);
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = fmaf(y[b][t][i].w, x[b][i].w, acc[t]);
          }
        }
        if (WALKS && ++stage == STAGES) stage = 0;
      }
      if constexpr (MODE == IN_TURN) {                       // a stretch ends
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          total[t] = turn ? total[t] + acc[t] : acc[t];
          acc[t] = 0.f;
        }
      }
    }
    if constexpr (MODE == IN_TURN) {
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[t] = total[t];
    }
    const int n = task * FEW_ROWS + row;
    if constexpr (MODE == BY_CLUSTER) {
      float* sums = reinterpret_cast<float*>(ring + (size_t)STAGES * rows * LD);
#pragma unroll
      for (int t = 0; t < NT; ++t)
        if (group + t * GROUPS < M) sums[(group + t * GROUPS) * FEW_ROWS + row] = acc[t];
      cluster_barrier();
      for (int i = cluster_rank() * THREADS + tid; i < M * FEW_ROWS; i += SEGMENTS * THREADS) {
        float v = ld_cluster(sums + i, 0);
#pragma unroll
        for (int r = 1; r < SEGMENTS; ++r) v += ld_cluster(sums + i, r);
        const int m = i / FEW_ROWS, col = task * FEW_ROWS + i % FEW_ROWS;
        if (col >= N) continue;
        if (bias) v += bias[col];
        TC* c = C + (size_t)m * ldc + col;
        if (accumulate) v += to_f32(*c);
        *c = from_f32<TC>(v);
      }
      cluster_barrier();                                     // the sums have been read; nobody writes others, or leaves, before
    } else if (n < N) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int m = group + t * GROUPS;
        if (m >= M) continue;
        float v = acc[t];
        if (bias) v += bias[n];
        TC* c = C + (size_t)m * ldc + n;
        if (accumulate) v += to_f32(*c);
        *c = from_f32<TC>(v);
      }
    }
  }
}

template <typename... KArgs, typename... Args>
int launch_cluster(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, int cluster, bool dependent, cudaStream_t stream,
                   Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = dependent ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = cluster;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

// Whether the sum over k is that of stretches: with few outputs and a chain of k worth cutting.
inline bool split_k(int N, int K) { return K >= 1024 && ceil_div_i(N, FEW_ROWS) <= 148; }

template <int BM, int BN, int TM, int TN, int PF, int MODE, typename T, typename TC>
int launch_tiles(const void* A, const void* W, void* C, const float* bias, int M, int N, int K, int lda, int ldw, int ldc,
                 int accumulate, cudaStream_t stream) {
  const int vecA = (lda % 4 == 0) && ((uintptr_t)A % 16 == 0);
  const int vecW = (ldw % 4 == 0) && ((uintptr_t)W % 16 == 0);
  auto kern = gemm_simt_kernel<BM, BN, TM, TN, PF, false, MODE, T, TC>;
  if constexpr (sizeof(T) == 2)
    if (vecA && vecW) kern = gemm_simt_kernel<BM, BN, TM, TN, PF, true, MODE, T, TC>;
  constexpr size_t smem = MODE != WHOLE ? sizeof(float) * BM * BN : 0;
  if constexpr (smem > 8 * 1024) {          // with the operands' buffers more than the 48 KB a block may have unasked
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  // Not launched ahead of the end of the kernel before: its blocks would then fall unevenly onto the SMs ([16, 1024] x 9216 twenty
  // times in a row: 47.8 us, 28.9 so).
  return launch_cluster(kern, dim3(ceil_div_i(N, BN), ceil_div_i(M, BM), MODE == BY_CLUSTER ? SEGMENTS : 1), (BM / TM) * (BN / TN), smem,
                        MODE == BY_CLUSTER ? SEGMENTS : 1, false, stream, (const T*)A, (const T*)W, (TC*)C, bias, M, N, K, lda, ldw,
                        ldc, accumulate, vecA, vecW);
}

template <int GROUPS, int NT, int STAGES, int MODE, typename T, typename TC>
int launch_few(const void* A, const void* W, void* C, const float* bias, int M, int N, int K, int lda, int ldw, int ldc,
               int accumulate, cudaStream_t stream) {
  auto kern = gemm_few_kernel<GROUPS, NT, STAGES, MODE, T, TC>;
  constexpr size_t ROW = (size_t)STAGES * (512 + 16), SUMS = MODE == BY_CLUSTER ? sizeof(float) * FEW_ROWS : 0;
  // The limit belongs to the instantiation and is shared by all threads of the process: every call sets it to what the largest M
  // needs, so that none lowers it between another's setting and launch.
  constexpr size_t LIMIT = ROW * (FEW_ROWS + GROUPS * NT) + SUMS * (GROUPS * NT);
  const size_t smem = ROW * (FEW_ROWS + M) + SUMS * M;
  if (smem > LIMIT) return ZK_EINVAL;
  if constexpr (LIMIT > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIMIT);
    if (e != cudaSuccess) return (int)e;
  }
  // One or two rows, and sums of stretches: no more blocks than fit beside one another, each with (nearly) as many tasks as any
  // other.  More rows whose sums are whole multiply longer per byte, and blocks that come one after the other hide more of it: 4 and
  // 8 rows, N = 65536, K = 1024, float32 75 and 114 us, 85 and 123 with blocks that stay.
  const int tasks = ceil_div_i(N, FEW_ROWS), clusters = MODE == BY_CLUSTER ? SEGMENTS : 1;
  const int per_sm = (int)(227 * 1024 / (smem + 1024)), at_once = 148 * (per_sm > 0 ? per_sm : 1) / clusters;
  const int rounds = MODE == IN_TURN || (MODE == WHOLE && GROUPS > 2) ? 1 : ceil_div_i(tasks, at_once);
  return launch_cluster(kern, dim3(ceil_div_i(tasks, rounds), 1, clusters), FEW_ROWS * GROUPS, smem, clusters, true, stream,
                        (const T*)A, (const T*)W, (TC*)C, bias, M, N, K, lda, ldw, ldc, accumulate);
}

template <int MODE, typename T, typename TC>
int launch_few_rows(const void* A, const void* W, void* C, const float* bias, int M, int N, int K, int lda, int ldw, int ldc,
                    int accumulate, cudaStream_t stream) {
  // One or two rows are blocks of a warp, whose bfloat16 products come faster than four stages fill: with three, seven blocks share an
  // SM instead of five (2 rows, N = 65536, K = 1024: 59 us, 66 with four).
  if (M <= 2) return launch_few<2, 1, sizeof(T) == 2 ? 3 : 4, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (M <= 4) return launch_few<4, 1, 6, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (M <= 8) return launch_few<8, 1, 6, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (M <= 16) return launch_few<16, 1, 5, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (M <= 32) return launch_few<16, 2, 4, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  return launch_few<16, 4, 3, MODE, T, TC>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
}

template <typename T, typename TC>
int launch(const void* A, const void* W, void* C, const float* bias, int M, int N, int K, int lda, int ldw, int ldc,
           int accumulate, cudaStream_t stream) {
  constexpr int PIECE = 16 / (int)sizeof(T);
  const bool pieces = K % PIECE == 0 && lda % PIECE == 0 && ldw % PIECE == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
  const bool split = split_k(N, K);
#define ZK_SIMT_ARGS A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream
  // The few-row form reads A once per 16 weight rows, which pays while the weights are the larger part or a tiled form would
  // leave most SMs idle.  Microseconds at 20 rows, few / 32 x 32 tiles: N = 1024 15 / 27 (K = 1024), 50 / 117 (K = 4608);
  // N = 9216 44 / 31.  A k block is 512 bytes of a row, and what K leaves of it is zeros: with less than one block the form pays
  // only where both hold (K = 64, bfloat16, few / tiles: 8 x 65536 33 / 21, 40 x 4736 16 / 8, 8 x 3072 8 / 8).
  const int tasks = ceil_div_i(N, FEW_ROWS);
  const bool little = M <= 8, narrow = tasks <= 2 * 148, whole = K * sizeof(T) >= 512;
  if (pieces && M <= FEW_MAX_M && (whole ? little || narrow : little && narrow)) {
    if (!split) return launch_few_rows<WHOLE, T, TC>(ZK_SIMT_ARGS);
    // A cluster per 16 weight rows while those leave SMs idle, or while the rows are so few that the chain of k is all there is.  From 57
    // rows on an SM holds one block, and 74 clusters of four no longer run in two rounds (64 rows, N = 1184, K = 1536, bfloat16: 47 us, 35 in
    // turn); 8 rows, N = 2304, K = 4608, bfloat16: 32 us, 26 in turn.
    const bool cluster = tasks <= (M > 56 ? 64 : 74) || M <= 2 || (M <= 4 && K >= 1536) || (M <= 8 && K >= 4096 && tasks <= 128);
    return cluster ? launch_few_rows<BY_CLUSTER, T, TC>(ZK_SIMT_ARGS) : launch_few_rows<IN_TURN, T, TC>(ZK_SIMT_ARGS);
  }
  // The largest tile that still gives (nearly) every SM a block, and no taller than the rows need: 128 rows of A cost their
  // FMAs whether they exist or not (16 rows, N = 65536, K = 1024: 350 / 190 / 154, and 277 with one buffer).  450 rows, microseconds with 128 x 128 / 64 x 64 / 32 x 32
  // tiles: N = 9216, K = 1024 195 / 224 / 326; N = 1024, K = 4608 474 / 169 / 199; 100 rows of the latter 463 / 165 / 111.
  const int blocks128 = ceil_div_i(M, 128) * ceil_div_i(N, 128), blocks64 = ceil_div_i(M, 64) * ceil_div_i(N, 64);
  if (split) {
    if (M > 64 && blocks128 >= 148) return launch_tiles<128, 128, 8, 8, 1, IN_TURN, T, TC>(ZK_SIMT_ARGS);
    if (M > 32 && blocks64 >= 140) return launch_tiles<64, 64, 8, 4, 2, IN_TURN, T, TC>(ZK_SIMT_ARGS);
    if (M > 32 && SEGMENTS * blocks64 >= 100) return launch_tiles<64, 64, 8, 4, 2, BY_CLUSTER, T, TC>(ZK_SIMT_ARGS);
    return launch_tiles<32, 32, 4, 4, 4, BY_CLUSTER, T, TC>(ZK_SIMT_ARGS);
  }
  if (M > 64 && blocks128 >= 148) return launch_tiles<128, 128, 8, 8, 1, WHOLE, T, TC>(ZK_SIMT_ARGS);
  if (M > 32 && blocks64 >= 100) return launch_tiles<64, 64, 8, 4, 2, WHOLE, T, TC>(ZK_SIMT_ARGS);
  return launch_tiles<32, 32, 4, 4, 4, WHOLE, T, TC>(ZK_SIMT_ARGS);
#undef ZK_SIMT_ARGS
}

}  // namespace

extern "C" int zk_gemm_simt(const void* A, const void* W, void* C, const float* bias, int M, int N, int K, int lda,
                            int ldw, int ldc, int in_dtype, int out_dtype, int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return ZK_EINVAL;
  if (in_dtype == ZK_F32 && out_dtype == ZK_F32)
    return launch<float, float>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (in_dtype == ZK_BF16 && out_dtype == ZK_F32)
    return launch<bf16, float>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  if (in_dtype == ZK_BF16 && out_dtype == ZK_BF16)
    return launch<bf16, bf16>(A, W, C, bias, M, N, K, lda, ldw, ldc, accumulate, stream);
  return ZK_EINVAL;
}
