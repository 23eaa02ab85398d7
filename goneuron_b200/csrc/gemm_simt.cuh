// gemm_simt.cuh -- strided, batched fp32 contraction on the CUDA cores.
//
// C[b](m,n) = act( alpha * sum_k A[b](m,k) * B[b](k,n) + bias[n] + R[b](m,n) )
// with arbitrary element strides for A and B, so every transpose variant of the
// training step (X*W^T, dZ*W, dZ^T*X, Q*K^T, P*V, dS^T*Q ...) and every sub-view
// (one head of a [tokens, d] tensor, the last token of every sequence) is the same
// kernel.  It is the exact-fp32 engine: small and oddly shaped contractions use it,
// and the tensor-core engine is checked against it.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace gn {

enum { GEMM_KBEG_AT_M0 = 1, GEMM_KEND_AT_M0 = 2, GEMM_SKIP_UPPER = 4 };

struct GemmDesc {
  int M = 0, N = 0, K = 0;
  const float* A = nullptr; long sa_m = 0, sa_k = 0;
  const float* B = nullptr; long sb_k = 0, sb_n = 0;   // B(k,n)
  float* C = nullptr; long ldc = 0;
  const float* bias = nullptr;                          // [N]
  const float* R = nullptr; long ldr = 0;               // residual added to the result (may alias C)
  int act = GN_ACT_LINEAR;                              // LINEAR or RELU
  // optional gate: result(m,n) is zeroed unless mask[(m / mask_group) * mask_ld + n] > 0 (the ReLU pattern of the
  // last token of row m's sequence, see relu_mask semantics in model.cu)
  const float* mask = nullptr; long mask_ld = 0; int mask_group = 1;
  float alpha = 1.f;
  bool reuse_a_planes = false;                          // A is the same tensor as in the previous tensor-core call of this context
  const void* b_planes = nullptr;                       // tensor-core engine: prepared operand planes of B (a BfPlanes), e.g. of a weight matrix
  const void* a_planes = nullptr;                       // ... and of A (written by the epilogue of the contraction that produced A)
  const void* plane_out = nullptr;                      // tensor-core engine: a TcPlaneOut; the result is written as operand planes instead of fp32
  float* a_sum = nullptr;                               // CUDA-core engine: receives sum_k A(m,k), [M] (the bias gradient next to a weight gradient)
  float* a_rownorm = nullptr;                           // tensor-core engine: receives the L2 norm of every row of A (from the split pass)
  // tensor-core engine, several products in one launch: the columns of the result come in segments of n_seg, segment j at C + j c_seg
  // (bias + j bias_seg): X [Wq; Wk; Wv]^T; the contraction runs over segments of k_seg of A's rows, segment j at A + j a_seg:
  // dQ Wq + dK Wk + dV Wv; the rows of a transposed A come in segments of m_seg at A + j a_seg.
  int* zmax = nullptr; int zmax_T = 0;                  // with n_seg: largest magnitudes per sequence and head of the result (TcParams::zmax)
  int n_seg = 0, k_seg = 0, m_seg = 0; long c_seg = 0, bias_seg = 0, a_seg = 0;
  int batch1 = 1, batch2 = 1;                           // batch index b -> (b / batch2, b % batch2)
  const int* z_first = nullptr;                         // tensor-core engine may leave out problem (i, j) where j < z_first[i] (device memory): nothing reads its result
  long a_b1 = 0, a_b2 = 0, b_b1 = 0, b_b2 = 0, c_b1 = 0, c_b2 = 0, r_b1 = 0, r_b2 = 0;
  // Causal structure of attention: tiles that are entirely masked are never touched.
  //   GEMM_SKIP_UPPER : do not compute output tiles with n0 > m0 + BM - 1 (S = Q K^T)
  //   GEMM_KEND_AT_M0 : contraction index stops at m0 + BM            (P V, dS K)
  //   GEMM_KBEG_AT_M0 : contraction index starts at m0                (dS^T Q, P^T dA)
  int flags = 0;
};

// ------------------------------------------------------------------ tiled kernel
// One BM x BN output tile per cluster of `splits` blocks (1, 2, 4 or 8).  The contraction is cut into `splits` equal runs, one
// per block of the cluster; the blocks leave their sums in shared memory, and after a cluster barrier each of them adds up and
// stores its share of the tile's elements, always in rank order, so a result does not depend on scheduling.  This is what
// these products need: they come from small batches and narrow layers (a [64, 784] x [784, 128] forward product, a
// [96, 96] weight gradient over 5000 rows), where a single 128 x 128 tile per block left all but a few SMs idle and one block
// walking the whole contraction -- 72 us for the former and 430 us for the latter, against 7 and 13 us now.
// Global loads of a k-step go to registers while the two before it are multiplied, then to the other shared-memory buffer.
// 16-byte loads along the operand's fast index where base, stride and range allow it.
constexpr int SG_PAD = 4, SG_MAX_SPLITS = 8, SG_RUN = 32;      // runs start at multiples of SG_RUN, whatever the tile
template <int BM, int BN, int BK, int TM, int TN> struct SgCfg {
  static constexpr int THREADS = (BM / TM) * (BN / TN);
  static constexpr int LDA = BM + SG_PAD, LDB = BN + SG_PAD;
  static constexpr int STAGE = BK * (LDA + LDB);
  static constexpr int SMEM_FLOATS = 2 * STAGE > BM * BN ? 2 * STAGE : BM * BN;
};

// A rows x BK slab of an operand: element (r, k) at p[r * s_r + k * s_k], r < nr, k < nk (both relative), zero outside.
// Thread t owns vectors of four: along k (KFAST) or along r.
template <int ROWS, int BK, int THREADS, bool KFAST>
struct SgSlab {
  static constexpr int NV = (ROWS * BK / 4 + THREADS - 1) / THREADS;
  float4 v[NV];
  static constexpr bool EXACT = (ROWS * BK / 4) % THREADS == 0;
  __device__ __forceinline__ static void place(int i, int& r, int& k) {
    if (KFAST) { k = (i % (BK / 4)) * 4; r = i / (BK / 4); } else { r = (i % (ROWS / 4)) * 4; k = i / (ROWS / 4); }
  }
  __device__ __forceinline__ void fetch(const float* __restrict__ p, long s_r, long s_k, int nr, int nk, bool vec) {
#pragma unroll
    for (int q = 0; q < NV; q++) {
      const int i = threadIdx.x + q * THREADS; int r, k; place(i, r, k);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (EXACT || i < ROWS * BK / 4) {
        if (KFAST) {
          const float* s = p + r * s_r + k;
          if (r < nr) {
            if (vec && k + 3 < nk) x = *reinterpret_cast<const float4*>(s);
            else { if (k < nk) x.x = s[0]; if (k + 1 < nk) x.y = s[1]; if (k + 2 < nk) x.z = s[2]; if (k + 3 < nk) x.w = s[3]; }
          }
        } else {
          const float* s = p + r + k * s_k;
          if (k < nk) {
            if (vec && r + 3 < nr) x = *reinterpret_cast<const float4*>(s);
            else { if (r < nr) x.x = s[0]; if (r + 1 < nr) x.y = s[1]; if (r + 2 < nr) x.z = s[2]; if (r + 3 < nr) x.w = s[3]; }
          }
        }
      }
      v[q] = x;
    }
  }
  __device__ __forceinline__ void put(float* __restrict__ sm, int ld) const {      // sm[k][r]
#pragma unroll
    for (int q = 0; q < NV; q++) {
      const int i = threadIdx.x + q * THREADS; int r, k; place(i, r, k);
      if (!EXACT && i >= ROWS * BK / 4) continue;
      if (KFAST) { sm[k * ld + r] = v[q].x; sm[(k + 1) * ld + r] = v[q].y; sm[(k + 2) * ld + r] = v[q].z; sm[(k + 3) * ld + r] = v[q].w; }
      else *reinterpret_cast<float4*>(sm + k * ld + r) = v[q];
    }
  }
};

__device__ __forceinline__ float sg_finish(const GemmDesc& g, const float* R, int m, int n, float acc) {
  float v = g.alpha * acc;
  if (g.bias) v += g.bias[n];
  if (R) v += R[m * g.ldr + n];
  if (g.act == GN_ACT_RELU) v = v > 0.f ? v : 0.f;
  if (g.mask && !(g.mask[(long)(m / g.mask_group) * g.mask_ld + n] > 0.f)) v = 0.f;
  return v;
}

template <int BM, int BN, int BK, int TM, int TN, bool A_KFAST, bool B_NFAST>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(const GemmDesc g, int splits, int vec_a, int vec_b, int y0) {
  using Cfg = SgCfg<BM, BN, BK, TM, TN>;
  constexpr int THREADS = Cfg::THREADS, LDA = Cfg::LDA, LDB = Cfg::LDB, CX = BN / TN;
  __shared__ __align__(16) float sm[Cfg::SMEM_FLOATS];
  __shared__ float asum_sh[BM];
  const int b = blockIdx.z, b1 = b / g.batch2, b2 = b % g.batch2, rank = blockIdx.x % splits, nt = blockIdx.x / splits;
  const float* A = g.A + b1 * g.a_b1 + b2 * g.a_b2;
  const float* B = g.B + b1 * g.b_b1 + b2 * g.b_b2;
  float* C = g.C + b1 * g.c_b1 + b2 * g.c_b2;
  const float* R = g.R ? g.R + b1 * g.r_b1 + b2 * g.r_b2 : nullptr;
  const int m0 = (y0 + blockIdx.y) * BM, n0 = nt * BN;
  if ((g.flags & GEMM_SKIP_UPPER) && n0 > m0 + BM - 1) return;             // (the whole cluster returns)
  int kbeg = 0, kend = g.K;
  if (g.flags & GEMM_KBEG_AT_M0) kbeg = (m0 / BK) * BK;
  if (g.flags & GEMM_KEND_AT_M0) kend = min(g.K, m0 + BM);
  if (splits > 1) {
    const int per = (((kend - kbeg + splits - 1) / splits + SG_RUN - 1) / SG_RUN) * SG_RUN;
    kbeg = min(kend, kbeg + rank * per); kend = min(kend, kbeg + per);
  }
  const int t = threadIdx.x, ty = t / CX, tx = t % CX;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
  const bool want_asum = g.a_sum != nullptr && nt == 0;
  float asum = 0.f;

  // two register sets: the loads of a k-step are issued two steps ahead (the products are short chains of steps, each of which
  // would otherwise wait for most of a memory latency)
  struct Step { SgSlab<BM, BK, THREADS, A_KFAST> a; SgSlab<BN, BK, THREADS, !B_NFAST> b; };
  Step s0, s1; int buf = 0;
  auto fetch = [&](Step& s, int k0) {
    const int nk = kend - k0;
    s.a.fetch(A + (long)m0 * g.sa_m + (long)k0 * g.sa_k, g.sa_m, g.sa_k, g.M - m0, nk, vec_a);
    s.b.fetch(B + (long)n0 * g.sb_n + (long)k0 * g.sb_k, g.sb_n, g.sb_k, g.N - n0, nk, vec_b);
  };
  auto step = [&](Step& next, Step& after, int k0) {          // `next` holds k-step k0 + BK
    if (k0 + 2 * BK < kend) fetch(after, k0 + 2 * BK);
    const float* As = sm + buf * Cfg::STAGE; const float* Bs = As + BK * LDA;
#pragma unroll
    for (int k = 0; k < BK; k++) {
      float av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; i++) av[i] = As[k * LDA + ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; j++) bv[j] = Bs[k * LDB + tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (want_asum && t < BM) {
#pragma unroll
      for (int k = 0; k < BK; k++) asum += As[k * LDA + t];
    }
    buf ^= 1;
    if (k0 + BK < kend) { float* nx = sm + buf * Cfg::STAGE; next.a.put(nx, LDA); next.b.put(nx + BK * LDA, LDB); }
    __syncthreads();
  };
  if (kbeg < kend) {
    fetch(s0, kbeg);
    if (kbeg + BK < kend) fetch(s1, kbeg + BK);
    s0.a.put(sm, LDA); s0.b.put(sm + BK * LDA, LDB);
    __syncthreads();
    for (int k0 = kbeg; k0 < kend; k0 += 2 * BK) {
      step(s1, s0, k0);
      if (k0 + BK < kend) step(s0, s1, k0 + BK);
    }
  }
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < TM; i++) {
      const int m = m0 + ty * TM + i;
      if (m >= g.M) continue;
#pragma unroll
      for (int j = 0; j < TN; j++) { const int n = n0 + tx * TN + j; if (n < g.N) C[m * g.ldc + n] = sg_finish(g, R, m, n, acc[i][j]); }
    }
    if (want_asum && t < BM && m0 + t < g.M) g.a_sum[m0 + t] = asum;
    return;
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) sm[(ty * TM + i) * BN + tx * TN + j] = acc[i][j];
  if (want_asum && t < BM) asum_sh[t] = asum;
  cluster.sync();
  const int share = BM * BN / splits;
  for (int e = rank * share + t; e < (rank + 1) * share; e += THREADS) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= g.M || n >= g.N) continue;
    float v = 0.f;
    for (int q = 0; q < splits; q++) v += cluster.map_shared_rank(sm, q)[e];
    C[m * g.ldc + n] = sg_finish(g, R, m, n, v);
  }
  if (want_asum && rank == 0 && t < BM && m0 + t < g.M) {
    float v = 0.f;
    for (int q = 0; q < splits; q++) v += cluster.map_shared_rank(asum_sh, q)[t];
    g.a_sum[m0 + t] = v;
  }
  cluster.sync();                                             // nobody leaves while its sums are being read
}

// Skinny outputs (N <= 16, both operands K-major, one problem): a tile would be mostly padding.  A cluster of `splits`
// blocks owns one output row: their threads stride over K with all N sums in registers, combine through shared memory, and
// rank 0 adds the blocks' sums in rank order.  C(m,n) = act(sum_k A(m,k) B(n,k) + bias[n] + R(m,n)).  One block per row (K = 4704,
// N = 10: 18 loads deep) took 18 us for 50 rows; eight take 7.
constexpr int SKINNY_N = 16;
__global__ void __launch_bounds__(256) gemm_skinny_kernel(const GemmDesc g, int splits) {
  __shared__ float red[8][SKINNY_N];
  __shared__ float tot[SKINNY_N];
  const int m = blockIdx.x / splits, rank = blockIdx.x % splits, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float* a = g.A + (long)m * g.sa_m;
  float acc[SKINNY_N];
#pragma unroll
  for (int n = 0; n < SKINNY_N; n++) acc[n] = 0.f;
  for (int k = rank * 256 + threadIdx.x; k < g.K; k += 256 * splits) {
    const float av = a[k];
#pragma unroll
    for (int n = 0; n < SKINNY_N; n++) if (n < g.N) acc[n] = fmaf(av, g.B[(long)n * g.sb_n + k], acc[n]);
  }
#pragma unroll
  for (int n = 0; n < SKINNY_N; n++) { if (n < g.N) { const float v = warp_sum(acc[n]); if (lane == 0) red[w][n] = v; } }
  __syncthreads();
  if (threadIdx.x < g.N) {
    float v = 0.f;
    for (int q = 0; q < 8; q++) v += red[q][threadIdx.x];
    tot[threadIdx.x] = v;
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (splits > 1) cluster.sync(); else __syncthreads();
  if (rank == 0 && threadIdx.x < g.N) {
    const int n = threadIdx.x;
    float v = 0.f;
    for (int q = 0; q < splits; q++) v += splits > 1 ? cluster.map_shared_rank(tot, q)[n] : tot[n];
    g.C[(long)m * g.ldc + n] = sg_finish(g, g.R, m, n, v);
  }
  if (splits > 1) cluster.sync();
}
inline bool gemm_skinny_ok(const GemmDesc& g) {
  return g.batch1 * g.batch2 == 1 && g.N <= SKINNY_N && g.K >= 128 && g.sa_k == 1 && g.sb_k == 1 && g.alpha == 1.f && g.flags == 0 && !g.a_sum;
}

// Sum of at most 64 outer products: C[M,N] = sum_k A(m,k) B(k,n) with both operands stored contraction-major (A(m,k) at
// A[k * sa_k + m], B(k,n) at B[k * sb_k + n]) -- the weight gradient of an inner Dense layer, which only sees one input
// row per sample (layer.go:591-625), when the batch (or a rank's shard of it) is small.  Every block stages both operand
// panels of its 16 TM x 64 output tile in shared memory once (16 bytes per asynchronous copy where the alignment allows it); each
// thread owns a TM x 4 patch.  The general kernel runs such a product on few blocks with a contraction of four 16-steps; this one
// fills the SMs.  TM = 8 halves the shared-memory reads per multiply-add and the panel traffic: for outputs with enough tiles of that
// size.  blockIdx.z: several products of one shape, their C (and a_sum) c_b apart (the Q, K and V projections' gradients).
constexpr int OS_KMAX = 64;
template <int TM>
__global__ void __launch_bounds__(256) outer_sum_kernel(const float* __restrict__ A, long sa_k, long a_b, const float* __restrict__ B, long sb_k, long b_b, float* __restrict__ C, long ldc, long c_b,
                                                        int M, int N, int K, float alpha, float* __restrict__ a_sum, int va, int vb) {
  constexpr int BM = 16 * TM;
  __shared__ __align__(16) float As[OS_KMAX][BM];
  __shared__ __align__(16) float Bs[OS_KMAX][64];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * 64, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  A += blockIdx.z * a_b; B += blockIdx.z * b_b; C += blockIdx.z * c_b;
  if (va && m0 + BM <= M) for (int i = tid; i < K * (BM / 4); i += 256) { const int k = i / (BM / 4), c = i % (BM / 4) * 4; cp_async16(&As[k][c], A + (long)k * sa_k + m0 + c); }
  else
#pragma unroll 4
    for (int i = tid; i < K * BM; i += 256) { const int k = i / BM, c = i % BM; As[k][c] = m0 + c < M ? A[(long)k * sa_k + m0 + c] : 0.f; }
  if (vb && n0 + 64 <= N) for (int i = tid; i < K * 16; i += 256) { const int k = i >> 4, c = (i & 15) * 4; cp_async16(&Bs[k][c], B + (long)k * sb_k + n0 + c); }
  else
#pragma unroll 4
    for (int i = tid; i < K * 64; i += 256) { const int k = i >> 6, c = i & 63; Bs[k][c] = n0 + c < N ? B[(long)k * sb_k + n0 + c] : 0.f; }
  cp_async_wait();
  __syncthreads();
  if (a_sum && blockIdx.x == 0 && tid < BM && m0 + tid < M) { float v = 0.f; for (int k = 0; k < K; k++) v += As[k][tid]; a_sum[blockIdx.z * c_b + m0 + tid] = v; }
  float acc[TM][4] = {};
#pragma unroll 4
  for (int k = 0; k < K; k++) {
    const float4 b = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]); const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int h = 0; h < TM / 4; h++) {
      const float4 a = *reinterpret_cast<const float4*>(&As[k][h * 64 + ty * 4]); const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[4 * h + i][j] = fmaf(av[i], bv[j], acc[4 * h + i][j]);
    }
  }
  const bool vec = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && n0 + tx * 4 + 3 < N;
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int m = m0 + (i >> 2) * 64 + ty * 4 + (i & 3); if (m >= M) continue;
    float* crow = C + (long)m * ldc + n0 + tx * 4;
    if (vec) *reinterpret_cast<float4*>(crow) = make_float4(alpha * acc[i][0], alpha * acc[i][1], alpha * acc[i][2], alpha * acc[i][3]);
    else
      for (int j = 0; j < 4; j++) if (n0 + tx * 4 + j < N) crow[j] = alpha * acc[i][j];
  }
}
inline bool gemm_outer_small_ok(const GemmDesc& g) {
  return g.sa_m == 1 && g.sb_n == 1 && g.K >= 1 && g.K <= OS_KMAX && g.batch2 == 1 && g.batch1 <= 65535 && !g.bias && !g.R && !g.mask && g.act == GN_ACT_LINEAR && g.flags == 0 &&
         !g.a_planes && !g.b_planes && !g.plane_out && !g.a_rownorm && !g.m_seg && (long)g.M * g.N >= 64 * 64;
}

template <int BM, int BN, int BK, int TM, int TN>
inline int gemm_simt_tile(Ctx* ctx, const GemmDesc& g, int splits) {
  auto vec = [](const float* p, long ld, long b1, long b2) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0 && b1 % 4 == 0 && b2 % 4 == 0; };
  const bool ak = g.sa_k == 1, bn = g.sb_n == 1;
  const int va = (ak || g.sa_m == 1) && vec(g.A, ak ? g.sa_m : g.sa_k, g.a_b1, g.a_b2), vb = (bn || g.sb_k == 1) && vec(g.B, bn ? g.sb_k : g.sb_n, g.b_b1, g.b_b2);
  const int tiles_m = cdiv(g.M, BM); constexpr int THREADS = SgCfg<BM, BN, BK, TM, TN>::THREADS;
  for (int y0 = 0; y0 < tiles_m; y0 += 65535) {             // (a grid's second dimension)
    const dim3 grid(cdiv(g.N, BN) * splits, std::min(tiles_m - y0, 65535), g.batch1 * g.batch2);
    if (ak && bn) GN_CLUSTER_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, true, true>), grid, THREADS, 0, splits, g, splits, va, vb, y0);
    else if (ak && g.sb_k == 1) GN_CLUSTER_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, true, false>), grid, THREADS, 0, splits, g, splits, va, vb, y0);
    else if (g.sa_m == 1 && bn) GN_CLUSTER_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, false, true>), grid, THREADS, 0, splits, g, splits, va, vb, y0);
    else if (g.sa_m == 1 && g.sb_k == 1) GN_CLUSTER_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, false, false>), grid, THREADS, 0, splits, g, splits, va, vb, y0);
    else return fail(GN_ERR_UNSUPPORTED, "gemm_simt: neither stride of an operand is 1");
  }
  return check_launch("gemm_simt");
}
// Blocks per output tile.  A run shorter than 64 is not worth a block.  Where the rows of A are samples (or tokens), the
// number does not depend on how many there are: a sample's result is the same in every batch.
inline int gemm_simt_splits(const GemmDesc& g, int sm_count, long tiles_all, long tiles_n) {
  const long have = g.sa_k == 1 ? tiles_n : tiles_all;
  int s = 1;
  while (s < SG_MAX_SPLITS && g.K >= 128 * s && have * s < sm_count) s *= 2;
  return s;
}
inline int gemm_simt(Ctx* ctx, const GemmDesc& g) {
  if (g.M <= 0 || g.N <= 0) return GN_OK;
  if (gemm_outer_small_ok(g)) {
    auto vec = [](const float* p, long ld, long bs) { return (int)((reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0 && bs % 4 == 0); };
    const int va = vec(g.A, g.sa_k, g.a_b1), vb = vec(g.B, g.sb_k, g.b_b1);
    // 128-row tiles once they give every SM two blocks
    if ((long)cdiv(g.N, 64) * cdiv(g.M, 128) * g.batch1 >= 2 * ctx->sm_count)
      GN_LAUNCH(ctx, outer_sum_kernel<8>, dim3(cdiv(g.N, 64), cdiv(g.M, 128), g.batch1), 256, 0, g.A, g.sa_k, g.a_b1, g.B, g.sb_k, g.b_b1, g.C, g.ldc, g.c_b1, g.M, g.N, g.K, g.alpha, g.a_sum, va, vb);
    else GN_LAUNCH(ctx, outer_sum_kernel<4>, dim3(cdiv(g.N, 64), cdiv(g.M, 64), g.batch1), 256, 0, g.A, g.sa_k, g.a_b1, g.B, g.sb_k, g.b_b1, g.C, g.ldc, g.c_b1, g.M, g.N, g.K, g.alpha, g.a_sum, va, vb);
    return check_launch("outer_sum");
  }
  if (gemm_skinny_ok(g)) {
    int s = 1; while (s < SG_MAX_SPLITS && g.K >= 512 * s) s *= 2;
    GN_CLUSTER_LAUNCH(ctx, gemm_skinny_kernel, dim3(g.M * s), 256, 0, s, g, s); return check_launch("gemm_skinny");
  }
  const long nb = (long)g.batch1 * g.batch2, t64 = (long)cdiv(g.M, 64) * cdiv(g.N, 64) * nb;
  const int s = gemm_simt_splits(g, ctx->sm_count, t64, (long)cdiv(g.N, 64));
  // 16-row tiles for a handful of rows; 32 x 32 tiles (a quarter of the work per block) when 64 x 64 would not give every SM one or
  // be half empty
  if (g.M <= 16) return gemm_simt_tile<16, 64, 32, 2, 4>(ctx, g, s);
  if (g.M <= 32 || t64 * s < ctx->sm_count) return gemm_simt_tile<32, 32, 32, 4, 2>(ctx, g, s);
  return gemm_simt_tile<64, 64, 16, 4, 4>(ctx, g, s);
}

}  // namespace gn
