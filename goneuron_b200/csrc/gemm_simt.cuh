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
// One BM x BN output tile per block.  Global loads of a k-step go to registers while the two before it are multiplied, then to the
// other shared-memory buffer.  16-byte loads along the operand's fast index where base, stride and range allow it.
constexpr int SG_PAD = 4;
template <int BM, int BN, int BK, int TM, int TN> struct SgCfg {
  static constexpr int THREADS = (BM / TM) * (BN / TN);
  static constexpr int LDA = BM + SG_PAD, LDB = BN + SG_PAD;
  static constexpr int STAGE = BK * (LDA + LDB);
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
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(const GemmDesc g, int vec_a, int vec_b, int y0) {
  using Cfg = SgCfg<BM, BN, BK, TM, TN>;
  constexpr int THREADS = Cfg::THREADS, LDA = Cfg::LDA, LDB = Cfg::LDB, CX = BN / TN;
  __shared__ __align__(16) float sm[2 * Cfg::STAGE];
  const int b = blockIdx.z, b1 = b / g.batch2, b2 = b % g.batch2, nt = blockIdx.x;
  const float* A = g.A + b1 * g.a_b1 + b2 * g.a_b2;
  const float* B = g.B + b1 * g.b_b1 + b2 * g.b_b2;
  float* C = g.C + b1 * g.c_b1 + b2 * g.c_b2;
  const float* R = g.R ? g.R + b1 * g.r_b1 + b2 * g.r_b2 : nullptr;
  const int m0 = (y0 + blockIdx.y) * BM, n0 = nt * BN;
  if ((g.flags & GEMM_SKIP_UPPER) && n0 > m0 + BM - 1) return;
  int kbeg = 0, kend = g.K;
  if (g.flags & GEMM_KBEG_AT_M0) kbeg = (m0 / BK) * BK;
  if (g.flags & GEMM_KEND_AT_M0) kend = min(g.K, m0 + BM);
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
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int m = m0 + ty * TM + i;
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; j++) { const int n = n0 + tx * TN + j; if (n < g.N) C[m * g.ldc + n] = sg_finish(g, R, m, n, acc[i][j]); }
  }
  if (want_asum && t < BM && m0 + t < g.M) g.a_sum[m0 + t] = asum;
}

// Skinny outputs (N <= 16, both operands K-major, one problem): a tile would be mostly padding.  A cluster of `splits`
// blocks owns RPB output rows: their threads stride over K with all N sums of each row in registers, combine through shared memory, and
// rank 0 adds the blocks' sums in rank order.  C(m,n) = act(sum_k A(m,k) B(n,k) + bias[n] + R(m,n)).  One block per row (K = 4704,
// N = 10: 18 loads deep) took 18 us for 50 rows; eight take 6.  Bound by what is fetched of B, once per block: four rows share it where there are
// enough (128 rows, K = 2048, N = 10: 8.5 -> 5.4 us; 300 rows, K = 128: 3.1 either way; 1000: 5.5 -> 4.0).
constexpr int SKINNY_N = 16;
template <int RPB>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(const GemmDesc g, int splits) {
  __shared__ float red[8][RPB][SKINNY_N];
  __shared__ float tot[RPB][SKINNY_N];
  const int m0 = blockIdx.x / splits * RPB, rank = blockIdx.x % splits, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float* a[RPB]; float acc[RPB][SKINNY_N];
#pragma unroll
  for (int r = 0; r < RPB; r++) {
    a[r] = g.A + (long)(RPB == 1 ? m0 : min(m0 + r, g.M - 1)) * g.sa_m;        // (a row beyond the last is the last one again, and not stored)
#pragma unroll
    for (int n = 0; n < SKINNY_N; n++) acc[r][n] = 0.f;
  }
  for (int k = rank * 256 + threadIdx.x; k < g.K; k += 256 * splits) {
    float av[RPB];
#pragma unroll
    for (int r = 0; r < RPB; r++) av[r] = a[r][k];
#pragma unroll
    for (int n = 0; n < SKINNY_N; n++) if (n < g.N) {
      const float bv = g.B[(long)n * g.sb_n + k];
#pragma unroll
      for (int r = 0; r < RPB; r++) acc[r][n] = fmaf(av[r], bv, acc[r][n]);
    }
  }
#pragma unroll
  for (int n = 0; n < SKINNY_N; n++) if (n < g.N) {
#pragma unroll
    for (int r = 0; r < RPB; r++) { const float v = warp_sum(acc[r][n]); if (lane == 0) red[w][r][n] = v; }
  }
  __syncthreads();
  const int r = threadIdx.x / SKINNY_N, n = threadIdx.x % SKINNY_N; const bool mine = r < RPB && n < g.N;
  if (mine) {
    float v = 0.f;
    for (int q = 0; q < 8; q++) v += red[q][r][n];
    tot[r][n] = v;
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (splits > 1) cluster.sync(); else __syncthreads();
  if (rank == 0 && mine && m0 + r < g.M) {
    float v = 0.f;
    for (int q = 0; q < splits; q++) v += splits > 1 ? cluster.map_shared_rank(&tot[0][0], q)[r * SKINNY_N + n] : tot[r][n];
    g.C[(long)(m0 + r) * g.ldc + n] = sg_finish(g, g.R, m0 + r, n, v);
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
__device__ __forceinline__ void outer_tile(const float* __restrict__ A, long sa_k, const float* __restrict__ B, long sb_k, float* __restrict__ C, long ldc, int M, int N, int K, float alpha,
                                           float* __restrict__ a_sum, int va, int vb, int m0, int n0) {
  constexpr int BM = 16 * TM;
  __shared__ __align__(16) float As[OS_KMAX][BM];
  __shared__ __align__(16) float Bs[OS_KMAX][64];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
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
  if (a_sum && n0 == 0 && tid < BM && m0 + tid < M) { float v = 0.f; for (int k = 0; k < K; k++) v += As[k][tid]; a_sum[m0 + tid] = v; }
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
template <int TM>
__global__ void __launch_bounds__(256) outer_sum_kernel(const float* __restrict__ A, long sa_k, long a_b, const float* __restrict__ B, long sb_k, long b_b, float* __restrict__ C, long ldc, long c_b,
                                                        int M, int N, int K, float alpha, float* __restrict__ a_sum, int va, int vb) {
  outer_tile<TM>(A + blockIdx.z * a_b, sa_k, B + blockIdx.z * b_b, sb_k, C + blockIdx.z * c_b, ldc, M, N, K, alpha, a_sum ? a_sum + blockIdx.z * c_b : nullptr, va, vb, blockIdx.y * 16 * TM, blockIdx.x * 64);
}
// Several such sums over the same number of rows in one launch, a tile per block: a launch of a few dozen tiles takes as long as one of 160, and
// a block's four gradients one after the other took as long as the rest of its backward pass beside them.
struct OuterGroup {
  struct P { const float *A, *B; float *C, *a_sum; long sa_k, sb_k, ldc; int M, N, va, vb, tile0; } p[4];
  int n = 0, K = 0;
};
template <int TM>
__global__ void __launch_bounds__(256) outer_group_kernel(const OuterGroup g) {
  int j = 0;
  while (j + 1 < g.n && (int)blockIdx.x >= g.p[j + 1].tile0) j++;
  const OuterGroup::P& q = g.p[j]; const int t = blockIdx.x - q.tile0, tn = (q.N + 63) / 64;
  outer_tile<TM>(q.A, q.sa_k, q.B, q.sb_k, q.C, q.ldc, q.M, q.N, g.K, 1.f, q.a_sum, q.va, q.vb, t / tn * 16 * TM, t % tn * 64);
}
inline bool gemm_outer_small_ok(const GemmDesc& g) {
  return g.sa_m == 1 && g.sb_n == 1 && g.K >= 1 && g.K <= OS_KMAX && g.batch2 == 1 && g.batch1 <= 65535 && !g.bias && !g.R && !g.mask && g.act == GN_ACT_LINEAR && g.flags == 0 &&
         !g.a_planes && !g.b_planes && !g.plane_out && !g.a_rownorm && !g.m_seg && (long)g.M * g.N >= 64 * 64;
}

// ------------------------------------------------------------------ small products
// Products whose 64 x 64 tiles leave most SMs idle: the few rows of a head, of a block's token rows or of a small batch, weight gradients of narrow
// layers.  They are bound by latency (64 rows by a [256, 256] matrix are 0.2 us of multiply-adds), so a block has as much in flight and as
// few dependent steps as possible.  A cluster of up to eight blocks owns a tile of 4 TM rows by 32 columns, each with a run of the
// contraction; a block asks for up to three stages of 64 indices ahead (asynchronous copies of 16 bytes in the operands' own order); each of its
// eight warps multiplies eight indices of every stage for the whole tile, TM x 4 outputs per lane; the warps' sums meet in shared
// memory; and a block's sums are written straight to the blocks of the cluster that own them: one exchange, after which nobody reads
// from anybody else.
// Order of an output's sum: the contraction is cut into chunks; within one, a warp's indices ascending, then the warps; the chunks pairwise.
// A block of the cluster takes a power of two of neighbouring chunks, so their number per block (it falls with the number of tiles) does not
// matter, and where the rows of A are samples a sample's result is the same in every batch.
// us per launch in a recorded chain, a 32 x 32 tile in two register-staged steps per run, results read from the other blocks -> this:
//   64 x 256 over 256 4.9 -> 3.7, over 1024 7.5 -> 5.9; 128 x 1024 over 256 7.6 -> 5.8; 1 x 128 over 784 5.6 -> 3.5; 8 x 8192 over 512 13.3 -> 7.4;
//   16 x 512 over 8192 25.7 -> 14.7; a 96 x 96 weight gradient over 5000 rows 14.3 -> 9.7.  The same chain of empty launches: 2.2.
constexpr int SP_KB = 64, SP_BN = 32, SP_STAGES = 4, SP_THREADS = 256, SP_MAX_SPLITS = 8;
constexpr int sp_smem(int tm) { return (SP_STAGES * SP_KB * (4 * tm + SP_BN) + 8 * 4 * tm * SP_BN) * (int)sizeof(float); }
// Brings ROWS operand rows x 64 indices into shared memory, stage by stage.  KFAST: [row][64], 16-byte units swizzled by the row's position among
// fours (eight lanes that read one unit of rows four apart find it in different banks); else [64][ROWS].
template <int ROWS, bool KFAST, int THREADS = SP_THREADS>
struct SpLoad {
  static constexpr int NV = ROWS * SP_KB / 4, NQ = (NV + THREADS - 1) / THREADS;
  const float *base, *src[NQ]; long s_r, s_k; int nr; bool vec;
  __device__ __forceinline__ static void place(int q, int& r, int& k) {
    const int e = q * THREADS + threadIdx.x;
    if (KFAST) { r = e >> 4; k = (e & 15) * 4; } else { r = e % (ROWS / 4) * 4; k = e / (ROWS / 4); }
  }
  __device__ __forceinline__ SpLoad(const float* p, long s_r_, long s_k_, int nr_, bool v) : base(p), s_r(s_r_), s_k(s_k_), nr(nr_), vec(v) {
#pragma unroll
    for (int q = 0; q < NQ; q++) { int r, k; place(q, r, k); src[q] = p + (KFAST ? r * s_r + k : r + k * s_k); }
  }
  // nk: indices that are left, this stage included.  PART (a check per copy of it cost the kernel below 2 %): only the first `upto` of the stage are wanted, and rows that 16-byte copies do not fit come by
  // loads and stores, 16 of a thread's at a time, instead of 4-byte asynchronous copies (whole stages waited for at once: 2 to 10 % quicker).
  template <bool PART = false>
  __device__ __forceinline__ void fetch(float* __restrict__ dst, int nk, int upto = SP_KB) {
    if (vec) {
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        int r, k; place(q, r, k);
        if (NV % THREADS != 0 && q * THREADS + (int)threadIdx.x >= NV) break;
        if (PART && k >= upto) continue;
        const int n = KFAST ? (r < nr ? min(max(nk - k, 0), 4) : 0) : (k < nk ? min(max(nr - r, 0), 4) : 0);
        cp_async16_part(dst + (KFAST ? r * SP_KB + (((k >> 2) ^ (r >> 2 & 7)) << 2) : k * ROWS + r), n ? src[q] : base, n);
        src[q] += KFAST ? (long)SP_KB : SP_KB * s_k;
      }
    } else {
      const int r0 = KFAST ? threadIdx.x >> 6 : threadIdx.x % ROWS, k0 = KFAST ? threadIdx.x & 63 : threadIdx.x / ROWS; const float* p = base + r0 * s_r + k0 * s_k;
      constexpr int RSTEP = THREADS / SP_KB, KSTEP = THREADS / ROWS;
      if (PART) {
        constexpr int NF = 16;
        for (int q0 = 0; q0 < ROWS * SP_KB / THREADS; q0 += NF) {
          float x[NF];
#pragma unroll
          for (int j = 0; j < NF; j++) {
            const int r = KFAST ? r0 + RSTEP * (q0 + j) : r0, k = KFAST ? k0 : k0 + KSTEP * (q0 + j);
            x[j] = r < nr && k < nk ? *p : 0.f; p += KFAST ? RSTEP * s_r : KSTEP * s_k;
          }
#pragma unroll
          for (int j = 0; j < NF; j++) {
            const int r = KFAST ? r0 + RSTEP * (q0 + j) : r0, k = KFAST ? k0 : k0 + KSTEP * (q0 + j);
            if (k < upto) dst[KFAST ? r * SP_KB + (((k >> 2) ^ (r >> 2 & 7)) << 2) + (k & 3) : k * ROWS + r] = x[j];
          }
        }
      } else
#pragma unroll
      for (int q = 0; q < ROWS * SP_KB / THREADS; q++) {
        const int r = KFAST ? r0 + RSTEP * q : r0, k = KFAST ? k0 : k0 + KSTEP * q; const bool ok = r < nr && k < nk;
        cp_async4(dst + (KFAST ? r * SP_KB + (((k >> 2) ^ (r >> 2 & 7)) << 2) + (k & 3) : k * ROWS + r), ok ? p : base, ok);
        p += KFAST ? RSTEP * s_r : KSTEP * s_k;
      }
      if (nk > SP_KB) base += SP_KB * s_k;
    }
  }
};
// `splits` blocks per cluster, `chunks` chunks per block, each of `per` indices (a multiple of 64)
template <int TM, bool A_KFAST, bool B_NFAST>
__global__ void __launch_bounds__(SP_THREADS, 2) gemm_small_kernel(const GemmDesc g, int splits, int chunks, int per, int vec_a, int vec_b, int y0) {
  constexpr int BM = 4 * TM, STAGE = SP_KB * (BM + SP_BN), NV = BM * SP_BN / 4;
  extern __shared__ __align__(16) float sm[];                 // ring of stages, A | B; the warps' sums [8][BM][32]
  __shared__ __align__(16) float4 xch[NV];                    // what the cluster's blocks send: [block][share]
  __shared__ float as_sm[8][BM], as_x[SP_MAX_SPLITS][BM];
  const int b = blockIdx.z, b1 = b / g.batch2, b2 = b % g.batch2, rank = blockIdx.x % splits, nt = blockIdx.x / splits;
  const float* A = g.A + b1 * g.a_b1 + b2 * g.a_b2;
  const float* B = g.B + b1 * g.b_b1 + b2 * g.b_b2;
  float* C = g.C + b1 * g.c_b1 + b2 * g.c_b2;
  const float* R = g.R ? g.R + b1 * g.r_b1 + b2 * g.r_b2 : nullptr;
  const int m0 = (y0 + blockIdx.y) * BM, n0 = nt * SP_BN;
  if ((g.flags & GEMM_SKIP_UPPER) && n0 > m0 + BM - 1) return;             // (the whole cluster returns)
  if (splits > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // "running": nobody is written to before
  int kbeg = rank * chunks * per, kend = min(g.K, kbeg + chunks * per);
  if (g.flags & GEMM_KBEG_AT_M0) kbeg = max(kbeg, m0 / SP_KB * SP_KB);
  if (g.flags & GEMM_KEND_AT_M0) kend = min(kend, m0 + BM);
  const int t = threadIdx.x, w = t >> 5, lane = t & 31, mg = lane >> 3, ng = lane & 7, stages = kend > kbeg ? (kend - kbeg + SP_KB - 1) / SP_KB : 0;
  const int k_at = stages ? kbeg : 0;                         // (a block without indices fetches nothing)
  SpLoad<BM, A_KFAST> la(A + (long)m0 * g.sa_m + (long)k_at * g.sa_k, g.sa_m, g.sa_k, g.M - m0, vec_a);
  SpLoad<SP_BN, !B_NFAST> lb(B + (long)n0 * g.sb_n + (long)k_at * g.sb_k, g.sb_n, g.sb_k, g.N - n0, vec_b);
  auto fetch = [&](int s) {
    if (s < stages) { float* d = sm + s % SP_STAGES * STAGE; la.fetch(d, kend - kbeg - s * SP_KB); lb.fetch(d + SP_KB * BM, kend - kbeg - s * SP_KB); }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < SP_STAGES - 1; s++) fetch(s);
  float asum[TM];
#pragma unroll
  for (int i = 0; i < TM; i++) asum[i] = 0.f;
  const bool want_asum = !A_KFAST && g.a_sum != nullptr && nt == 0;
  auto add = [](const float4& a, const float4& x) { return make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w); };
  float4* red = reinterpret_cast<float4*>(sm + SP_STAGES * STAGE);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f); float4 v = zero, s1 = zero, s2 = zero, s4 = zero;      // of this thread's four outputs: the sum, and sums of 1, 2, 4 chunks that wait for their neighbours
  int s = 0;
  for (int c = 0; c < chunks; c++) {
    const int s_end = min(stages, ((rank * chunks + c + 1) * per - kbeg) / SP_KB);
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (; s < s_end; s++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(SP_STAGES - 2) : "memory");
      __syncthreads();
      const float* As = sm + s % SP_STAGES * STAGE; const float* Bs = As + SP_KB * BM;
#pragma unroll
      for (int h = 0; h < 2; h++) {                           // four indices at a time
        const int k = 8 * w + 4 * h; float a[4][TM], bv[4][4];
        if (TM == 8 && h == 0) fetch(s + SP_STAGES - 1);      // into the stage that everybody has left behind
#pragma unroll
        for (int i = 0; i < TM; i += A_KFAST ? 1 : TM < 4 ? TM : 4) {
          if (A_KFAST) {
            const int r = mg * TM + i; const float4 x = *reinterpret_cast<const float4*>(As + r * SP_KB + (((k >> 2) ^ (r >> 2 & 7)) << 2));
            a[0][i] = x.x; a[1][i] = x.y; a[2][i] = x.z; a[3][i] = x.w;
          } else {
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const float* p = As + (k + q) * BM + mg * TM + i;
              if (TM < 4) { const float2 x = *reinterpret_cast<const float2*>(p); a[q][i] = x.x; a[q][i + 1] = x.y; }
              else { const float4 x = *reinterpret_cast<const float4*>(p); a[q][i] = x.x; a[q][(i + 1) % TM] = x.y; a[q][(i + 2) % TM] = x.z; a[q][(i + 3) % TM] = x.w; }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (B_NFAST) {
            const float4 x = *reinterpret_cast<const float4*>(Bs + (k + j) * SP_BN + 4 * ng); bv[j][0] = x.x; bv[j][1] = x.y; bv[j][2] = x.z; bv[j][3] = x.w;
          } else {
            const int r = 4 * ng + j; const float4 x = *reinterpret_cast<const float4*>(Bs + r * SP_KB + (((k >> 2) ^ (r >> 2 & 7)) << 2));
            bv[0][j] = x.x; bv[1][j] = x.y; bv[2][j] = x.z; bv[3][j] = x.w;
          }
        }
        if (TM < 8 && h == 0) fetch(s + SP_STAGES - 1);       // (under the first loads, where the registers allow it)
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[q][i], bv[q][j], acc[i][j]);
        if (want_asum) {
#pragma unroll
          for (int q = 0; q < 4; q++)
#pragma unroll
            for (int i = 0; i < TM; i++) asum[i] += a[q][i];
        }
      }
    }
    if (c > 0) __syncthreads();                               // (the sums of the chunk before have been read)
#pragma unroll
    for (int i = 0; i < TM; i++) red[w * NV + (mg * TM + i) * 8 + ng] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    if (c + 1 == chunks && want_asum && ng == 0) {
#pragma unroll
      for (int i = 0; i < TM; i++) as_sm[w][mg * TM + i] = asum[i];
    }
    __syncthreads();
    if (t < NV) {
      v = red[t];
#pragma unroll
      for (int q = 1; q < 8; q++) v = add(v, red[q * NV + t]);
      if (c & 1) {
        v = add(s1, v);
        if (c & 2) { v = add(s2, v); if (c & 4) v = add(s4, v); else s4 = v; } else s2 = v;
      } else s1 = v;
    }
  }
  float as = 0.f;
  if (want_asum && t < BM) {
#pragma unroll
    for (int q = 0; q < 8; q++) as += as_sm[q][t];
  }
  int at = t; bool mine = t < NV;                             // the four outputs this thread finishes
  if (splits > 1) {
    const int share = NV / splits;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (t < NV) cluster.map_shared_rank(xch, t / share)[rank * share + t % share] = v;
    if (want_asum && t < BM) cluster.map_shared_rank(&as_x[0][0], 0)[rank * BM + t] = as;
    cluster.sync();
    mine = t < share; at = rank * share + t;
    if (mine) {
      v = add(xch[t], xch[share + t]);
      if (splits > 2) v = add(v, add(xch[2 * share + t], xch[3 * share + t]));
      if (splits > 4) v = add(v, add(add(xch[4 * share + t], xch[5 * share + t]), add(xch[6 * share + t], xch[7 * share + t])));
    }
    if (want_asum && rank == 0 && t < BM) { as = 0.f; for (int q = 0; q < splits; q++) as += as_x[q][t]; }
  }
  if (want_asum && rank == 0 && t < BM && m0 + t < g.M) g.a_sum[m0 + t] = as;
  const int m = m0 + (at >> 3), n = n0 + (at & 7) * 4;
  if (!mine || m >= g.M || n >= g.N) return;
  float* c = C + (long)m * g.ldc + n; const float x[4] = {v.x, v.y, v.z, v.w}; float o[4];
#pragma unroll
  for (int j = 0; j < 4; j++) o[j] = n + j < g.N ? sg_finish(g, R, m, n + j, x[j]) : 0.f;
  if (n + 3 < g.N && (reinterpret_cast<uintptr_t>(c) & 15) == 0) *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
  else for (int j = 0; j < 4; j++) if (n + j < g.N) c[j] = o[j];
}
// The same sums, bit for bit, where there are many tiles: 64 x 32 outputs per block, 4 x 4 per thread, a chunk of the contraction (up to RS_MAX_PER indices) in
// shared memory at a time.  The kernel above passes eight partial sums of every output through shared memory and starts anew for each 32 x 32 tile: two
// blocks per SM hide that in one round of blocks, several rounds do not.  Here a thread adds up the eight parts by itself, one after the other (indices
// 0 .. 7 of every stage, then 8 .. 15 of every stage, ...), and keeps the sums of one, two or four chunks (CHUNKS) in registers; further chunks are those of
// the cluster's other blocks, which leave their sums in shared memory and finish a share of the tile each.  Figures at gemm_small.
constexpr int RS_BM = 64, RS_BN = 32, RS_THREADS = RS_BM * RS_BN / 16, RS_STAGE = SP_KB * (RS_BM + RS_BN), RS_MAX_PER = 4 * SP_KB;
template <int CHUNKS, bool B_NFAST>
__global__ void __launch_bounds__(RS_THREADS, 4) gemm_rows_kernel(const GemmDesc g, int splits, int per, int vec_a, int vec_b, int y0) {
  constexpr int TX = RS_BN / 4;
  extern __shared__ __align__(16) float sm[];                 // the stages of a chunk, A | B, laid out as above
  const int b = blockIdx.z, b1 = b / g.batch2, b2 = b % g.batch2, rank = blockIdx.x % splits;
  const float* A = g.A + b1 * g.a_b1 + b2 * g.a_b2;
  const float* B = g.B + b1 * g.b_b1 + b2 * g.b_b2;
  float* C = g.C + b1 * g.c_b1 + b2 * g.c_b2;
  const float* R = g.R ? g.R + b1 * g.r_b1 + b2 * g.r_b2 : nullptr;
  const int m0 = (y0 + blockIdx.y) * RS_BM, n0 = blockIdx.x / splits * RS_BN, tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  if ((g.flags & GEMM_SKIP_UPPER) && n0 > m0 + RS_BM - 1) return;
  const int kbeg = g.flags & GEMM_KBEG_AT_M0 ? m0 : 0, kend = g.flags & GEMM_KEND_AT_M0 ? min(g.K, m0 + RS_BM) : g.K;
  float v[4][4], s1[4][4], s2[4][4];                          // the sum; sums of one and two chunks that wait for their neighbours
#pragma unroll
  for (int c = 0; c < CHUNKS; c++) {
    const int at = (rank * CHUNKS + c) * per, k0 = max(at, kbeg), k1 = min(at + per, kend), stages = k1 > k0 ? (k1 - k0 + SP_KB - 1) / SP_KB : 0, k_at = stages ? k0 : 0;
    if (c > 0) __syncthreads();                               // (the chunk before has been read)
    SpLoad<RS_BM, true, RS_THREADS> la(A + (long)m0 * g.sa_m + k_at, g.sa_m, 1, g.M - m0, vec_a);
    SpLoad<RS_BN, !B_NFAST, RS_THREADS> lb(B + (long)n0 * g.sb_n + (long)k_at * g.sb_k, g.sb_n, g.sb_k, g.N - n0, vec_b);
    for (int s = 0; s < stages; s++) {
      float* d = sm + s * RS_STAGE; const int nk = k1 - k0 - s * SP_KB, upto = min((nk + 7) & ~7, SP_KB);
      la.template fetch<true>(d, nk, upto); lb.template fetch<true>(d + SP_KB * RS_BM, nk, upto);
    }
    cp_async_wait();
    __syncthreads();
#pragma unroll 1
    for (int w = 0; w < 8; w++) {
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
      const int ws = max(0, k1 - k0 - 8 * w + SP_KB - 1) / SP_KB;      // stages that hold indices of this part
      for (int s = 0; s < ws; s++) {
        const float* As = sm + s * RS_STAGE; const float* Bs = As + SP_KB * RS_BM;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int k = 8 * w + 4 * h; float a[4][4], bv[4][4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float4 x = *reinterpret_cast<const float4*>(As + (4 * ty + i) * SP_KB + (((k >> 2) ^ (ty & 7)) << 2));
            a[0][i] = x.x; a[1][i] = x.y; a[2][i] = x.z; a[3][i] = x.w;
          }
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (B_NFAST) {
              const float4 x = *reinterpret_cast<const float4*>(Bs + (k + j) * RS_BN + 4 * tx); bv[j][0] = x.x; bv[j][1] = x.y; bv[j][2] = x.z; bv[j][3] = x.w;
            } else {
              const float4 x = *reinterpret_cast<const float4*>(Bs + (4 * tx + j) * SP_KB + (((k >> 2) ^ tx) << 2));
              bv[0][j] = x.x; bv[1][j] = x.y; bv[2][j] = x.z; bv[3][j] = x.w;
            }
          }
#pragma unroll
          for (int q = 0; q < 4; q++)
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
              for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[q][i], bv[q][j], acc[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) v[i][j] = w == 0 ? acc[i][j] : v[i][j] + acc[i][j];
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (c & 1) { v[i][j] = s1[i][j] + v[i][j]; if (c & 2) v[i][j] = s2[i][j] + v[i][j]; else s2[i][j] = v[i][j]; }
        else s1[i][j] = v[i][j];
      }
  }
  auto store = [&](int m, int n, float x0, float x1, float x2, float x3) {
    if (m >= g.M || n >= g.N) return;
    float* c = C + (long)m * g.ldc + n; const float x[4] = {x0, x1, x2, x3}; float o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = n + j < g.N ? sg_finish(g, R, m, n + j, x[j]) : 0.f;
    if (n + 3 < g.N && (reinterpret_cast<uintptr_t>(c) & 15) == 0) *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
    else {
#pragma unroll
      for (int j = 0; j < 4; j++) if (n + j < g.N) c[j] = o[j];
    }
  };
  if (splits > 1) {                                            // the blocks' sums, pairwise; every block finishes a share of the tile
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    float4* xch = reinterpret_cast<float4*>(sm);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) xch[(4 * ty + i) * TX + tx] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
    cluster.sync();
    const int share = RS_BM * TX / splits;
    for (int e = rank * share + threadIdx.x; e < (rank + 1) * share; e += RS_THREADS) {
      auto add = [](const float4& a, const float4& x) { return make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w); };
      auto pair = [&](int q) { return add(cluster.map_shared_rank(xch, q)[e], cluster.map_shared_rank(xch, q + 1)[e]); };
      float4 x = pair(0);
      if (splits > 2) x = add(x, pair(2));
      if (splits > 4) { const float4 y = pair(4); x = add(x, add(y, pair(6))); }
      store(m0 + e / TX, n0 + e % TX * 4, x.x, x.y, x.z, x.w);
    }
    cluster.sync();                                            // nobody leaves while its sums are being read
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; i++) store(m0 + 4 * ty + i, n0 + 4 * tx, v[i][0], v[i][1], v[i][2], v[i][3]);
}
inline bool sg_vec(const float* p, long ld, long b1, long b2) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0 && b1 % 4 == 0 && b2 % 4 == 0; }
inline int gemm_rows(Ctx* ctx, const GemmDesc& g, int splits, int chunks, int per) {
  const bool bn = g.sb_n == 1; if (!bn && g.sb_k != 1) return fail(GN_ERR_UNSUPPORTED, "gemm_rows: neither stride of an operand is 1");
  const int va = sg_vec(g.A, g.sa_m, g.a_b1, g.a_b2), vb = sg_vec(g.B, bn ? g.sb_k : g.sb_n, g.b_b1, g.b_b2), tiles_m = cdiv(g.M, RS_BM), smem = per / SP_KB * RS_STAGE * (int)sizeof(float);
  for (int y0 = 0; y0 < tiles_m; y0 += 65535) {
    const dim3 grid(cdiv(g.N, RS_BN) * splits, std::min(tiles_m - y0, 65535), g.batch1 * g.batch2);
    auto run = [&](auto* K) -> int {
      GN_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (splits > 1) GN_CLUSTER_LAUNCH(ctx, K, grid, RS_THREADS, smem, splits, g, splits, per, va, vb, y0);
      else GN_LAUNCH(ctx, K, grid, RS_THREADS, smem, g, splits, per, va, vb, y0);
      return GN_OK;
    };
    if (bn) GN_TRY(chunks == 1 ? run(gemm_rows_kernel<1, true>) : chunks == 2 ? run(gemm_rows_kernel<2, true>) : run(gemm_rows_kernel<4, true>));
    else GN_TRY(chunks == 1 ? run(gemm_rows_kernel<1, false>) : chunks == 2 ? run(gemm_rows_kernel<2, false>) : run(gemm_rows_kernel<4, false>));
  }
  return check_launch("gemm_rows");
}
template <int TM>
inline int gemm_small_tile(Ctx* ctx, const GemmDesc& g, int splits, int chunks, int per) {
  const bool ak = g.sa_k == 1 && !g.a_sum, bn = g.sb_n == 1;      // (the sums of A's rows come with the other layout; one row has both)
  const int va = (ak || g.sa_m == 1) && sg_vec(g.A, ak ? g.sa_m : g.sa_k, g.a_b1, g.a_b2), vb = (bn || g.sb_k == 1) && sg_vec(g.B, bn ? g.sb_k : g.sb_n, g.b_b1, g.b_b2);
  const int tiles_m = cdiv(g.M, 4 * TM), smem = sp_smem(TM);
  for (int y0 = 0; y0 < tiles_m; y0 += 65535) {             // (a grid's second dimension)
    const dim3 grid(cdiv(g.N, SP_BN) * splits, std::min(tiles_m - y0, 65535), g.batch1 * g.batch2);
    auto run = [&](auto* K) -> int {
      GN_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      GN_CLUSTER_LAUNCH(ctx, K, grid, SP_THREADS, smem, splits, g, splits, chunks, per, va, vb, y0); return GN_OK;
    };
    if (ak && bn) GN_TRY(run(gemm_small_kernel<TM, true, true>));
    else if (ak && g.sb_k == 1) GN_TRY(run(gemm_small_kernel<TM, true, false>));
    else if (g.sa_m == 1 && bn) GN_TRY(run(gemm_small_kernel<TM, false, true>));
    else if (g.sa_m == 1 && g.sb_k == 1) GN_TRY(run(gemm_small_kernel<TM, false, false>));
    else return fail(GN_ERR_UNSUPPORTED, "gemm_small: neither stride of an operand is 1");
  }
  return check_launch("gemm_small");
}
// How many chunks, over how many blocks they go, and which kernel.  A chunk shorter than 64 indices (96 where a sample has more than 256 outputs) is not worth
// its own sum; the number of chunks goes by the matrix alone where the rows of A are samples (or tokens), see above: few enough for five eighths of the SMs, or
// for all of them with runs of 384 indices, and seven tenths of them have to have indices (640 in eight chunks of whole stages would be five of 128).
// The rest changes no bit.  Weight gradients and 16 rows or fewer: blocks by the same measure.  Else by estimated time, from measurements of 1900 shapes between
// 17 and 16 384 rows (us; 5 and 10 % off).  gemm_small_kernel: 1.4, and for every round of two blocks per SM 1.65 times what a block alone takes, 0.57 + 0.73 per stage
// of 64 indices + 0.45 per chunk + 0.45 for an exchange.  gemm_rows_kernel: 2.6, and 1.38 per 64 indices + 1.25 per chunk, 0.55 more of that for each further block
// on the SM; 1.15 times as much where 16-byte copies do not fit.  us, 32 x 32 tiles -> 64 x 32: 4096 x 200 over 72 15.3 -> 9.7, 16 384 x 40 over 64 11.8 -> 8.7, 3000 x 300
// over 64 11.5 -> 8.6, 500 x 1500 over 130 20.7 -> 14.5, 1024 x 200 over 256 10.4 -> 9.3, 511 x 300 over 500 15.5 -> 11.3; the other way 256 x 600 over 80 5.1 -> 6.0, 1024 x 100 over
// 192 5.1 -> 6.1.  Chunks, geometric mean of the time of 1900 smaller shapes against these lines: half, three quarters, all of the
// SMs 1.000, 1.002, 1.003; runs of 256, 768 instead of 384 1.001, 1.000; chunks of 64, 128 instead of 96 1.002, 0.999, of 96, 128 instead of 64 1.015, 1.027.
// Still slower than one pass over 64 x 64 tiles (whose order of sums is another one): more than 1000 tiles over 64 to 96 indices, 16 384 x 40 over 64 8.7 against 7.4, and rows
// that 16-byte copies do not fit, 777 x 1500 over 65 17.0 against 12.5.
inline int gemm_small(Ctx* ctx, const GemmDesc& g) {
  const int tm = g.M <= 8 ? 2 : g.M <= 16 ? 4 : 8; const bool rows = g.sa_k == 1;
  const long nb = (long)g.batch1 * g.batch2, tn = cdiv(g.N, SP_BN), tiles = tn * cdiv(g.M, 4 * tm) * nb; const int run = rows && tn > 8 ? 96 : 64, sms = ctx->sm_count;
  auto more = [&](long blocks, int n) { return blocks * n < 5L * sms / 8 || (blocks * n <= sms && g.K >= 384 * n); };
  auto length = [&](int n) { return (int)cdiv(cdiv(g.K, n), SP_KB) * SP_KB; };
  int all = 1, splits = 1; bool big = false;
  while (all < SP_MAX_SPLITS && g.K >= 2 * run * all && more(rows ? tn : tiles, all) && 10 * cdiv(g.K, length(2 * all)) >= 14u * all) all *= 2;
  const int per = length(all);
  if (tm < 8 || !rows) { while (splits < all && more(tiles, splits)) splits *= 2; }
  else {
    const bool bn = g.sb_n == 1, can = !g.a_sum && per <= RS_MAX_PER;
    const double odd = sg_vec(g.A, g.sa_m, g.a_b1, g.a_b2) && sg_vec(g.B, bn ? g.sb_k : g.sb_n, g.b_b1, g.b_b2) ? 1.0 : 1.15; double best = 1e30;
    for (int s = 1; s <= all; s *= 2) {
      const int chunks = all / s, len = std::min(g.K, chunks * per);
      const long rest = (tiles * s - 1) % (2L * sms) + 1, full = (tiles * s - rest) / (2L * sms);
      const double one = 0.57 + 0.73 * cdiv(len, SP_KB) + 0.45 * chunks + (s > 1 ? 0.45 : 0.0), t = 1.4 + one * (1.65 * full + (rest > sms ? 1.65 : 1.0));
      if (t < best) { best = t; splits = s; big = false; }
      if (!can || chunks > 4) continue;
      const double fit = std::min(4L, 227L * 1024 / (per / SP_KB * RS_STAGE * 4 + 1024)), q = (double)(tn * cdiv(g.M, RS_BM) * nb * s) / sms, work = 1.38 * len / SP_KB + 1.25 * chunks;
      const double u = odd * (2.6 + work * (q <= fit ? 1.0 + 0.55 * (std::ceil(q) - 1.0) : (1.0 + 0.55 * (fit - 1.0)) * q / fit));
      if (u < best) { best = u; splits = s; big = true; }
    }
  }
  const int chunks = all / splits;
  if (big) return gemm_rows(ctx, g, splits, chunks, per);
  return tm == 2 ? gemm_small_tile<2>(ctx, g, splits, chunks, per) : tm == 4 ? gemm_small_tile<4>(ctx, g, splits, chunks, per) : gemm_small_tile<8>(ctx, g, splits, chunks, per);
}

// One launch for the products `d` (each gemm_outer_small_ok with the same K, alpha 1 and no batch)
inline int gemm_outer_group(Ctx* ctx, const GemmDesc* d, int n) {
  OuterGroup g; g.n = n; g.K = d[0].K;
  auto vec = [](const float* p, long ld) { return (int)((reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0); };
  auto lay = [&](int bm) { int tiles = 0; for (int j = 0; j < n; j++) { g.p[j].tile0 = tiles; tiles += (int)(cdiv(d[j].M, bm) * cdiv(d[j].N, 64)); } return tiles; };
  for (int j = 0; j < n; j++) g.p[j] = OuterGroup::P{d[j].A, d[j].B, d[j].C, d[j].a_sum, d[j].sa_k, d[j].sb_k, d[j].ldc, d[j].M, d[j].N, vec(d[j].A, d[j].sa_k), vec(d[j].B, d[j].sb_k), 0};
  // 128-row tiles once they give every SM two blocks
  int tiles = lay(128);
  if (tiles >= 2 * ctx->sm_count) GN_LAUNCH(ctx, outer_group_kernel<8>, tiles, 256, 0, g);
  else { tiles = lay(64); GN_LAUNCH(ctx, outer_group_kernel<4>, tiles, 256, 0, g); }
  return check_launch("outer_group");
}

template <int BM, int BN, int BK, int TM, int TN>
inline int gemm_simt_tile(Ctx* ctx, const GemmDesc& g) {
  const bool ak = g.sa_k == 1, bn = g.sb_n == 1;
  const int va = (ak || g.sa_m == 1) && sg_vec(g.A, ak ? g.sa_m : g.sa_k, g.a_b1, g.a_b2), vb = (bn || g.sb_k == 1) && sg_vec(g.B, bn ? g.sb_k : g.sb_n, g.b_b1, g.b_b2);
  const int tiles_m = cdiv(g.M, BM); constexpr int THREADS = SgCfg<BM, BN, BK, TM, TN>::THREADS;
  for (int y0 = 0; y0 < tiles_m; y0 += 65535) {             // (a grid's second dimension)
    const dim3 grid(cdiv(g.N, BN), std::min(tiles_m - y0, 65535), g.batch1 * g.batch2);
    if (ak && bn) GN_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, true, true>), grid, THREADS, 0, g, va, vb, y0);
    else if (ak && g.sb_k == 1) GN_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, true, false>), grid, THREADS, 0, g, va, vb, y0);
    else if (g.sa_m == 1 && bn) GN_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, false, true>), grid, THREADS, 0, g, va, vb, y0);
    else if (g.sa_m == 1 && g.sb_k == 1) GN_LAUNCH(ctx, (gemm_simt_kernel<BM, BN, BK, TM, TN, false, false>), grid, THREADS, 0, g, va, vb, y0);
    else return fail(GN_ERR_UNSUPPORTED, "gemm_simt: neither stride of an operand is 1");
  }
  return check_launch("gemm_simt");
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
    int s = 1; while (s < SP_MAX_SPLITS && g.K >= 512 * s) s *= 2;
    if ((long)g.M * s > 4L * ctx->sm_count) GN_CLUSTER_LAUNCH(ctx, gemm_skinny_kernel<4>, dim3(cdiv(g.M, 4) * s), 256, 0, s, g, s);
    else GN_CLUSTER_LAUNCH(ctx, gemm_skinny_kernel<1>, dim3(g.M * s), 256, 0, s, g, s);
    return check_launch("gemm_skinny");
  }
  // (which kernel adds up a sample's sums must not depend on the number of samples either)
  const long t64 = (long)cdiv(g.M, 64) * cdiv(g.N, 64) * g.batch1 * g.batch2;
  // (weight gradients of short contractions: more tiles than two per SM are quicker without the sums of eight warps, 1100 x 333 over 100 7.9 -> 7.0)
  const bool quick = g.sa_k != 1 && g.K < 128 && (long)cdiv(g.M, 32) * cdiv(g.N, 32) * g.batch1 * g.batch2 > 2L * ctx->sm_count;
  if (g.K >= SP_KB && (g.sa_k == 1 || (t64 < ctx->sm_count && !quick)) && (!g.a_sum || g.sa_m == 1)) return gemm_small(ctx, g);
  // 16-row tiles for a handful of rows; 32 x 32 tiles (a quarter of the work per block) when 64 x 64 would not give every SM one or
  // be half empty
  if (g.M <= 16) return gemm_simt_tile<16, 64, 32, 2, 4>(ctx, g);
  if (g.M <= 32 || t64 < ctx->sm_count) return gemm_simt_tile<32, 32, 32, 4, 2>(ctx, g);
  return gemm_simt_tile<64, 64, 16, 4, 4>(ctx, g);
}

}  // namespace gn
