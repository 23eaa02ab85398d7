// attention.cuh -- fused causal multi-head attention, forward and backward, without materialising the
// [T, T] score matrices in HBM.
//
// reference: internal/layer/transformer.go:470-503 (forward: scores = q.k / sqrt(hd), masked entries -1e9,
// row softmax, weighted sum of v) and :589-657 (backward: probabilities recomputed from q and k, explicit
// softmax Jacobian, dQ / dK / dV).  The Jacobian row term sum_k dP_k P_k equals dO . O (O = P V), which is
// what the backward kernels use; the row maximum and the row sum of the forward softmax are kept per row.
//
// Arithmetic: fp32-level products from two fp16 parts per operand, x s = hi + lo with a power-of-two scale s per row (22 bits below
// the row's maximum), hi hi + hi lo + lo hi with fp32 accumulation on warp-level tensor-core MMAs (m16n8k16).  The split happens
// once per tile, on the way into shared memory, and the fragments come out by ldmatrix: three MMAs per fragment load of 16
// contraction indices.  (Splitting fp32 fragments into TF32 parts in registers cost two loads and four logic operations per three
// MMAs of 8 indices, in every warp again: 36 us forward and 140 backward at 24 x 150 tokens, 12 heads of 32.)  Where rows are
// summed over (P V, dS K, ...) their inverse scales go into the other operand, which gets a scale per row from its maximum in turn.
// One CTA = 64 query (or key) rows of one head, 4 warps x 16 rows, key (query) blocks of 64 streamed through shared memory;
// causal blocks above the diagonal are never visited.  These kernels take what the tcgen05 kernels do not: heads of 16 and 32, and
// sequences that are not a multiple of 128, where a tile of 128 would be mostly padding.
//
// Q, K, V, O, dO and the outputs are [batch*T, D] row-major with head h in columns [h*HD, (h+1)*HD).
#pragma once
#include "common.cuh"
#include "gemm_tc.cuh"

namespace gn {

constexpr int AT_BLK = 64, AT_THREADS = 128;

__device__ __forceinline__ float quad_max(float v) { v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1)); return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2)); }
__device__ __forceinline__ float quad_sum(float v) { v += __shfl_xor_sync(0xffffffffu, v, 1); return v + __shfl_xor_sync(0xffffffffu, v, 2); }
template <int HD> struct AtCfg {
  static constexpr int LDH = 2 * HD + 8;                     // halves per tile row: hi | lo | pad; an odd number of 16-byte units, so ldmatrix is free of bank conflicts
  static constexpr int TILE = AT_BLK * LDH;
  static constexpr int V4 = HD / 4, RP = AT_THREADS / V4, NP = AT_BLK / RP;      // threads per row, rows per pass, passes of a tile load
};
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
// 64 rows of a [*, D] tensor into a tile (hi | lo), inverse row scales into `inv`; rows >= T read as zero.  With `other`: also the
// dot products of the rows with those of `other`, into `dot` (dO . O).
template <int HD, bool DOT>
__device__ __forceinline__ void at_load(__half* s, float* inv, const float* __restrict__ src, long base, int row0, int T, int D, const float* __restrict__ other = nullptr, float* dot = nullptr) {
  using C = AtCfg<HD>;
  const int c4 = threadIdx.x % C::V4, rr = threadIdx.x / C::V4;
  float4 v[C::NP], w[DOT ? C::NP : 1];
#pragma unroll
  for (int p = 0; p < C::NP; p++) {
    const int row = row0 + p * C::RP + rr; const long o = base + (long)row * D + c4 * 4;
    v[p] = row < T ? *reinterpret_cast<const float4*>(src + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (DOT) w[p] = row < T ? *reinterpret_cast<const float4*>(other + o) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int p = 0; p < C::NP; p++) {
    const int r = p * C::RP + rr;
    float mx = fmaxf(fmaxf(fabsf(v[p].x), fabsf(v[p].y)), fmaxf(fabsf(v[p].z), fabsf(v[p].w))), d = 0.f;
    if constexpr (DOT) d = (v[p].x * w[p].x + v[p].y * w[p].y) + (v[p].z * w[p].z + v[p].w * w[p].w);
#pragma unroll
    for (int o = C::V4 / 2; o > 0; o >>= 1) { mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); if constexpr (DOT) d += __shfl_xor_sync(0xffffffffu, d, o); }
    float iv; const float sc = row_scale(mx, &iv);
    uint2 hi, lo; split2_pair(v[p].x, v[p].y, sc, hi.x, lo.x); split2_pair(v[p].z, v[p].w, sc, hi.y, lo.y);
    *reinterpret_cast<uint2*>(s + r * C::LDH + c4 * 4) = hi; *reinterpret_cast<uint2*>(s + r * C::LDH + HD + c4 * 4) = lo;
    if (c4 == 0) { inv[r] = iv; if constexpr (DOT) dot[r] = d; }
  }
}
// acc[n] = A(rows r0 .. r0 + 15) B(rows 8 n .. 8 n + 7)^T over the HD columns of two tiles, in units of the rows' scales.  Four
// accumulators at a time, so that the three MMAs of one are four instructions apart (a dependent MMA waits 25 cycles, an
// independent one 9).
template <int HD, int NN>
__device__ __forceinline__ void at_rows_product(float (&acc)[NN][4], const __half* A, const __half* B, int r0, int lane) {
  using C = AtCfg<HD>;
#pragma unroll
  for (int n = 0; n < NN; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const __half* ap = A + (r0 + (lane & 15)) * C::LDH + (lane >> 4) * 8;
  const __half* bp = B + (lane & 7) * C::LDH + ((lane >> 3) & 1) * 8 + (lane >> 4) * HD;
#pragma unroll
  for (int k = 0; k < HD; k += 16) {
    uint32_t ah[4], al[4]; ldm4(ah, ap + k); ldm4(al, ap + HD + k);
#pragma unroll
    for (int n0 = 0; n0 < NN; n0 += 4) {
      uint32_t b[4][4];
#pragma unroll
      for (int n = 0; n < 4; n++) ldm4(b[n], bp + (n0 + n) * 8 * C::LDH + k);
#pragma unroll
      for (int n = 0; n < 4; n++) mma16(acc[n0 + n], al, b[n][0], b[n][1]);
#pragma unroll
      for (int n = 0; n < 4; n++) mma16(acc[n0 + n], ah, b[n][2], b[n][3]);
#pragma unroll
      for (int n = 0; n < 4; n++) mma16(acc[n0 + n], ah, b[n][0], b[n][1]);
    }
  }
}
// out = out * keep + X B for a 16 x 8 NN accumulator fragment X and the 8 NN rows of a tile from B on, whose inverse scales `inv` are
// taken into X here; X gets a scale per row (g, g + 8) from its maximum, so it is destroyed.
template <int HD, int NN>
__device__ __forceinline__ void at_sum_rows(float (&out)[HD / 8][4], float keep0, float keep1, float (&x)[NN][4], const __half* B, const float* inv, int lane) {
  using C = AtCfg<HD>;
  const int t = lane & 3; float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int n = 0; n < NN; n++) {
    const float2 iv = *reinterpret_cast<const float2*>(inv + n * 8 + 2 * t);
    x[n][0] *= iv.x; x[n][1] *= iv.y; x[n][2] *= iv.x; x[n][3] *= iv.y;
    m0 = fmaxf(m0, fmaxf(fabsf(x[n][0]), fabsf(x[n][1]))); m1 = fmaxf(m1, fmaxf(fabsf(x[n][2]), fabsf(x[n][3])));
  }
  float i0, i1; const float s0 = row_scale(quad_max(m0), &i0), s1 = row_scale(quad_max(m1), &i1);
  float acc[HD / 8][4];
#pragma unroll
  for (int d = 0; d < HD / 8; d++) acc[d][0] = acc[d][1] = acc[d][2] = acc[d][3] = 0.f;
  const __half* bp = B + ((lane & 7) + ((lane >> 3) & 1) * 8) * C::LDH + (lane >> 4) * HD;
  constexpr int DG = HD / 8 < 4 ? HD / 8 : 4;
#pragma unroll
  for (int k = 0; k < NN / 2; k++) {
    uint32_t ah[4], al[4];
    split2_pair(x[2 * k][0], x[2 * k][1], s0, ah[0], al[0]); split2_pair(x[2 * k][2], x[2 * k][3], s1, ah[1], al[1]);
    split2_pair(x[2 * k + 1][0], x[2 * k + 1][1], s0, ah[2], al[2]); split2_pair(x[2 * k + 1][2], x[2 * k + 1][3], s1, ah[3], al[3]);
#pragma unroll
    for (int d0 = 0; d0 < HD / 8; d0 += DG) {
      uint32_t b[DG][4];
#pragma unroll
      for (int d = 0; d < DG; d++) ldm4t(b[d], bp + k * 16 * C::LDH + (d0 + d) * 8);
#pragma unroll
      for (int d = 0; d < DG; d++) mma16(acc[d0 + d], al, b[d][0], b[d][1]);
#pragma unroll
      for (int d = 0; d < DG; d++) mma16(acc[d0 + d], ah, b[d][2], b[d][3]);
#pragma unroll
      for (int d = 0; d < DG; d++) mma16(acc[d0 + d], ah, b[d][0], b[d][1]);
    }
  }
#pragma unroll
  for (int d = 0; d < HD / 8; d++) {
    out[d][0] = fmaf(acc[d][0], i0, out[d][0] * keep0); out[d][1] = fmaf(acc[d][1], i0, out[d][1] * keep0);
    out[d][2] = fmaf(acc[d][2], i1, out[d][2] * keep1); out[d][3] = fmaf(acc[d][3], i1, out[d][3] * keep1);
  }
}
template <int HD>
__device__ __forceinline__ void at_store(float* __restrict__ dst, const float (&v)[HD / 8][4], float f0, float f1, long base, int i0, int i1, int T, int D, int t) {
#pragma unroll
  for (int d = 0; d < HD / 8; d++) {
    if (i0 < T) *reinterpret_cast<float2*>(dst + base + (long)i0 * D + d * 8 + 2 * t) = make_float2(v[d][0] * f0, v[d][1] * f0);
    if (i1 < T) *reinterpret_cast<float2*>(dst + base + (long)i1 * D + d * 8 + 2 * t) = make_float2(v[d][2] * f1, v[d][3] * f1);
  }
}

// ---------------------------------------------------------------- forward
template <int HD>
__global__ void __launch_bounds__(AT_THREADS) attn_fwd_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                                                               float* __restrict__ O, float* __restrict__ Mst, float* __restrict__ Lst,
                                                               int T, int D, int H, int causal, float inv_scale) {
  using C = AtCfg<HD>;
  extern __shared__ __align__(16) uint8_t at_sm[];
  __half* Qs = reinterpret_cast<__half*>(at_sm); __half* Ks = Qs + C::TILE; __half* Vs = Ks + C::TILE;
  float* iq = reinterpret_cast<float*>(Vs + C::TILE); float* ik = iq + AT_BLK; float* iv = ik + AT_BLK;
  const int qb = causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x, h = blockIdx.y, b = blockIdx.z, q0 = qb * AT_BLK;      // (causal: the long rows first)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long base = (long)b * T * D + (long)h * HD;
  at_load<HD, false>(Qs, iq, Q, base, q0, T, D);
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  const int nkb = causal ? qb + 1 : (T + AT_BLK - 1) / AT_BLK;
  const int r0 = warp * 16, i0 = q0 + r0 + g, i1 = i0 + 8;
  for (int kb = 0; kb < nkb; kb++) {
    __syncthreads();
    at_load<HD, false>(Ks, ik, K, base, kb * AT_BLK, T, D); at_load<HD, false>(Vs, iv, V, base, kb * AT_BLK, T, D);
    __syncthreads();
    if (q0 + r0 >= T) continue;                              // (this warp's rows are all padding)
    float s[8][4]; at_rows_product<HD, 8>(s, Qs, Ks, r0, lane);
    const float f0 = iq[r0 + g] * inv_scale, f1 = iq[r0 + g + 8] * inv_scale;
    const bool edge = (kb + 1) * AT_BLK > T || (causal && kb == qb);
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const float2 kk = *reinterpret_cast<const float2*>(ik + n * 8 + 2 * t);
      s[n][0] *= f0 * kk.x; s[n][1] *= f0 * kk.y; s[n][2] *= f1 * kk.x; s[n][3] *= f1 * kk.y;
      if (edge) {
#pragma unroll
        for (int e = 0; e < 4; e++) { const int j = kb * AT_BLK + n * 8 + 2 * t + (e & 1); if (j >= T || (causal && j > (e < 2 ? i0 : i1))) s[n][e] = -INFINITY; }
      }
      mx0 = fmaxf(mx0, fmaxf(s[n][0], s[n][1])); mx1 = fmaxf(mx1, fmaxf(s[n][2], s[n][3]));
    }
    const float mn0 = fmaxf(m[0], quad_max(mx0)), mn1 = fmaxf(m[1], quad_max(mx1));
    const float c0 = __expf(m[0] - mn0), c1 = __expf(m[1] - mn1);
    float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
    for (int n = 0; n < 8; n++) {
      s[n][0] = __expf(s[n][0] - mn0); s[n][1] = __expf(s[n][1] - mn0); s[n][2] = __expf(s[n][2] - mn1); s[n][3] = __expf(s[n][3] - mn1);
      rs0 += s[n][0] + s[n][1]; rs1 += s[n][2] + s[n][3];
    }
    l[0] = l[0] * c0 + quad_sum(rs0); l[1] = l[1] * c1 + quad_sum(rs1); m[0] = mn0; m[1] = mn1;
    at_sum_rows<HD, 8>(o, c0, c1, s, Vs, iv, lane);
  }
  if (q0 + r0 >= T) return;
  at_store<HD>(O, o, 1.f / l[0], 1.f / l[1], base, i0, i1, T, D, t);
  if (t == 0) {
    const long sb = ((long)b * H + h) * T;
    if (i0 < T) { Mst[sb + i0] = m[0]; Lst[sb + i0] = l[0]; }
    if (i1 < T) { Mst[sb + i1] = m[1]; Lst[sb + i1] = l[1]; }
  }
}

// Dv[b,h,i] = sum_d dO[b,i,h*64+d] * O[b,i,h*64+d]   (= sum_k dP_ik P_ik, the softmax-Jacobian row term), for head size 64 and
// D = 64 H (rows of all heads are then consecutive 64-float segments): 16 threads per row, 16-byte loads, two rows in flight
// per thread.
__global__ void __launch_bounds__(256) attn_rowdot64_kernel(const float* __restrict__ dO, const float* __restrict__ O, float* __restrict__ Dv, int T, int H, long rows) {
  const long gid = (long)blockIdx.x * 256 + threadIdx.x, half = (long)gridDim.x * 16;      // rows per pass of the grid
  const int l16 = threadIdx.x & 15;
  for (long w = gid >> 4; w < rows; w += 2 * half) {
    const long w2 = w + half;
    const float4 a = *reinterpret_cast<const float4*>(dO + w * 64 + l16 * 4), b = *reinterpret_cast<const float4*>(O + w * 64 + l16 * 4);
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f), d = c;
    if (w2 < rows) { c = *reinterpret_cast<const float4*>(dO + w2 * 64 + l16 * 4); d = *reinterpret_cast<const float4*>(O + w2 * 64 + l16 * 4); }
    float s = (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w), s2 = (c.x * d.x + c.y * d.y) + (c.z * d.z + c.w * d.w);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) { s += __shfl_xor_sync(0xffffffffu, s, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); }
    if (l16 == 0) {
      { const int h = (int)(w % H); const long tok = w / H; Dv[((tok / T) * H + h) * T + tok % T] = s; }
      if (w2 < rows) { const int h = (int)(w2 % H); const long tok = w2 / H; Dv[((tok / T) * H + h) * T + tok % T] = s2; }
    }
  }
}

// ---------------------------------------------------------------- backward
// The first half of the grid's blocks: dQ of 64 query rows.  For every key block at or below the diagonal: S = Q K^T,
// P = exp(S/sqrt(hd) - m) / l, dP = dO V^T, dS = P (dP - dO . O) / sqrt(hd), dQ += dS K.
// The second half: dK and dV of 64 key rows.  For every query block at or above the diagonal the TRANSPOSED tiles are formed
// directly: S^T = K Q^T, P^T, dP^T = V dO^T, dS^T; dK += dS^T Q, dV += P^T dO.
// One launch, so that a few hundred blocks of either kind fill the SMs together; dO . O is formed while dO is loaded.
template <int HD>
__global__ void __launch_bounds__(AT_THREADS, HD == 64 ? 3 : 4) attn_bwd_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ O,
                                                              const float* __restrict__ dO, const float* __restrict__ Mst, const float* __restrict__ Lst,
                                                              float* __restrict__ dQ, float* __restrict__ dK, float* __restrict__ dV, int T, int D, int H, int causal, float inv_scale) {
  using C = AtCfg<HD>;
  extern __shared__ __align__(16) uint8_t at_sm[];
  __half* Qs = reinterpret_cast<__half*>(at_sm); __half* Gs = Qs + C::TILE; __half* Ks = Gs + C::TILE; __half* Vs = Ks + C::TILE;
  float* iq = reinterpret_cast<float*>(Vs + C::TILE); float* ig = iq + AT_BLK; float* ik = ig + AT_BLK; float* iv = ik + AT_BLK;
  float* st_m = iv + AT_BLK; float* st_il = st_m + AT_BLK; float* st_d = st_il + AT_BLK;
  const int nb = (T + AT_BLK - 1) / AT_BLK, h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r0 = warp * 16;
  const long base = (long)b * T * D + (long)h * HD, sb = ((long)b * H + h) * T;
  if (blockIdx.x < nb) {
    const int qb = nb - 1 - blockIdx.x, q0 = qb * AT_BLK;
    at_load<HD, false>(Qs, iq, Q, base, q0, T, D); at_load<HD, true>(Gs, ig, dO, base, q0, T, D, O, st_d);
    __syncthreads();
    const int i0 = q0 + r0 + g, i1 = i0 + 8;
    const float m0 = i0 < T ? Mst[sb + i0] : 0.f, m1 = i1 < T ? Mst[sb + i1] : 0.f;
    const float il0 = i0 < T ? 1.f / Lst[sb + i0] : 0.f, il1 = i1 < T ? 1.f / Lst[sb + i1] : 0.f;
    const float d0 = st_d[r0 + g], d1 = st_d[r0 + g + 8], f0 = iq[r0 + g] * inv_scale, f1 = iq[r0 + g + 8] * inv_scale, g0 = ig[r0 + g], g1 = ig[r0 + g + 8];
    float acc[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int nkb = causal ? qb + 1 : nb;
    for (int kb = 0; kb < nkb; kb++) {
      __syncthreads();
      at_load<HD, false>(Ks, ik, K, base, kb * AT_BLK, T, D); at_load<HD, false>(Vs, iv, V, base, kb * AT_BLK, T, D);
      __syncthreads();
      if (q0 + r0 >= T) continue;
      const bool edge = (kb + 1) * AT_BLK > T || (causal && kb == qb);
#pragma unroll 1
      for (int kh = 0; kh < AT_BLK; kh += 32) {              // 32 keys at a time: half the accumulators of a whole block
        if (kb * AT_BLK + kh >= T) break;
        float s[4][4], dp[4][4]; at_rows_product<HD, 4>(s, Qs, Ks + kh * C::LDH, r0, lane); at_rows_product<HD, 4>(dp, Gs, Vs + kh * C::LDH, r0, lane);
#pragma unroll
        for (int n = 0; n < 4; n++) {
          const float2 kk = *reinterpret_cast<const float2*>(ik + kh + n * 8 + 2 * t), vv = *reinterpret_cast<const float2*>(iv + kh + n * 8 + 2 * t);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float fk = e & 1 ? kk.y : kk.x, fv = e & 1 ? vv.y : vv.x;
            const int j = kb * AT_BLK + kh + n * 8 + 2 * t + (e & 1), i = e < 2 ? i0 : i1;
            const float p = edge && (j >= T || (causal && j > i)) ? 0.f : __expf(s[n][e] * ((e < 2 ? f0 : f1) * fk) - (e < 2 ? m0 : m1)) * (e < 2 ? il0 : il1);      // (rows beyond T: il = 0)
            s[n][e] = p * (dp[n][e] * ((e < 2 ? g0 : g1) * fv) - (e < 2 ? d0 : d1)) * inv_scale;        // dS
          }
        }
        at_sum_rows<HD, 4>(acc, 1.f, 1.f, s, Ks + kh * C::LDH, ik + kh, lane);
      }
    }
    at_store<HD>(dQ, acc, 1.f, 1.f, base, i0, i1, T, D, t);
    return;
  }
  const int kbk = blockIdx.x - nb, k0 = kbk * AT_BLK;
  at_load<HD, false>(Ks, ik, K, base, k0, T, D); at_load<HD, false>(Vs, iv, V, base, k0, T, D);
  __syncthreads();
  const int j0 = k0 + r0 + g, j1 = j0 + 8;
  const float f0 = ik[r0 + g] * inv_scale, f1 = ik[r0 + g + 8] * inv_scale, v0 = iv[r0 + g], v1 = iv[r0 + g + 8];
  float ak[HD / 8][4], av[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; i++) { ak[i][0] = ak[i][1] = ak[i][2] = ak[i][3] = 0.f; av[i][0] = av[i][1] = av[i][2] = av[i][3] = 0.f; }
  for (int qb = causal ? kbk : 0; qb < nb; qb++) {
    __syncthreads();
    at_load<HD, false>(Qs, iq, Q, base, qb * AT_BLK, T, D); at_load<HD, true>(Gs, ig, dO, base, qb * AT_BLK, T, D, O, st_d);
    if (threadIdx.x < AT_BLK) {
      const int i = qb * AT_BLK + threadIdx.x;
      st_m[threadIdx.x] = i < T ? Mst[sb + i] : 0.f; st_il[threadIdx.x] = i < T ? 1.f / Lst[sb + i] : 0.f;
    }
    __syncthreads();
    if (k0 + r0 >= T) continue;
    const bool edge = k0 + AT_BLK > T || (causal && kbk == qb);
    // rows = keys j (g, g+8), columns = queries i (2t, 2t+1 of n-tile n), 32 queries at a time
#pragma unroll 1
    for (int qh = 0; qh < AT_BLK; qh += 32) {
      if (qb * AT_BLK + qh >= T) break;
      float s[4][4], dp[4][4]; at_rows_product<HD, 4>(s, Ks, Qs + qh * C::LDH, r0, lane); at_rows_product<HD, 4>(dp, Vs, Gs + qh * C::LDH, r0, lane);
#pragma unroll
      for (int n = 0; n < 4; n++) {
        const int c0 = qh + n * 8 + 2 * t;
        const float2 qq = *reinterpret_cast<const float2*>(iq + c0), gg = *reinterpret_cast<const float2*>(ig + c0), mm = *reinterpret_cast<const float2*>(st_m + c0),
                     ll = *reinterpret_cast<const float2*>(st_il + c0), dd = *reinterpret_cast<const float2*>(st_d + c0);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int i = qb * AT_BLK + c0 + (e & 1), j = e < 2 ? j0 : j1;
          const float p = edge && (j >= T || (causal && j > i)) ? 0.f : __expf(s[n][e] * ((e < 2 ? f0 : f1) * (e & 1 ? qq.y : qq.x)) - (e & 1 ? mm.y : mm.x)) * (e & 1 ? ll.y : ll.x);      // (columns beyond T: il = 0)
          dp[n][e] = p * (dp[n][e] * ((e < 2 ? v0 : v1) * (e & 1 ? gg.y : gg.x)) - (e & 1 ? dd.y : dd.x)) * inv_scale;      // dS^T
          s[n][e] = p;                                                                                                     // P^T
        }
      }
      at_sum_rows<HD, 4>(av, 1.f, 1.f, s, Gs + qh * C::LDH, ig + qh, lane); at_sum_rows<HD, 4>(ak, 1.f, 1.f, dp, Qs + qh * C::LDH, iq + qh, lane);
    }
  }
  at_store<HD>(dK, ak, 1.f, 1.f, base, j0, j1, T, D, t); at_store<HD>(dV, av, 1.f, 1.f, base, j0, j1, T, D, t);
}

// ---------------------------------------------------------------- whole heads
// The same arithmetic in the same order, a block per head: short sequences fit shared memory as a whole, so every tensor is read and split
// once (the blocks of 64 rows above read and split each one again for every block of the other side, between two barriers, with nothing in flight meanwhile)
// and then every warp walks its rows by itself.  Rows are padded to 32, and keys (queries) go 32 at a time where 64 are not there: what is
// left out is masked or zero.  With a causal mask a warp's query rows and key rows cost the same together, whichever they are.  Bound by
// the latency of its chains of dependent MMAs and element-wise work; figures at at_head_better.
__host__ __device__ __forceinline__ int at_pad(int T) { return (T + 31) & ~31; }
template <int HD> inline size_t at_head_smem(int T, bool bwd) { return (size_t)at_pad(T) * ((bwd ? 4 : 3) * AtCfg<HD>::LDH * sizeof(__half) + (bwd ? 7 : 3) * sizeof(float)); }
// all rows of a head (zeros from T to the padded end); see at_load
template <int HD, bool DOT>
__device__ __forceinline__ void at_load_head(__half* s, float* inv, const float* __restrict__ src, long base, int T, int D, const float* __restrict__ other = nullptr, float* dot = nullptr) {
  using C = AtCfg<HD>; constexpr int NP = DOT ? 2 : 4;
  const int c4 = threadIdx.x % C::V4, step = blockDim.x / C::V4, Tp = at_pad(T);
  for (int p0 = threadIdx.x / C::V4; p0 - (int)(threadIdx.x / C::V4) < Tp; p0 += NP * step) {      // (the same number of rounds in every thread)
    float4 v[NP], w[DOT ? NP : 1];
#pragma unroll
    for (int p = 0; p < NP; p++) {
      const int row = p0 + p * step; const long o = base + (long)row * D + c4 * 4;
      v[p] = row < T ? *reinterpret_cast<const float4*>(src + o) : make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (DOT) w[p] = row < T ? *reinterpret_cast<const float4*>(other + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int p = 0; p < NP; p++) {
      const int r = p0 + p * step;
      float mx = fmaxf(fmaxf(fabsf(v[p].x), fabsf(v[p].y)), fmaxf(fabsf(v[p].z), fabsf(v[p].w))), d = 0.f;
      if constexpr (DOT) d = (v[p].x * w[p].x + v[p].y * w[p].y) + (v[p].z * w[p].z + v[p].w * w[p].w);
#pragma unroll
      for (int o = C::V4 / 2; o > 0; o >>= 1) { mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); if constexpr (DOT) d += __shfl_xor_sync(0xffffffffu, d, o); }
      float iv; const float sc = row_scale(mx, &iv);
      uint2 hi, lo; split2_pair(v[p].x, v[p].y, sc, hi.x, lo.x); split2_pair(v[p].z, v[p].w, sc, hi.y, lo.y);
      if (r < Tp) {
        *reinterpret_cast<uint2*>(s + r * C::LDH + c4 * 4) = hi; *reinterpret_cast<uint2*>(s + r * C::LDH + HD + c4 * 4) = lo;
        if (c4 == 0) { inv[r] = iv; if constexpr (DOT) dot[r] = d; }
      }
    }
  }
}
template <int HD, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) attn_head_fwd_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                                                                      float* __restrict__ O, float* __restrict__ Mst, float* __restrict__ Lst, int T, int D, int H, int causal, float inv_scale) {
  using C = AtCfg<HD>;
  extern __shared__ __align__(16) uint8_t at_sm[];
  const int Tp = at_pad(T), h = blockIdx.x, b = blockIdx.y, nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __half* Qs = reinterpret_cast<__half*>(at_sm); __half* Ks = Qs + Tp * C::LDH; __half* Vs = Ks + Tp * C::LDH;
  float* iq = reinterpret_cast<float*>(Vs + Tp * C::LDH); float* ik = iq + Tp; float* iv = ik + Tp;
  const long base = (long)b * T * D + (long)h * HD, sb = ((long)b * H + h) * T;
  at_load_head<HD, false>(Qs, iq, Q, base, T, D); at_load_head<HD, false>(Ks, ik, K, base, T, D); at_load_head<HD, false>(Vs, iv, V, base, T, D);
  __syncthreads();
  for (int r0 = warp * 16; r0 < T; r0 += nw * 16) {
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    const int i0 = r0 + g, i1 = i0 + 8, kend = causal ? min(Tp, at_pad(r0 + 16)) : Tp;
    const float f0 = iq[i0] * inv_scale, f1 = iq[i1] * inv_scale;
    auto block = [&](int k0, auto nn) {
      constexpr int NN = decltype(nn)::value;
      float s[NN][4]; at_rows_product<HD, NN>(s, Qs, Ks + k0 * C::LDH, r0, lane);
      const bool edge = k0 + 8 * NN > T || (causal && k0 + 8 * NN > r0);
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int n = 0; n < NN; n++) {
        const float2 kk = *reinterpret_cast<const float2*>(ik + k0 + n * 8 + 2 * t);
        s[n][0] *= f0 * kk.x; s[n][1] *= f0 * kk.y; s[n][2] *= f1 * kk.x; s[n][3] *= f1 * kk.y;
        if (edge) {
#pragma unroll
          for (int e = 0; e < 4; e++) { const int j = k0 + n * 8 + 2 * t + (e & 1); if (j >= T || (causal && j > (e < 2 ? i0 : i1))) s[n][e] = -INFINITY; }
        }
        mx0 = fmaxf(mx0, fmaxf(s[n][0], s[n][1])); mx1 = fmaxf(mx1, fmaxf(s[n][2], s[n][3]));
      }
      const float mn0 = fmaxf(m[0], quad_max(mx0)), mn1 = fmaxf(m[1], quad_max(mx1));
      const float c0 = __expf(m[0] - mn0), c1 = __expf(m[1] - mn1);
      float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
      for (int n = 0; n < NN; n++) {
        s[n][0] = __expf(s[n][0] - mn0); s[n][1] = __expf(s[n][1] - mn0); s[n][2] = __expf(s[n][2] - mn1); s[n][3] = __expf(s[n][3] - mn1);
        rs0 += s[n][0] + s[n][1]; rs1 += s[n][2] + s[n][3];
      }
      l[0] = l[0] * c0 + quad_sum(rs0); l[1] = l[1] * c1 + quad_sum(rs1); m[0] = mn0; m[1] = mn1;
      at_sum_rows<HD, NN>(o, c0, c1, s, Vs + k0 * C::LDH, iv + k0, lane);
    };
    int k0 = 0;
    for (; k0 + 64 <= kend; k0 += 64) block(k0, std::integral_constant<int, 8>{});
    if (k0 < kend) block(k0, std::integral_constant<int, 4>{});
    at_store<HD>(O, o, 1.f / l[0], 1.f / l[1], base, i0, i1, T, D, t);
    if (t == 0) {
      if (i0 < T) { Mst[sb + i0] = m[0]; Lst[sb + i0] = l[0]; }
      if (i1 < T) { Mst[sb + i1] = m[1]; Lst[sb + i1] = l[1]; }
    }
  }
}
template <int HD, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) attn_head_bwd_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ O,
                                                                      const float* __restrict__ dO, const float* __restrict__ Mst, const float* __restrict__ Lst,
                                                                      float* __restrict__ dQ, float* __restrict__ dK, float* __restrict__ dV, int T, int D, int H, int causal, float inv_scale) {
  using C = AtCfg<HD>;
  extern __shared__ __align__(16) uint8_t at_sm[];
  const int Tp = at_pad(T), h = blockIdx.x, b = blockIdx.y, nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __half* Qs = reinterpret_cast<__half*>(at_sm); __half* Gs = Qs + Tp * C::LDH; __half* Ks = Gs + Tp * C::LDH; __half* Vs = Ks + Tp * C::LDH;
  float* iq = reinterpret_cast<float*>(Vs + Tp * C::LDH); float* ig = iq + Tp; float* ik = ig + Tp; float* iv = ik + Tp; float* st_m = iv + Tp; float* st_il = st_m + Tp; float* st_d = st_il + Tp;
  const long base = (long)b * T * D + (long)h * HD, sb = ((long)b * H + h) * T;
  for (int i = threadIdx.x; i < Tp; i += blockDim.x) { st_m[i] = i < T ? Mst[sb + i] : 0.f; st_il[i] = i < T ? 1.f / Lst[sb + i] : 0.f; }
  at_load_head<HD, false>(Qs, iq, Q, base, T, D); at_load_head<HD, true>(Gs, ig, dO, base, T, D, O, st_d);
  at_load_head<HD, false>(Ks, ik, K, base, T, D); at_load_head<HD, false>(Vs, iv, V, base, T, D);
  __syncthreads();
  for (int r0 = warp * 16; r0 < T; r0 += nw * 16) {
    {   // dQ of 16 query rows
      const int i0 = r0 + g, i1 = i0 + 8, kend = causal ? min(Tp, at_pad(r0 + 16)) : Tp;
      const float m0 = st_m[i0], m1 = st_m[i1], il0 = st_il[i0], il1 = st_il[i1], d0 = st_d[i0], d1 = st_d[i1], f0 = iq[i0] * inv_scale, f1 = iq[i1] * inv_scale, g0 = ig[i0], g1 = ig[i1];
      float acc[HD / 8][4];
#pragma unroll
      for (int i = 0; i < HD / 8; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
      for (int k0 = 0; k0 < kend; k0 += 32) {
        const bool edge = k0 + 32 > T || (causal && k0 + 32 > r0);
        float s[4][4], dp[4][4]; at_rows_product<HD, 4>(s, Qs, Ks + k0 * C::LDH, r0, lane); at_rows_product<HD, 4>(dp, Gs, Vs + k0 * C::LDH, r0, lane);
#pragma unroll
        for (int n = 0; n < 4; n++) {
          const float2 kk = *reinterpret_cast<const float2*>(ik + k0 + n * 8 + 2 * t), vv = *reinterpret_cast<const float2*>(iv + k0 + n * 8 + 2 * t);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float fk = e & 1 ? kk.y : kk.x, fv = e & 1 ? vv.y : vv.x;
            const int j = k0 + n * 8 + 2 * t + (e & 1), i = e < 2 ? i0 : i1;
            const float p = edge && (j >= T || (causal && j > i)) ? 0.f : __expf(s[n][e] * ((e < 2 ? f0 : f1) * fk) - (e < 2 ? m0 : m1)) * (e < 2 ? il0 : il1);      // (rows beyond T: il = 0)
            s[n][e] = p * (dp[n][e] * ((e < 2 ? g0 : g1) * fv) - (e < 2 ? d0 : d1)) * inv_scale;        // dS
          }
        }
        at_sum_rows<HD, 4>(acc, 1.f, 1.f, s, Ks + k0 * C::LDH, ik + k0, lane);
      }
      at_store<HD>(dQ, acc, 1.f, 1.f, base, i0, i1, T, D, t);
    }
    {   // dK and dV of 16 key rows
      const int j0 = r0 + g, j1 = j0 + 8;
      const float f0 = ik[j0] * inv_scale, f1 = ik[j1] * inv_scale, v0 = iv[j0], v1 = iv[j1];
      float ak[HD / 8][4], av[HD / 8][4];
#pragma unroll
      for (int i = 0; i < HD / 8; i++) { ak[i][0] = ak[i][1] = ak[i][2] = ak[i][3] = 0.f; av[i][0] = av[i][1] = av[i][2] = av[i][3] = 0.f; }
#pragma unroll 1
      for (int q0 = causal ? r0 & ~31 : 0; q0 < Tp; q0 += 32) {
        const bool edge = r0 + 16 > T || (causal && q0 < r0 + 16);
        float s[4][4], dp[4][4]; at_rows_product<HD, 4>(s, Ks, Qs + q0 * C::LDH, r0, lane); at_rows_product<HD, 4>(dp, Vs, Gs + q0 * C::LDH, r0, lane);
#pragma unroll
        for (int n = 0; n < 4; n++) {
          const int c0 = q0 + n * 8 + 2 * t;
          const float2 qq = *reinterpret_cast<const float2*>(iq + c0), gg = *reinterpret_cast<const float2*>(ig + c0), mm = *reinterpret_cast<const float2*>(st_m + c0),
                       ll = *reinterpret_cast<const float2*>(st_il + c0), dd = *reinterpret_cast<const float2*>(st_d + c0);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int i = c0 + (e & 1), j = e < 2 ? j0 : j1;
            const float p = edge && (j >= T || (causal && j > i)) ? 0.f : __expf(s[n][e] * ((e < 2 ? f0 : f1) * (e & 1 ? qq.y : qq.x)) - (e & 1 ? mm.y : mm.x)) * (e & 1 ? ll.y : ll.x);      // (columns beyond T: il = 0)
            dp[n][e] = p * (dp[n][e] * ((e < 2 ? v0 : v1) * (e & 1 ? gg.y : gg.x)) - (e & 1 ? dd.y : dd.x)) * inv_scale;      // dS^T
            s[n][e] = p;                                                                                                     // P^T
          }
        }
        at_sum_rows<HD, 4>(av, 1.f, 1.f, s, Gs + q0 * C::LDH, ig + q0, lane); at_sum_rows<HD, 4>(ak, 1.f, 1.f, dp, Qs + q0 * C::LDH, iq + q0, lane);
      }
      at_store<HD>(dK, ak, 1.f, 1.f, base, j0, j1, T, D, t); at_store<HD>(dV, av, 1.f, 1.f, base, j0, j1, T, D, t);
    }
  }
}

// ---------------------------------------------------------------- a few query rows
// Attention of TE = 1 or 2 query rows per sequence (token 0, and the last token) against all T keys, any head size: what the
// top block below a CLSPooling needs (plan_token_rows in model.cu).  Q and O are [B * TE, D], K and V [B * T, D].  One block per
// (head, sequence); a thread forms the scores of its keys (16-byte loads along a key's row where they are aligned: `vec`), then
// the threads split into groups of hd columns for the weighted sum.  Bound by reading K and V once.
constexpr int AR_THREADS = 512;                             // (64 heads of 64 and 384 keys: 9.6 us, 15 with 256 threads and four loads in flight)
__device__ __forceinline__ float ar_dot(const float* __restrict__ q, const float* __restrict__ k, int hd, bool vec) {
  float s = 0.f;
  if (vec) {
#pragma unroll 8
    for (int d = 0; d < hd; d += 4) {
      const float4 x = *reinterpret_cast<const float4*>(k + d);
      s = fmaf(q[d], x.x, s); s = fmaf(q[d + 1], x.y, s); s = fmaf(q[d + 2], x.z, s); s = fmaf(q[d + 3], x.w, s);
    }
  } else for (int d = 0; d < hd; d++) s = fmaf(q[d], k[d], s);
  return s;
}
// out[d] = sum_j w[j] X[j * D + d], d < hd, in a fixed order; `part`: AR_THREADS floats
__device__ __forceinline__ void ar_weighted(const float* __restrict__ w, const float* __restrict__ X, int n, int D, int hd, float* part, float* out) {
  for (int d0 = 0; d0 < hd; d0 += AR_THREADS) {
    const int cols = min(hd - d0, AR_THREADS), groups = AR_THREADS / cols, g = threadIdx.x / cols, d = threadIdx.x - g * cols;
    float s = 0.f;
    if (g < groups) {
      const float* x = X + d0 + d;
#pragma unroll 8
      for (int j = g; j < n; j += groups) s = fmaf(w[j], x[(long)j * D], s);
    }
    __syncthreads();
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < cols) { float a = 0.f; for (int q = 0; q < groups; q++) a += part[q * cols + threadIdx.x]; out[d0 + threadIdx.x] = a; }
  }
}
__global__ void __launch_bounds__(AR_THREADS) attn_rows_fwd_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V, float* __restrict__ O,
                                                                   int T, int TE, int D, int hd, int causal, float inv_scale, int vec) {
  extern __shared__ float sm[];
  __shared__ float red[33], part[AR_THREADS];
  float* q = sm; float* p = sm + hd;                        // one query at a time: its row, its T scores
  const int h = blockIdx.x; const long b = blockIdx.y; const float* Kh = K + b * T * D + (long)h * hd; const float* Vh = V + b * T * D + (long)h * hd;
  for (int e = 0; e < TE; e++) {
    const int n = causal && e == 0 ? 1 : T;                 // keys that token 0 / the last token sees
    const long row = (b * TE + e) * D + (long)h * hd;
    __syncthreads();
    for (int d = threadIdx.x; d < hd; d += AR_THREADS) q[d] = Q[row + d];
    __syncthreads();
    float mx = -INFINITY;
    for (int j = threadIdx.x; j < n; j += AR_THREADS) { const float s = ar_dot(q, Kh + (long)j * D, hd, vec) * inv_scale; p[j] = s; mx = fmaxf(mx, s); }
    mx = block_max(mx, red);
    float l = 0.f;
    for (int j = threadIdx.x; j < n; j += AR_THREADS) { const float v = expf(p[j] - mx); p[j] = v; l += v; }
    l = block_sum(l, red);
    const float il = 1.f / l;
    for (int j = threadIdx.x; j < n; j += AR_THREADS) p[j] *= il;
    __syncthreads();
    ar_weighted(p, Vh, n, D, hd, part, O + row);
  }
}
// Backward of query token 0 without a mask (transformer.go:589-657 for one query): dq [B, D]; dk, dv [B * T, D]; and the sums of
// dk and dv over the tokens, [B, D].  q rows are `ldq` floats apart per sequence; probabilities are recomputed.
__global__ void __launch_bounds__(AR_THREADS) attn_rows_bwd_kernel(const float* __restrict__ Q, long ldq, const float* __restrict__ K, const float* __restrict__ V,
                                                                   const float* __restrict__ dO, float* __restrict__ dQ, float* __restrict__ dK, float* __restrict__ dV,
                                                                   float* __restrict__ dKsum, float* __restrict__ dVsum, int T, int D, int hd, float inv_scale, int vec) {
  extern __shared__ float sm[];
  __shared__ float red[33], part[AR_THREADS];
  float* q = sm; float* g = q + hd; float* p = g + hd; float* ds = p + T;
  const int h = blockIdx.x; const long b = blockIdx.y, base = b * T * D + (long)h * hd, row = b * D + (long)h * hd;
  for (int d = threadIdx.x; d < hd; d += AR_THREADS) { q[d] = Q[b * ldq + (long)h * hd + d]; g[d] = dO[row + d]; }
  __syncthreads();
  float mx = -INFINITY;
  for (int j = threadIdx.x; j < T; j += AR_THREADS) {
    const float s = ar_dot(q, K + base + (long)j * D, hd, vec) * inv_scale;
    p[j] = s; mx = fmaxf(mx, s); ds[j] = ar_dot(g, V + base + (long)j * D, hd, vec);
  }
  mx = block_max(mx, red);
  float l = 0.f;
  for (int j = threadIdx.x; j < T; j += AR_THREADS) { const float v = expf(p[j] - mx); p[j] = v; l += v; }
  l = block_sum(l, red);
  const float il = 1.f / l;
  float dd = 0.f, ps = 0.f;
  for (int j = threadIdx.x; j < T; j += AR_THREADS) { const float v = p[j] * il; p[j] = v; ps += v; dd = fmaf(v, ds[j], dd); }
  dd = block_sum(dd, red); ps = block_sum(ps, red);
  float ss = 0.f;
  for (int j = threadIdx.x; j < T; j += AR_THREADS) { const float v = p[j] * (ds[j] - dd) * inv_scale; ds[j] = v; ss += v; }
  ss = block_sum(ss, red);
  for (int d = threadIdx.x; d < hd; d += AR_THREADS) { dKsum[row + d] = ss * q[d]; dVsum[row + d] = ps * g[d]; }
  for (int e = threadIdx.x; e < T * hd; e += AR_THREADS) {
    const int j = e / hd, d = e - j * hd; const long o = base + (long)j * D + d;
    dK[o] = ds[j] * q[d]; dV[o] = p[j] * g[d];
  }
  ar_weighted(ds, K + base, T, D, hd, part, dQ + row);
}
// The scores of a row (twice, in the backward kernel) and two rows of the head live in shared memory; beyond that all tokens are computed.
constexpr int AR_MAX_T = 16384, AR_SMEM = 200 * 1024;
inline bool attn_rows_fit(int T, int hd) { return T <= AR_MAX_T && ((size_t)2 * hd + 2 * T) * sizeof(float) <= AR_SMEM; }
inline bool ar_vec(const float* a, const float* b, int D, int hd) { return D % 4 == 0 && hd % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0; }
inline int attn_rows_fwd(Ctx* ctx, const float* Q, const float* K, const float* V, float* O, int B, int T, int TE, int D, int H, int causal) {
  const int hd = D / H; const size_t smem = ((size_t)hd + T) * sizeof(float);
  if (smem > 40 * 1024) GN_CUDA(cudaFuncSetAttribute(attn_rows_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, attn_rows_fwd_kernel, dim3(H, B), AR_THREADS, smem, Q, K, V, O, T, TE, D, hd, causal, 1.f / sqrtf((float)hd), ar_vec(K, K, D, hd) ? 1 : 0);
  return check_launch("attn_rows_fwd");
}
inline int attn_rows_bwd(Ctx* ctx, const float* Q, long ldq, const float* K, const float* V, const float* dO, float* dQ, float* dK, float* dV, float* dKsum, float* dVsum,
                         int B, int T, int D, int H) {
  const int hd = D / H; const size_t smem = ((size_t)2 * hd + 2 * T) * sizeof(float);
  if (smem > 40 * 1024) GN_CUDA(cudaFuncSetAttribute(attn_rows_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, attn_rows_bwd_kernel, dim3(H, B), AR_THREADS, smem, Q, ldq, K, V, dO, dQ, dK, dV, dKsum, dVsum, T, D, hd, 1.f / sqrtf((float)hd), ar_vec(K, V, D, hd) ? 1 : 0);
  return check_launch("attn_rows_bwd");
}

// ---------------------------------------------------------------- launchers
inline bool attn_fused_supported(int hd, int D) { return (hd == 16 || hd == 32 || hd == 64) && D % 4 == 0; }

// Warps of a block per head: one per 16 rows up to 16, then as few as take the same number of turns.  Heads of 32 and 64 count the rows of padding: where the number
// would be odd, the padding took a second pass of loads (288 heads of 200 tokens, size 32, causal 28.1 -> 24.3 us, of 80 tokens 9.6 -> 8.0).
template <int HD> inline int at_head_warps(int T) { const int n = HD == 16 ? cdiv(T, 16) : at_pad(T) / 16; return n <= 16 ? n : cdiv(n, cdiv(n, 16)); }
// Blocks of 64 rows or a block per head?  By estimated time (us, from measured rates).  A block per head takes `h0` and `h1` per 32 keys and turn; two that share an
// SM take 1.4 times as long as one.  A round of the others, as many as are resident, takes `t0` and `t1` per 64 keys (rows of padding count half), the last
// round's end a quarter of one, and a block by itself 0.62 of one.  Not by estimate: forward with a causal mask more than two heads per SM (three for narrow heads of
// which two share one), whose blocks last as long as their last rows while the others fill the gaps; backward, size 64, heads of one pass.
// Measured, 64 rows against a head, heads x tokens, forward / backward (- where a head does not fit): size 32, no mask: 288 x 150 24 - 17 / 68 - 45, 512 x 128 19 - 23 / 65 - 64,
// 288 x 200 39 - 31 / 115 - 88, 160 x 150 16 - 16 / 43 - 45; causal: 288 x 150 18.6 - 12.9 / 54 - 31, 512 x 200 44 - 46 / 143 - 125.  Size 64: 288 x 150 39 - 40 / 139 - 103,
// 288 x 200 71 - 53 / -.  Size 16 (rates of 32): 288 x 150 18.0 - 12.9 / 46 - 31; causal 13.9 - 10.9 / 37 - 21, 512 x 200 31.6 - 38.2 / 95 - 84.  Over 2900 shapes of 8 to 1000 heads and
// 17 to 512 tokens, both directions, the choice is slower than blocks of 64 rows in 0.5 %, by 17 % at most (7 us instead of 6); it takes the head's kernel in 13 %, where that is
// 1.24 times as fast on average.
template <int HD> inline bool at_head_better(const Ctx* ctx, long heads, int T, int causal, bool bwd) {
  const size_t smem = at_head_smem<HD>(T, bwd); if (smem > 227 * 1024) return false;
  constexpr bool wide = HD == 64;
  const double h0 = bwd ? (wide ? 1 : 3) : (wide ? 4 : 2.5), h1 = bwd ? (wide ? 9.6 : 6.2) : (wide ? 3.6 : 1.9), t0 = bwd ? (wide ? 7 : 5) : (wide ? 5 : 4), t1 = bwd ? (wide ? 11 : 6.7) : (wide ? 6.3 : 4);
  const int warps = at_head_warps<HD>(T), kc = at_pad(T) / 32, turns = cdiv(cdiv(T, 16), warps), nb = cdiv(T, AT_BLK);
  const bool pairs = warps <= 10 && 2 * (smem + 1024) <= 228 * 1024 && !(wide && bwd); const long n = cdiv(heads, ctx->sm_count);
  if (bwd ? wide && kc == 1 : causal && n > 2 && (wide || !pairs)) return false;
  const double u = h0 + h1 * kc * turns * (causal ? 0.5 * (kc + 1) / kc : 1.0), head = u * (pairs ? n / 2 * 1.4 + n % 2 : n);
  const double w = t0 + t1 * 0.5 * (nb + T / 64.0) * (causal ? 0.5 * (nb + 1) / nb : 1.0), rounds = (double)heads * nb * (bwd ? 2 : 1) / ((wide ? 3.0 : 4.0) * ctx->sm_count);
  return head < 0.92 * w * std::max(0.62, rounds + 0.25);
}
template <int HD>
inline int attn_head_fwd(Ctx* ctx, const float* Q, const float* K, const float* V, float* O, float* M, float* L, int B, int T, int D, int H, int causal) {
  const int smem = (int)at_head_smem<HD>(T, false), warps = at_head_warps<HD>(T); auto* kern = warps <= 10 ? attn_head_fwd_kernel<HD, 320, 2> : attn_head_fwd_kernel<HD, 512, 1>;
  GN_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GN_LAUNCH(ctx, kern, dim3(H, B), 32 * warps, smem, Q, K, V, O, M, L, T, D, H, causal, 1.f / sqrtf((float)HD));
  return check_launch("attn_head_fwd");
}
template <int HD>
inline int attn_head_bwd(Ctx* ctx, const float* Q, const float* K, const float* V, const float* O, const float* dO, const float* M, const float* L,
                         float* dQ, float* dK, float* dV, int B, int T, int D, int H, int causal) {
  const int smem = (int)at_head_smem<HD>(T, true), warps = at_head_warps<HD>(T); auto* kern = warps <= 10 ? attn_head_bwd_kernel<HD, 320, HD == 64 ? 1 : 2> : attn_head_bwd_kernel<HD, 512, 1>;
  GN_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GN_LAUNCH(ctx, kern, dim3(H, B), 32 * warps, smem, Q, K, V, O, dO, M, L, dQ, dK, dV, T, D, H, causal, 1.f / sqrtf((float)HD));
  return check_launch("attn_head_bwd");
}
enum AtKernel { AT_AUTO, AT_ROWS, AT_HEAD };                   // the kernel of the shape, blocks of 64 rows, or a block per head (the tests ask for one)
template <int HD> inline int at_choose(const Ctx* ctx, AtKernel pick, long heads, int T, int causal, bool bwd, bool* head) {
  *head = pick == AT_HEAD || (pick == AT_AUTO && at_head_better<HD>(ctx, heads, T, causal, bwd));
  return *head && at_head_smem<HD>(T, bwd) > 227 * 1024 ? fail(GN_ERR_UNSUPPORTED, "attention: a head of %d tokens, size %d, does not fit shared memory", T, HD) : GN_OK;
}
template <int HD>
inline int attn_fwd_launch(Ctx* ctx, const float* Q, const float* K, const float* V, float* O, float* M, float* L, int B, int T, int D, int H, int causal, AtKernel pick) {
  bool head; GN_TRY(at_choose<HD>(ctx, pick, (long)B * H, T, causal, false, &head));
  if (head) return attn_head_fwd<HD>(ctx, Q, K, V, O, M, L, B, T, D, H, causal);
  const int smem = 3 * AtCfg<HD>::TILE * (int)sizeof(__half) + 3 * AT_BLK * (int)sizeof(float);
  GN_CUDA(cudaFuncSetAttribute(attn_fwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GN_LAUNCH(ctx, attn_fwd_kernel<HD>, dim3(cdiv(T, AT_BLK), H, B), AT_THREADS, smem, Q, K, V, O, M, L, T, D, H, causal, 1.f / sqrtf((float)HD));
  return check_launch("attn_fwd");
}
template <int HD>
inline int attn_bwd_launch(Ctx* ctx, const float* Q, const float* K, const float* V, const float* O, const float* dO, const float* M, const float* L,
                           float* dQ, float* dK, float* dV, int B, int T, int D, int H, int causal, AtKernel pick) {
  bool head; GN_TRY(at_choose<HD>(ctx, pick, (long)B * H, T, causal, true, &head));
  if (head) return attn_head_bwd<HD>(ctx, Q, K, V, O, dO, M, L, dQ, dK, dV, B, T, D, H, causal);
  const int smem = 4 * AtCfg<HD>::TILE * (int)sizeof(__half) + 7 * AT_BLK * (int)sizeof(float);
  GN_CUDA(cudaFuncSetAttribute(attn_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GN_LAUNCH(ctx, attn_bwd_kernel<HD>, dim3(2 * cdiv(T, AT_BLK), H, B), AT_THREADS, smem, Q, K, V, O, dO, M, L, dQ, dK, dV, T, D, H, causal, 1.f / sqrtf((float)HD));
  return check_launch("attn_bwd");
}
inline int attn_fwd(Ctx* ctx, int hd, const float* Q, const float* K, const float* V, float* O, float* M, float* L, int B, int T, int D, int H, int causal, AtKernel pick = AT_AUTO) {
  if (hd == 64) return attn_fwd_launch<64>(ctx, Q, K, V, O, M, L, B, T, D, H, causal, pick);
  if (hd == 32) return attn_fwd_launch<32>(ctx, Q, K, V, O, M, L, B, T, D, H, causal, pick);
  return attn_fwd_launch<16>(ctx, Q, K, V, O, M, L, B, T, D, H, causal, pick);
}
inline int attn_bwd(Ctx* ctx, int hd, const float* Q, const float* K, const float* V, const float* O, const float* dO, const float* M, const float* L,
                    float* dQ, float* dK, float* dV, int B, int T, int D, int H, int causal, AtKernel pick = AT_AUTO) {
  if (hd == 64) return attn_bwd_launch<64>(ctx, Q, K, V, O, dO, M, L, dQ, dK, dV, B, T, D, H, causal, pick);
  if (hd == 32) return attn_bwd_launch<32>(ctx, Q, K, V, O, dO, M, L, dQ, dK, dV, B, T, D, H, causal, pick);
  return attn_bwd_launch<16>(ctx, Q, K, V, O, dO, M, L, dQ, dK, dV, B, T, D, H, causal, pick);
}

}  // namespace gn
