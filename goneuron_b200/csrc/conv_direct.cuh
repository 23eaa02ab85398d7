// conv_direct.cuh -- Conv2D with stride 1 and a 1 x 1, 3 x 3 or 5 x 5 window on the CUDA cores, all three directions, register-tiled.
//
// A convolution over a few dozen channels is a contraction of length inC k^2 (27 to a few hundred) with a few dozen output
// columns: on the tensor-core engine (conv_tc.cuh) its time goes into writing the operand planes, 9 fold for a 3 x 3 window,
// and into tiles that are mostly padding.  For 128 images of 32 x 32 x 3 -> 16 channels and 16 x 16 x 16 -> 32 a training step spent
// 390 us there; the multiply-adds themselves are 1.15 GFLOP, 16 us at the CUDA cores' fp32 rate.
#pragma once
#include <type_traits>
#include "common.cuh"
#include "conv_lstm.cuh"

namespace gn {

// dst[ch * plane + r * ld + x] = src[ch][ylo + r][xlo + x], x < ld (a multiple of four), of `nch` channels with `rows` rows each; zero
// outside the image and from channel `have` on (bare: columns from W on are left alone).  All copies of a thread are in flight at once (one after the other, a load and
// a store at a time, they were 60 us of the weight gradient); whole 16-byte pieces where the rows allow it and the
// pointer does (`aligned`: decided by the host; a first layer reads the caller's batch).
__device__ __forceinline__ void conv_stage(float* dst, int plane, int ld, const float* __restrict__ src, int nch, int have, int rows, int ylo, int H, int W, int xlo, bool aligned, bool bare = false) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5; const bool v4 = aligned && xlo == 0 && (W & 3) == 0 && (W == ld || bare);
  const int n = v4 ? W >> 2 : ld, lw = n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32, step = nw * (32 / lw), lx = lane & (lw - 1);
  int q = warp * (32 / lw) + lane / lw, ch = q / rows, r = q - ch * rows;
  for (; ch < nch;) {
    const int y = ylo + r; const bool in = ch < have && y >= 0 && y < H; const float* s = src + ((long)ch * H + y) * W + xlo; float* d = dst + ch * plane + r * ld;
    if (v4) { for (int x = lx; x < n; x += lw) { if (in) cp_async16(d + 4 * x, s + 4 * x); else *reinterpret_cast<float4*>(d + 4 * x) = make_float4(0.f, 0.f, 0.f, 0.f); } }
    else for (int x = lx; x < n; x += lw) { const bool ok = in && xlo + x >= 0 && xlo + x < W; cp_async4(d + x, ok ? s + x : src, ok); }
    for (r += step; r >= rows; r -= rows) ch++;
  }
}

// ------------------------------------------------------------------ forward and input gradient
// dst[b, d, y, x] = act( bias[d] + sum_{s, kh, kw} w(d, s, kh, kw) src[b, s, y + kh - p, x + kw - p] ), zeros outside.  Forward: w = W[d][s].
// Input gradient (BWD): src = gradient of the pre-activation, w = W[s][d] mirrored, p = K - 1 - pad.
// A thread owns 4 neighbouring pixels of RP = two rows (one, where there are few threads, or the activation is the longer part) x 4 channels and every `ks`-th source channel; a block a band of `rb` rows of one image and
// `og` groups of 4 channels, with the source rows and the weights of `icc` source channels at a time in shared memory.  What bounds it is less
// the arithmetic than everything around it: index arithmetic and uncoalesced copies on the way into shared memory, by few threads, took most
// of its time.  So the weights are copied in their own order, image rows in 16-byte pieces where the window keeps the image's size (SAME; the border is
// then left out where the pixels are read, not stored), and the input gradient's source channels are dealt out to `ks` groups of threads (by the
// shapes alone: a sample's sums are the same in every batch), whose sums meet in shared memory.  A 3 x 3 window's weights stay in registers for both rows.
// SMOOTH: an activation other than ReLU and linear (in a kernel of its own: beside it ReLU's took 2 to 3 % longer).
// One row and up to 8 channels per thread, everything copied element by element in the order of shared memory -> this, us in a recorded chain: 3 -> 16 channels, 128
// images of 32 x 32 14.3 -> 7.0; 16 -> 32, 16 x 16 forward 23.4 -> 13.4, input gradient 36.5 -> 13.2; 1 -> 24, 50 of 28 x 28 5.9 -> 4.5.
struct ConvTile { int Cs, Cd, sH, sW, dH, dW, p, rb, og, icc, qw, swp, aligned, ks; };
template <int K, bool BWD, bool SAME, int RP, bool SMOOTH>
__global__ void __launch_bounds__(256) conv_tile_kernel(const float* __restrict__ src, const float* __restrict__ W, const float* __restrict__ bias,
                                                        float* __restrict__ z, float* __restrict__ out, const ConvTile c, int act, float alpha) {
  constexpr int KK = K * K, OC = 4, HALO = (K - 1) / 2;
  extern __shared__ __align__(16) float sm[];
  const int rows = c.rb + K - 1, ocb = c.og * OC, wn = BWD ? ocb * KK : c.icc * KK | 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  float* xs = sm; float* ws = xs + c.icc * rows * c.swp;            // [icc][rows][swp]; weights [ocb][wn] (forward: icc K K of them, odd: channel groups in different banks) or [icc][wn]
  const int y0 = blockIdx.x * c.rb, b = blockIdx.y, d0 = blockIdx.z * ocb, npx = c.rb / RP * c.qw;
  const int px = tid % npx, gk = tid / npx, g = gk % c.og, kq = gk / c.og, ry = px / c.qw * RP, qx = px % c.qw; const bool live = kq < c.ks;
  const float* sb = src + (long)b * c.Cs * c.sH * c.sW;
  float acc[RP][OC][4];
#pragma unroll
  for (int r = 0; r < RP; r++)
#pragma unroll
    for (int o = 0; o < OC; o++) { acc[r][o][0] = acc[r][o][1] = acc[r][o][2] = acc[r][o][3] = 0.f; }
  for (int s0 = 0; s0 < c.Cs; s0 += c.icc) {
    const int ns = min(c.icc, c.Cs - s0);
    if (s0 > 0) __syncthreads();
    conv_stage(xs, rows * c.swp, c.swp, sb + (long)s0 * c.sH * c.sW, ns, ns, rows, y0 - c.p, c.sH, c.sW, SAME ? 0 : -c.p, c.aligned, SAME);
    for (int k = warp; k < (BWD ? ns : ocb); k += nw) {              // a warp per run of the weights
      const float* q = BWD ? W + ((long)(s0 + k) * c.Cd + d0) * KK : W + ((long)(d0 + k) * c.Cs + s0) * KK;
      const int n = BWD ? wn : ns * KK, have = BWD ? min(ocb, c.Cd - d0) * KK : d0 + k < c.Cd ? n : 0;
#pragma unroll 4
      for (int e = lane; e < n; e += 32) cp_async4(ws + k * wn + e, e < have ? q + e : W, e < have);
    }
    cp_async_wait();
    __syncthreads();
    if (live) for (int s = kq; s < ns; s += c.ks) {
      const float* xr = xs + (s * rows + ry) * c.swp + 4 * qx; const float* wr = BWD ? ws + s * wn + OC * KK * g : ws + OC * wn * g + s * KK;
      auto weight = [&](int t, int o) -> float { return BWD ? wr[o * KK + KK - 1 - t] : wr[o * wn + t]; };
      auto row = [&](int r, float (&v)[8]) {                        // v[kw + i]: source column 4 qx + i + kw - p
        const float* q = xr + r * c.swp; const float4 m = *reinterpret_cast<const float4*>(q);
        if (SAME) {
          v[HALO] = m.x; v[HALO + 1] = m.y; v[HALO + 2] = m.z; v[HALO + 3] = m.w;
          if constexpr (K == 3) { v[0] = qx > 0 ? q[-1] : 0.f; v[5] = qx + 1 < c.qw ? q[4] : 0.f; }
          if constexpr (K == 5) {
            const float2 zero = make_float2(0.f, 0.f), l = qx > 0 ? *reinterpret_cast<const float2*>(q - 2) : zero, h = qx + 1 < c.qw ? *reinterpret_cast<const float2*>(q + 4) : zero;
            v[0] = l.x; v[1] = l.y; v[6] = h.x; v[7] = h.y;
          }
        } else {
          v[0] = m.x; v[1] = m.y; v[2] = m.z; v[3] = m.w;
          if (K > 1) *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(q + 4);
        }
      };
      float w[K == 5 ? K : KK][OC];
      if constexpr (K < 5) {
#pragma unroll
        for (int t = 0; t < KK; t++)
#pragma unroll
          for (int o = 0; o < OC; o++) w[t][o] = weight(t, o);
      }
#pragma unroll
      for (int r = 0; r < K + RP - 1; r++) {
        float v[8]; row(r, v);
#pragma unroll
        for (int k = 0; k < RP; k++) if (r - k >= 0 && r - k < K) {
#pragma unroll
          for (int kw = 0; kw < K; kw++) {
            const int t = (r - k) * K + kw;
#pragma unroll
            for (int o = 0; o < OC; o++) {
              const float wv = K < 5 ? w[K < 5 ? t : 0][o] : weight(t, o);
#pragma unroll
              for (int i = 0; i < 4; i++) acc[k][o][i] = fmaf(wv, v[kw + i], acc[k][o][i]);
            }
          }
        }
      }
    }
  }
  auto place = [&](int r, int o, long& at) -> bool {                 // where a thread's four pixels of row r, channel o go
    const int y = y0 + ry + r, d = d0 + OC * g + o; at = (((long)b * c.Cd + d) * c.dH + y) * c.dW + 4 * qx; return y < c.dH && d < c.Cd;
  };
  auto put = [&](float* p, long at, const float (&v)[4]) {
    if ((c.dW & 3) == 0) *reinterpret_cast<float4*>(p + at) = make_float4(v[0], v[1], v[2], v[3]);
    else {
#pragma unroll
      for (int i = 0; i < 4; i++) if (4 * qx + i < c.dW) p[at + i] = v[i];
    }
  };
  if constexpr (BWD) {
    if (c.ks > 1) {                                                  // the groups' sums, in order; every group finishes a share of the rows and channels
      const int all = npx * c.og, at = tid - kq * all;
      __syncthreads();
      if (live) {
#pragma unroll
        for (int e = 0; e < RP * OC * 4; e++) sm[(kq * RP * OC * 4 + e) * all + at] = acc[e / (OC * 4)][e / 4 % OC][e % 4];
      }
      __syncthreads();
      if (live) for (int q = kq; q < RP * OC; q += c.ks) {
        float v[4] = {0.f, 0.f, 0.f, 0.f}; long o;
        for (int k = 0; k < c.ks; k++) {
#pragma unroll
          for (int i = 0; i < 4; i++) v[i] += sm[(k * RP * OC * 4 + q * 4 + i) * all + at];
        }
        if (place(q / OC, q % OC, o)) put(out, o, v);
      }
      return;
    }
  }
  if (live) {
#pragma unroll
    for (int o = 0; o < OC; o++) {
      const int d = d0 + OC * g + o; const float bv = bias && d < c.Cd ? bias[d] : 0.f;
#pragma unroll
      for (int r = 0; r < RP; r++) {
#pragma unroll
        for (int i = 0; i < 4; i++) acc[r][o][i] += bv;
        if constexpr (SMOOTH) { long at; if (z && place(r, o, at)) put(z, at, acc[r][o]); }
      }
    }
  }
  if constexpr (SMOOTH) {
    // Through shared memory into a loop with one copy of each activation's code, four or eight values side by side.  (32 inlined copies of all of them, run once, came
    // from a cold instruction cache: ReLU took 14 us instead of 9 for 128 images of 32 x 32, 3 -> 16 channels.)
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int e = 0; e < RP * OC * 4; e++) sm[e * blockDim.x + tid] = acc[e / (OC * 4)][e / 4 % OC][e % 4];
    auto apply = [&](auto kind) {
#pragma unroll 1
      for (int o = 0; o < OC; o++) {
        float v[RP][4]; long at;
#pragma unroll
        for (int e = 0; e < RP * 4; e++) v[e / 4][e % 4] = act_fwd(decltype(kind)::value, sm[((e / 4 * OC + o) * 4 + e % 4) * blockDim.x + tid], alpha);
#pragma unroll
        for (int r = 0; r < RP; r++) if (place(r, o, at)) put(out, at, v[r]);
      }
    };
    switch (act) {
      case GN_ACT_SIGMOID: apply(std::integral_constant<int, GN_ACT_SIGMOID>{}); break;
      case GN_ACT_TANH: apply(std::integral_constant<int, GN_ACT_TANH>{}); break;
      case GN_ACT_LEAKY_RELU: apply(std::integral_constant<int, GN_ACT_LEAKY_RELU>{}); break;
      case GN_ACT_ELU: apply(std::integral_constant<int, GN_ACT_ELU>{}); break;
      case GN_ACT_GELU: apply(std::integral_constant<int, GN_ACT_GELU>{}); break;
      case GN_ACT_SILU: apply(std::integral_constant<int, GN_ACT_SILU>{}); break;
      default: apply(std::integral_constant<int, GN_ACT_LINEAR>{});
    }
    return;
  }
  if (!live) return;
#pragma unroll
  for (int q = 0; q < RP * OC; q++) {
    float (&v)[4] = acc[q / OC][q % OC]; long at;
    if (act == GN_ACT_RELU) {
#pragma unroll
      for (int i = 0; i < 4; i++) v[i] = v[i] > 0.f ? v[i] : 0.f;
    }
    if (place(q / OC, q % OC, at)) put(out, at, v);
  }
}

// ------------------------------------------------------------------ weight and bias gradient
// dW[o, s, kh, kw] = sum_{b, y, x} g[b, o, y, x] src[b, s, y + kh - p, x + kw - p].  A thread owns OT output channels x one input channel x all
// taps and walks the rows y = pg (mod PG) of a band, four pixels at a time: K 2 + OT 16-byte shared loads per 4 OT K^2
// multiply-adds.  A block takes the bands of several images in turn (unit = image, band) and leaves one set of partial sums;
// conv_wgrad_tile_final_kernel adds the blocks' sets in order.  Channel planes in shared memory lie 4 (mod 8) floats apart, so that
// the lanes of a warp (neighbouring channels) hit different banks.
struct ConvWg { int Cs, Cd, H, W, oH, oW, p, rb, bands, ocb, icb, pg, swp, gwp, xplane, gplane, units, aligned; };
template <int K> struct ConvWgOT { static constexpr int v = K == 1 ? 8 : K == 3 ? 4 : 2; };
template <int K>
__global__ void __launch_bounds__(256) conv_wgrad_tile_kernel(const float* __restrict__ g, const float* __restrict__ src, float* __restrict__ part, const ConvWg c) {
  constexpr int OT = ConvWgOT<K>::v, KK = K * K;
  extern __shared__ __align__(16) float sm[];
  float* xs = sm; float* gs = xs + c.icb * c.xplane;                // [icb][rb + K - 1][swp], [ocb][rb][gwp]
  const int tid = threadIdx.x, rows = c.rb + K - 1;
  const int ict = (c.Cs + c.icb - 1) / c.icb, i0 = (blockIdx.y % ict) * c.icb, o0 = (blockIdx.y / ict) * c.ocb;
  const int items = (c.ocb / OT) * c.icb, it = tid % items, pg = tid / items, ic = it % c.icb, oq = it / c.icb; const bool live = pg < c.pg;
  float acc[OT][KK], sb[OT];
#pragma unroll
  for (int o = 0; o < OT; o++) {
    sb[o] = 0.f;
#pragma unroll
    for (int t = 0; t < KK; t++) acc[o][t] = 0.f;
  }
  for (int u = blockIdx.x; u < c.units; u += gridDim.x) {
    const int b = u / c.bands, y0 = (u - b * c.bands) * c.rb, nr = min(c.rb, c.oH - y0);
    __syncthreads();
    conv_stage(xs, c.xplane, c.swp, src + ((long)b * c.Cs + i0) * c.H * c.W, c.icb, c.Cs - i0, rows, y0 - c.p, c.H, c.W, -c.p, c.aligned);
    conv_stage(gs, c.gplane, c.gwp, g + ((long)b * c.Cd + o0) * c.oH * c.oW, c.ocb, c.Cd - o0, c.rb, y0, c.oH, c.oW, 0, true);
    cp_async_wait();
    __syncthreads();
    if (live) for (int r = pg; r < nr; r += c.pg) {
      const float* xr = xs + ic * c.xplane + r * c.swp; const float* gr = gs + oq * OT * c.gplane + r * c.gwp;
      for (int x = 0; x < c.gwp; x += 4) {
        float gv[OT][4];
#pragma unroll
        for (int o = 0; o < OT; o++) { *reinterpret_cast<float4*>(gv[o]) = *reinterpret_cast<const float4*>(gr + o * c.gplane + x); sb[o] += (gv[o][0] + gv[o][1]) + (gv[o][2] + gv[o][3]); }
#pragma unroll
        for (int kh = 0; kh < K; kh++) {
          float v[8];
          *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(xr + kh * c.swp + x);
          if (K > 1) *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(xr + kh * c.swp + x + 4);
#pragma unroll
          for (int kw = 0; kw < K; kw++)
#pragma unroll
            for (int o = 0; o < OT; o++)
#pragma unroll
              for (int i = 0; i < 4; i++) acc[o][kh * K + kw] = fmaf(gv[o][i], v[kw + i], acc[o][kh * K + kw]);
        }
      }
    }
  }
  // the pixel groups' sums, in order, through shared memory
  constexpr int NV = OT * (KK + 1); const int all = items * c.pg; float* prow = part + ((long)blockIdx.x * gridDim.y + blockIdx.y) * items * NV;
  float* red = sm;                                                   // [NV][pg][items]
  __syncthreads();
  if (live) {
#pragma unroll
    for (int o = 0; o < OT; o++) {
#pragma unroll
      for (int t = 0; t < KK; t++) red[(o * (KK + 1) + t) * all + tid] = acc[o][t];
      red[(o * (KK + 1) + KK) * all + tid] = sb[o];
    }
  }
  __syncthreads();
  auto sum = [&](int v, int q) { float a = 0.f; for (int k = 0; k < c.pg; k++) a += red[v * all + k * items + q]; prow[v * items + q] = a; };      // (in the order of the threads; the kernel below finds the places)
  if (2 * all > (int)blockDim.x) { if (live) for (int v = pg; v < NV; v += c.pg) sum(v, it); }
  else for (int e = tid; e < items * NV; e += blockDim.x) sum(e / items, e % items);      // (few items: all threads add up)
}
// dst[i] = sum over the blocks' sets, in order: 32 elements x 8 groups of sets per block (weights, then biases: the gradient slice is laid out W | b)
__global__ void __launch_bounds__(256) conv_wgrad_final_kernel(const float* __restrict__ part, int sets, int n, float* __restrict__ dst) {
  __shared__ float red[8][33];
  const int tx = threadIdx.x & 31, grp = threadIdx.x >> 5, i = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (i < n) {
#pragma unroll 8
    for (int k = grp; k < sets; k += 8) s += part[(long)k * n + i];
  }
  red[grp][tx] = s;
  __syncthreads();
  if (grp == 0 && i < n) {
    for (int k = 1; k < 8; k++) s += red[k][tx];
    dst[i] = s;
  }
}
// The same for the sets of conv_wgrad_tile_kernel; an element's place in a set: channel tile, OT x (taps, bias), item.
template <int K>
__global__ void __launch_bounds__(256) conv_wgrad_tile_final_kernel(const float* __restrict__ part, int sets, int n, float* __restrict__ dst, const ConvWg c) {
  constexpr int OT = ConvWgOT<K>::v, KK = K * K, NV = OT * (KK + 1);
  __shared__ float red[8][33];
  const int tx = threadIdx.x & 31, grp = threadIdx.x >> 5, i = blockIdx.x * 32 + tx, items = c.ocb / OT * c.icb;
  float s = 0.f;
  if (i < n) {
#pragma unroll 8
    for (int k = grp; k < sets; k += 8) s += part[(long)k * n + i];
  }
  red[grp][tx] = s;
  __syncthreads();
  if (grp > 0 || i >= n) return;
  const int tile = i / (items * NV), e = i - tile * items * NV, v = e / items, q = e - v * items, ict = (c.Cs + c.icb - 1) / c.icb;
  const int o = v / (KK + 1), t = v - o * (KK + 1), d = tile / ict * c.ocb + q / c.icb * OT + o, s_ = tile % ict * c.icb + q % c.icb;
  if (d >= c.Cd || s_ >= c.Cs || (t == KK && s_ > 0)) return;
  for (int k = 1; k < 8; k++) s += red[k][tx];
  dst[t < KK ? ((long)d * c.Cs + s_) * KK + t : (long)c.Cd * c.Cs * KK + d] = s;
}

// ------------------------------------------------------------------ host side
constexpr size_t CD_SMEM = 96 * 1024;
inline bool conv_direct_supported(const ConvShape& c) {
  if (!(c.s == 1 && (c.k == 1 || c.k == 3 || c.k == 5) && c.p >= 0 && c.p < c.k && c.oH > 0 && c.oW > 0 && c.B <= 65535)) return false;
  return c.W <= 512 && c.oW <= 512;                                 // (four rows of an image and a few channels have to fit shared memory)
}
// Up to here the multiply-adds cost less than the tensor-core engine's operand planes.  Forward / weight / input gradient of 128
// images of 16 x 16 pixels, 3 x 3 window, direct against tensor cores: 64 -> 64 channels 123 / 121 / 113 us against 140 / 269 / 143;
// 64 -> 128: 219 / 217 / 218 against 147 / 312 / 271; 128 -> 128: 427 / 379 / 422 against 270 / 571 / 274.
inline bool conv_direct_preferred(const ConvShape& c) { return conv_direct_supported(c) && (long)c.inC * c.outC * c.k * c.k <= 64L * 96 * 9; }

// Input gradients: source channels in up to four groups of threads while a block still has three groups of two rows (or all): by the shapes alone.  us with 1 / 2 / 4: 16 -> 32
// channels, 128 images of 16 x 16 17.0 / 14.2 / 13.2; 32 -> 64, 64 of 20 x 20 43 / 41 / 48; 16 -> 64, 20 of 16 x 16 30 / 21 / 15.  Forward in one group: a block has
// enough threads there (13.4 / - / 15.3), and ReLU and pooling see sums in the order of the channels.
inline int conv_dgrad_groups(const ConvTile& c) {
  int ks = c.Cs >= 16 ? 4 : c.Cs >= 8 ? 2 : 1; const int qw = cdiv(c.dW, 4), groups = cdiv(c.Cd, 4);
  while (ks > 1 && 256 / ks < qw * std::min(groups, 8) * std::min((int)cdiv(c.dH, 2), 3)) ks /= 2;
  return ks;
}
template <int K, bool BWD, bool SAME, int RP, bool SMOOTH>
inline int conv_tile_run(Ctx* ctx, int B, ConvTile c, const float* src, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  constexpr int OC = 4;
  c.qw = cdiv(c.dW, 4); c.swp = SAME ? c.sW : 4 * c.qw + (K > 1 ? 4 : 0);
  if (SAME && (c.qw == 2 || c.qw == 4)) while (RP * c.swp % 32 != 4 * c.qw) c.swp += 4;      // neighbouring rows of threads in neighbouring banks
  const int groups = cdiv(c.Cd, OC), row_groups = cdiv(c.dH, RP);                 // groups of two rows
  c.ks = BWD ? conv_dgrad_groups(c) : 1;
  const int most = 256 / c.ks;
  c.og = std::min(groups, std::max(1, std::min(32 / OC, most / c.qw)));
  int rg = std::max(1, std::min(row_groups, most / (c.qw * c.og)));
  if (RP == 1) {
    // the busiest SM's rows, with one and a half per block for what a block costs by itself (100 images of 28 x 28, 1 -> 12 channels, tanh: 300 blocks of 10 rows
    // 11.2 us, 400 of 7 8.8)
    auto cost = [&](int r) { return cdiv((long)B * cdiv(row_groups, r) * cdiv(groups, c.og), ctx->sm_count) * (r + 1.5); };
    for (int r = rg - 1; r >= 1 && r * c.qw * c.og * c.ks >= 64; r--) if (cost(r) < cost(rg)) rg = r;
  } else
  // three blocks for two SMs at least (one each: 13 % slower for 50 images of 28 x 28, three each: 14 % for 16 -> 32 channels)
  while (rg > 1 && rg * c.qw * c.og * c.ks > 64 && 2L * B * cdiv(row_groups, rg) * cdiv(groups, c.og) < 3L * ctx->sm_count) rg = (rg + 1) / 2;
  rg = cdiv(row_groups, cdiv(row_groups, rg));                       // even bands
  c.rb = rg * RP;
  const size_t per = ((size_t)(c.rb + K - 1) * c.swp + (size_t)K * K * c.og * OC) * sizeof(float);
  c.icc = std::max<int>(1, std::min<int>(c.Cs, 48 * 1024 / per));
  if (c.icc < c.Cs) c.icc = std::max(c.ks, c.icc / c.ks * c.ks);     // (a channel's group of threads does not depend on how many are staged at once)
  const int all = c.qw * rg * c.og, threads = (all * c.ks + 31) & ~31;
  const size_t smem = std::max(c.icc * per + (size_t)c.og * OC * sizeof(float), (size_t)(c.ks > 1 ? c.ks * all : SMOOTH ? threads : 0) * RP * OC * 4 * sizeof(float));
  GN_CUDA(cudaFuncSetAttribute(conv_tile_kernel<K, BWD, SAME, RP, SMOOTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, (conv_tile_kernel<K, BWD, SAME, RP, SMOOTH>), dim3(cdiv(c.dH, c.rb), B, cdiv(groups, c.og)), threads, smem, src, W, bias, z, out, c, act, alpha);
  return check_launch("conv_tile");
}
template <int K, bool BWD>
inline int conv_tile_launch(Ctx* ctx, int B, ConvTile c, const float* src, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  c.aligned = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  const bool same = c.aligned && c.sW % 4 == 0 && c.dW == c.sW && 2 * c.p == K - 1;
  if constexpr (!BWD) {
    if (act != GN_ACT_RELU && act != GN_ACT_LINEAR) {
      // One row per thread, unless there are enough threads for two and the sums are the longer part.  us with two / one rows, tanh: 1 -> 24 channels, 50 images of 28 x 28
      // 11.3 / 8.6; 24 -> 24, 64 of 30 x 30, 1 x 1 26.5 / 18.3; 32 -> 64, 128 of 8 x 8 28.1 / 19.4; 3 -> 32, 64 of 40 x 40 30.2 / 27.9; 16 -> 32, 128 of 16 x 16 20.2 / 18.9, 256 29.4 / 33.5; 24 -> 24, 64 of 32 x 32 32.1 / 43.2.
      const bool two = c.Cs * K * K >= 72 && (long)B * cdiv(c.dH, 2) * cdiv(c.dW, 4) * cdiv(c.Cd, 4) > 260L * ctx->sm_count;
      if (two) return same ? conv_tile_run<K, BWD, true, 2, true>(ctx, B, c, src, W, bias, z, out, act, alpha) : conv_tile_run<K, BWD, false, 2, true>(ctx, B, c, src, W, bias, z, out, act, alpha);
      return same ? conv_tile_run<K, BWD, true, 1, true>(ctx, B, c, src, W, bias, z, out, act, alpha) : conv_tile_run<K, BWD, false, 1, true>(ctx, B, c, src, W, bias, z, out, act, alpha);
    }
  }
  if constexpr (BWD) {
    // One row per thread where there are few threads (fewer where rows come in 16-byte pieces: 3 -> 26, 120 of 28 x 28 14.9 with one row, 13.1 with two), or nothing that
    // two rows share (1 x 1 windows, unless rows come in 16-byte pieces).  us with two / one: 16 -> 64 channels, 20
    // images of 16 x 16, 3 x 3 15.1 / 11.7, 1 x 1 9.8 / 5.6; 24 -> 24, 64 of 30 x 30 39.9 / 31.0, 1 x 1 14.1 / 10.5; 16 -> 32, 128 of 16 x 16 12.9 / 15.9; 32 -> 64, 64 of 20 x 20 40.6 / 48.8.
    const bool two = (K > 1 || same) && (long)B * cdiv(c.dH, 2) * cdiv(c.dW, 4) * cdiv(c.Cd, 4) * conv_dgrad_groups(c) > (same ? 300L : 320L) * ctx->sm_count;
    if (!two) return same ? conv_tile_run<K, BWD, true, 1, false>(ctx, B, c, src, W, bias, z, out, act, alpha) : conv_tile_run<K, BWD, false, 1, false>(ctx, B, c, src, W, bias, z, out, act, alpha);
  }
  return same ? conv_tile_run<K, BWD, true, 2, false>(ctx, B, c, src, W, bias, z, out, act, alpha) : conv_tile_run<K, BWD, false, 2, false>(ctx, B, c, src, W, bias, z, out, act, alpha);
}
// z may be null (LINEAR, RELU)
inline int conv_direct_forward(Ctx* ctx, const ConvShape& s, const float* x, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  ConvTile c{s.inC, s.outC, s.H, s.W, s.oH, s.oW, s.p};
  if (s.k == 1) return conv_tile_launch<1, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
  if (s.k == 3) return conv_tile_launch<3, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
  return conv_tile_launch<5, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
}
inline int conv_direct_dgrad(Ctx* ctx, const ConvShape& s, const float* g, const float* W, float* dx) {
  ConvTile c{s.outC, s.inC, s.oH, s.oW, s.H, s.W, s.k - 1 - s.p};
  if (s.k == 1) return conv_tile_launch<1, true>(ctx, s.B, c, g, W, nullptr, nullptr, dx, GN_ACT_LINEAR, 0.f);
  if (s.k == 3) return conv_tile_launch<3, true>(ctx, s.B, c, g, W, nullptr, nullptr, dx, GN_ACT_LINEAR, 0.f);
  return conv_tile_launch<5, true>(ctx, s.B, c, g, W, nullptr, nullptr, dx, GN_ACT_LINEAR, 0.f);
}
inline ConvWg conv_wgrad_plan(Ctx* ctx, const ConvShape& s, int OT, int* sets, size_t* smem) {
  ConvWg c{s.inC, s.outC, s.H, s.W, s.oH, s.oW, s.p};
  c.gwp = (s.oW + 3) & ~3; c.swp = c.gwp + (s.k > 1 ? 4 : 0);
  const int og = cdiv(s.outC, OT);
  c.icb = std::min(s.inC, 32); c.ocb = std::min(og, std::max(1, 256 / c.icb)) * OT;
  auto plane = [](int n) { return ((n + 3) & ~7) + 4; };            // >= n, 4 (mod 8)
  auto bytes = [&](int rb) { return ((size_t)c.icb * plane((rb + s.k - 1) * c.swp) + (size_t)c.ocb * plane(rb * c.gwp)) * sizeof(float); };
  c.rb = s.oH; while (c.rb > 1 && bytes(c.rb) > CD_SMEM) c.rb--;
  while (bytes(c.rb) > CD_SMEM && c.icb > 1) c.icb = (c.icb + 1) / 2;
  while (bytes(c.rb) > CD_SMEM && c.ocb > OT) c.ocb = std::max(OT, c.ocb / 2 / OT * OT);
  const long tiles = (long)cdiv(s.inC, c.icb) * cdiv(s.outC, c.ocb);
  c.bands = cdiv(s.oH, c.rb);
  if ((long)s.B * c.bands * tiles < ctx->sm_count) {                 // few images: shorter bands, more blocks
    const int want = std::max<int>(1, std::min<long>(s.oH, ctx->sm_count / std::max<long>(1, s.B * tiles)));
    c.rb = std::min(c.rb, (int)cdiv(s.oH, want)); c.bands = cdiv(s.oH, c.rb);
  }
  c.rb = cdiv(s.oH, c.bands);                                        // even bands (a short last one takes a block as well: 3 -> 32 channels, 64 images of 40 x 40 24.2 -> 20.7 us, 32 -> 64, 20 x 20 63.9 -> 45.0)
  c.xplane = plane((c.rb + s.k - 1) * c.swp); c.gplane = plane(c.rb * c.gwp);
  const int items = c.ocb / OT * c.icb; c.pg = std::max(1, std::min(c.rb, 256 / items));
  c.units = s.B * c.bands;
  *sets = (int)std::min<long>(c.units, std::max<long>(1, 2L * ctx->sm_count / tiles));
  *smem = std::max(bytes(c.rb), (size_t)items * c.pg * OT * (s.k * s.k + 1) * sizeof(float));
  return c;
}
inline size_t conv_wgrad_part_floats(Ctx* ctx, const ConvShape& s) {
  const int OT = s.k == 1 ? 8 : s.k == 3 ? 4 : 2; int sets; size_t smem; const ConvWg c = conv_wgrad_plan(ctx, s, OT, &sets, &smem);
  return (size_t)sets * cdiv(s.inC, c.icb) * cdiv(s.outC, c.ocb) * c.icb * c.ocb * (s.k * s.k + 1);
}
template <int K>
inline int conv_wgrad_launch(Ctx* ctx, const ConvShape& s, const float* g, const float* x, float* part, float* gW) {
  constexpr int OT = ConvWgOT<K>::v; int sets; size_t smem;
  ConvWg c = conv_wgrad_plan(ctx, s, OT, &sets, &smem); c.aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int items = c.ocb / OT * c.icb, threads = (items * c.pg + 31) & ~31, tiles = cdiv(s.inC, c.icb) * cdiv(s.outC, c.ocb), n = tiles * items * OT * (K * K + 1);
  GN_CUDA(cudaFuncSetAttribute(conv_wgrad_tile_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, conv_wgrad_tile_kernel<K>, dim3(sets, tiles), threads, smem, g, x, part, c);
  GN_LAUNCH(ctx, conv_wgrad_tile_final_kernel<K>, cdiv(n, 32), 256, 0, (const float*)part, sets, n, gW, c);
  return check_launch("conv_wgrad");
}
// weight and bias gradients (gb follows gW); `part`: conv_wgrad_part_floats
inline int conv_direct_wgrad(Ctx* ctx, const ConvShape& s, const float* g, const float* x, float* part, float* gW) {
  if (s.k == 1) return conv_wgrad_launch<1>(ctx, s, g, x, part, gW);
  if (s.k == 3) return conv_wgrad_launch<3>(ctx, s, g, x, part, gW);
  return conv_wgrad_launch<5>(ctx, s, g, x, part, gW);
}

}  // namespace gn
