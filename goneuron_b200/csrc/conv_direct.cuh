// conv_direct.cuh -- Conv2D with stride 1 and a 1 x 1, 3 x 3 or 5 x 5 window on the CUDA cores, all three directions, register-tiled.
//
// A convolution over a few dozen channels is a contraction of length inC k^2 (27 to a few hundred) with a few dozen output
// columns: on the tensor-core engine (conv_tc.cuh) its time goes into writing the operand planes, 9 fold for a 3 x 3 window,
// and into tiles that are mostly padding.  For 128 images of 32 x 32 x 3 -> 16 channels and 16 x 16 x 16 -> 32 a training step spent
// 390 us there; the multiply-adds themselves are 1.15 GFLOP, 16 us at the CUDA cores' fp32 rate.
#pragma once
#include "common.cuh"
#include "conv_lstm.cuh"

namespace gn {

// dst[ch * plane + r * ld + x] = src[ch][ylo + r][xlo + x], x < ld (a multiple of four), of `nch` channels with `rows` rows each; zero
// outside the image and from channel `have` on.  All copies of a thread are in flight at once (one after the other, a load and
// a store at a time, they were 60 us of the weight gradient); whole 16-byte pieces where the rows allow it and the
// pointer does (`aligned`: decided by the host; a first layer reads the caller's batch).
__device__ __forceinline__ void conv_stage(float* dst, int plane, int ld, const float* __restrict__ src, int nch, int have, int rows, int ylo, int H, int W, int xlo, bool aligned) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5; const bool v4 = aligned && xlo == 0 && ld == W;      // W a multiple of four
  const int n = v4 ? ld >> 2 : ld, lw = n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32, step = nw * (32 / lw), lx = lane & (lw - 1);
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
// A thread owns 4 neighbouring pixels x OC = 8 (or 4) channels; a block a band of `rb` rows of one image and `og` groups of OC
// channels, with the source rows and the weights of `icc` source channels at a time in shared memory: 2 + 2 K 16-byte shared
// loads per 32 K multiply-adds.
struct ConvTile { int Cs, Cd, sH, sW, dH, dW, p, rb, og, icc, qw, swp, aligned; };
template <int K, int OC, bool BWD>
__global__ void __launch_bounds__(256) conv_tile_kernel(const float* __restrict__ src, const float* __restrict__ W, const float* __restrict__ bias,
                                                        float* __restrict__ z, float* __restrict__ out, const ConvTile c, int act, float alpha) {
  extern __shared__ __align__(16) float sm[];
  const int rows = c.rb + K - 1, ocb = c.og * OC, tid = threadIdx.x;
  float* xs = sm; float* ws = xs + c.icc * rows * c.swp;            // [icc][rows][swp], [icc][K K][ocb]
  const int y0 = blockIdx.x * c.rb, b = blockIdx.y, d0 = blockIdx.z * ocb;
  const int px = tid % (c.rb * c.qw), g = tid / (c.rb * c.qw), ry = px / c.qw, qx = px - ry * c.qw; const bool live = g < c.og;
  const float* sb = src + (long)b * c.Cs * c.sH * c.sW;
  float acc[OC][4];
#pragma unroll
  for (int o = 0; o < OC; o++) { acc[o][0] = acc[o][1] = acc[o][2] = acc[o][3] = 0.f; }
  for (int s0 = 0; s0 < c.Cs; s0 += c.icc) {
    const int ns = min(c.icc, c.Cs - s0);
    if (s0 > 0) __syncthreads();
    conv_stage(xs, rows * c.swp, c.swp, sb + (long)s0 * c.sH * c.sW, ns, ns, rows, y0 - c.p, c.sH, c.sW, -c.p, c.aligned);
    for (int e = tid; e < ocb * ns * K * K; e += blockDim.x) {
      const int o = e % ocb, r = e / ocb, t = r % (K * K), s = r / (K * K);      // neighbouring threads, neighbouring words of shared memory
      const bool in = d0 + o < c.Cd;
      const float* wp = BWD ? W + ((long)(s0 + s) * c.Cd + d0 + o) * (K * K) + (K * K - 1 - t) : W + ((long)(d0 + o) * c.Cs + s0 + s) * (K * K) + t;
      cp_async4(ws + (s * K * K + t) * ocb + o, in ? wp : W, in);
    }
    cp_async_wait();
    __syncthreads();
    if (live) for (int s = 0; s < ns; s++) {
#pragma unroll
      for (int kh = 0; kh < K; kh++) {
        const float* xr = xs + (s * rows + ry + kh) * c.swp + 4 * qx;
        float v[8];
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(xr);
        if (K > 1) *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(xr + 4);
#pragma unroll
        for (int kw = 0; kw < K; kw++) {
          const float* wr = ws + (s * K * K + kh * K + kw) * ocb + OC * g;
          float wv[OC];
#pragma unroll
          for (int o = 0; o < OC; o += 4) *reinterpret_cast<float4*>(wv + o) = *reinterpret_cast<const float4*>(wr + o);
#pragma unroll
          for (int o = 0; o < OC; o++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[o][i] = fmaf(wv[o], v[kw + i], acc[o][i]);
        }
      }
    }
  }
  const int y = y0 + ry;
  if (!live || y >= c.dH) return;
#pragma unroll
  for (int o = 0; o < OC; o++) {
    const int d = d0 + OC * g + o; if (d >= c.Cd) break;
    const float bv = bias ? bias[d] : 0.f; const long at = (((long)b * c.Cd + d) * c.dH + y) * c.dW + 4 * qx;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = acc[o][i] + bv;
    if (z) {
#pragma unroll
      for (int i = 0; i < 4; i++) if (4 * qx + i < c.dW) z[at + i] = v[i];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = act_fwd(act, v[i], alpha);
    if ((c.dW & 3) == 0) *reinterpret_cast<float4*>(out + at) = make_float4(v[0], v[1], v[2], v[3]);
    else {
#pragma unroll
      for (int i = 0; i < 4; i++) if (4 * qx + i < c.dW) out[at + i] = v[i];
    }
  }
}

// ------------------------------------------------------------------ weight and bias gradient
// dW[o, s, kh, kw] = sum_{b, y, x} g[b, o, y, x] src[b, s, y + kh - p, x + kw - p].  A thread owns OT output channels x one input channel x all
// taps and walks the rows y = pg (mod PG) of a band, four pixels at a time: K 2 + OT 16-byte shared loads per 4 OT K^2
// multiply-adds.  A block takes the bands of several images in turn (unit = image, band) and leaves one set of partial sums;
// conv_wgrad_final_kernel adds the blocks' sets in order.  Channel planes in shared memory lie 4 (mod 8) floats apart, so that
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
  constexpr int NV = OT * (KK + 1); const int nW = c.Cd * c.Cs * KK, all = items * c.pg; float* prow = part + (long)blockIdx.x * (nW + c.Cd);
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
  for (int e = tid; e < items * NV; e += blockDim.x) {
    const int q = e % items, v = e / items, o = v / (KK + 1), t = v - o * (KK + 1), d = o0 + (q / c.icb) * OT + o, s = i0 + q % c.icb;
    if (d >= c.Cd || s >= c.Cs || (t == KK && s > 0)) continue;
    float a = 0.f;
    for (int k = 0; k < c.pg; k++) a += red[v * all + k * items + q];
    prow[t < KK ? ((long)d * c.Cs + s) * KK + t : (long)nW + d] = a;
  }
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

template <int K, int OC, bool BWD>
inline int conv_tile_run(Ctx* ctx, int B, ConvTile c, const float* src, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  c.aligned = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  c.qw = cdiv(c.dW, 4); c.swp = 4 * c.qw + (K > 1 ? 4 : 0);
  const int groups = cdiv(c.Cd, OC);
  c.og = std::min(groups, std::max(1, std::min(32 / OC, 256 / c.qw)));
  c.rb = std::max(1, std::min(c.dH, 256 / (c.qw * c.og)));
  // at least three blocks per SM, so that one computes while another's copies are under way
  while (c.rb > 1 && c.rb * c.qw * c.og > 64 && (long)B * cdiv(c.dH, c.rb) * cdiv(groups, c.og) < 3L * ctx->sm_count) c.rb = (c.rb + 1) / 2;
  const size_t per = ((size_t)(c.rb + K - 1) * c.swp + (size_t)K * K * c.og * OC) * sizeof(float);
  c.icc = std::max<int>(1, std::min<int>(c.Cs, 48 * 1024 / per));
  const size_t smem = c.icc * per; const int threads = (c.qw * c.rb * c.og + 31) & ~31;
  GN_CUDA(cudaFuncSetAttribute(conv_tile_kernel<K, OC, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, (conv_tile_kernel<K, OC, BWD>), dim3(cdiv(c.dH, c.rb), B, cdiv(groups, c.og)), threads, smem, src, W, bias, z, out, c, act, alpha);
  return check_launch("conv_tile");
}
template <int K, bool BWD>
inline int conv_tile_launch(Ctx* ctx, int B, const ConvTile& c, const float* src, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  // four channels per thread where eight would not give every SM sub-partition three warps (or where there are no more)
  const long warps = (long)B * c.dH * cdiv(c.dW, 4) * cdiv(c.Cd, 8) / 32;
  if (c.Cd <= 4 || warps < 12L * ctx->sm_count) return conv_tile_run<K, 4, BWD>(ctx, B, c, src, W, bias, z, out, act, alpha);
  return conv_tile_run<K, 8, BWD>(ctx, B, c, src, W, bias, z, out, act, alpha);
}
// z may be null (LINEAR, RELU)
inline int conv_direct_forward(Ctx* ctx, const ConvShape& s, const float* x, const float* W, const float* bias, float* z, float* out, int act, float alpha) {
  const ConvTile c{s.inC, s.outC, s.H, s.W, s.oH, s.oW, s.p};
  if (s.k == 1) return conv_tile_launch<1, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
  if (s.k == 3) return conv_tile_launch<3, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
  return conv_tile_launch<5, false>(ctx, s.B, c, x, W, bias, z, out, act, alpha);
}
inline int conv_direct_dgrad(Ctx* ctx, const ConvShape& s, const float* g, const float* W, float* dx) {
  const ConvTile c{s.outC, s.inC, s.oH, s.oW, s.H, s.W, s.k - 1 - s.p};
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
  c.xplane = plane((c.rb + s.k - 1) * c.swp); c.gplane = plane(c.rb * c.gwp);
  const int items = c.ocb / OT * c.icb; c.pg = std::max(1, std::min(c.rb, 256 / items));
  c.units = s.B * c.bands;
  *sets = (int)std::min<long>(c.units, std::max<long>(1, 2L * ctx->sm_count / tiles));
  *smem = std::max(bytes(c.rb), (size_t)items * c.pg * OT * (s.k * s.k + 1) * sizeof(float));
  return c;
}
inline size_t conv_wgrad_part_floats(Ctx* ctx, const ConvShape& s) {
  int sets; size_t smem; conv_wgrad_plan(ctx, s, s.k == 1 ? 8 : s.k == 3 ? 4 : 2, &sets, &smem);
  return (size_t)sets * ((size_t)s.outC * s.inC * s.k * s.k + s.outC);
}
template <int K>
inline int conv_wgrad_launch(Ctx* ctx, const ConvShape& s, const float* g, const float* x, float* part, float* gW) {
  constexpr int OT = ConvWgOT<K>::v; int sets; size_t smem;
  ConvWg c = conv_wgrad_plan(ctx, s, OT, &sets, &smem); c.aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int items = c.ocb / OT * c.icb, threads = (items * c.pg + 31) & ~31, n = s.outC * s.inC * K * K + s.outC;
  GN_CUDA(cudaFuncSetAttribute(conv_wgrad_tile_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, conv_wgrad_tile_kernel<K>, dim3(sets, cdiv(s.inC, c.icb) * cdiv(s.outC, c.ocb)), threads, smem, g, x, part, c);
  GN_LAUNCH(ctx, conv_wgrad_final_kernel, cdiv(n, 32), 256, 0, (const float*)part, sets, n, gW);
  return check_launch("conv_wgrad");
}
// weight and bias gradients (gb follows gW); `part`: conv_wgrad_part_floats
inline int conv_direct_wgrad(Ctx* ctx, const ConvShape& s, const float* g, const float* x, float* part, float* gW) {
  if (s.k == 1) return conv_wgrad_launch<1>(ctx, s, g, x, part, gW);
  if (s.k == 3) return conv_wgrad_launch<3>(ctx, s, g, x, part, gW);
  return conv_wgrad_launch<5>(ctx, s, g, x, part, gW);
}

}  // namespace gn
