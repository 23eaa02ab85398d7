// rowops.cuh -- the memory-bound kernels of the training step: activations and their
// derivatives, (log-)softmax heads with the reference's loss gradients, LayerNorm,
// embedding / positional table / CLS pooling, the attention row kernels, reductions over
// samples and tokens, and the fused Adam update.  All are coalesced, 128-bit where the
// shape allows, and reduce with warp shuffles.
#pragma once
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include "common.cuh"
#include "fmath.cuh"

namespace gn {

// ---------------------------------------------------------------- activations
// reference: internal/activations/activations.go:25-58, :135-143 (float64 libm then rounded), :62-82 (LeakyReLU),
// :241-275 (GELU, tanh form: Activate in float32 around a float64 tanh, Derivative in float64), :277-309 (SiLU), :311-340 (ELU)
__host__ __device__ inline float act_alpha_of(int act, int bits) {
  float a = 0.f; memcpy(&a, &bits, 4);
  if (bits == 0) a = act == GN_ACT_LEAKY_RELU ? 0.01f : (act == GN_ACT_ELU ? 1.0f : 0.f);
  return a;
}
__device__ __forceinline__ float act_fwd(int act, float x, float alpha = 0.f) {
  switch (act) {
    case GN_ACT_RELU: return x > 0.f ? x : 0.f;
    case GN_ACT_SIGMOID: return 1.f / (1.f + exp_rn(-x));
    case GN_ACT_TANH: return tanh_rn(x);
    case GN_ACT_LEAKY_RELU: return x > 0.f ? x : alpha * x;
    case GN_ACT_ELU: return x > 0.f ? x : alpha * (exp_rn(x) - 1.f);
    case GN_ACT_GELU: return gelu_f(x);
    case GN_ACT_SILU: { if (x >= 0.f) return x * (1.f / (1.f + exp_rn(-x))); float e = exp_rn(x); return x * e / (1.f + e); }
    default: return x;
  }
}
__device__ __forceinline__ float act_der(int act, float x, float alpha = 0.f) {
  switch (act) {
    case GN_ACT_RELU: return x > 0.f ? 1.f : 0.f;
    case GN_ACT_SIGMOID: { float s = 1.f / (1.f + exp_rn(-x)); return s * (1.f - s); }
    case GN_ACT_TANH: { float t = tanh_rn(x); return 1.f - t * t; }
    case GN_ACT_LEAKY_RELU: return x > 0.f ? 1.f : alpha;
    case GN_ACT_ELU: return x > 0.f ? 1.f : alpha * exp_rn(x);
    case GN_ACT_GELU: {
      const double c = 0.044715, k = 0.7978845608028654, xd = (double)x, x2 = xd * xd, t = tanh(k * (xd + c * xd * x2));
      return (float)(0.5 * (1.0 + t) + 0.5 * xd * (1.0 - t * t) * k * (1.0 + 3.0 * c * x2));
    }
    case GN_ACT_SILU: { const float e = exp_rn(x >= 0.f ? -x : x), sg = (x >= 0.f ? 1.f : e) / (1.f + e); return sg + x * sg * (1.f - sg); }
    default: return 1.f;
  }
}
__global__ void act_forward_kernel(const float* __restrict__ z, float* __restrict__ a, long n, int act, float alpha = 0.f) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) a[i] = act_fwd(act, z[i], alpha);
}
// dz = dA * act'(z)   (Dense.Backward default branch, layer.go:563-567; Conv2D.Backward conv2d.go:1133)
__global__ void act_backward_kernel(const float* __restrict__ dA, const float* __restrict__ z, float* __restrict__ dz, long n, int act, float alpha = 0.f) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) dz[i] = dA[i] * act_der(act, z[i], alpha);
}

// ---------------------------------------------------------------- softmax heads
// One block per row.  reference: activations.go:160-183 / :204-236
// (1024 threads for wide rows: the three passes over a row are bound by latency, 5.7 us for 8192 columns, 12 with 256)
__global__ void softmax_rows_kernel(const float* __restrict__ z, float* __restrict__ out, int n, int log_mode) {
  __shared__ float red[33];
  const float* zr = z + (long)blockIdx.x * n; float* o = out + (long)blockIdx.x * n;
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmaxf(mx, zr[i]);
  mx = block_max(mx, red);
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += expf(zr[i] - mx);
  s = block_sum(s, red);
  if (log_mode) { float ls = logf(s); for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = zr[i] - mx - ls; }
  else for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = expf(zr[i] - mx) / s;
}

// The batch's loss sum (net.go:711-716), formed by the block that finishes last: `ticket` counts finished rows and is left at zero.
// Strided sums per thread, then the block's tree: a fixed order.
__device__ __forceinline__ void loss_row_done(float value, float* __restrict__ loss, int row, int rows, unsigned* __restrict__ ticket, float* __restrict__ total, float* red) {
  __shared__ int is_last;
  if (threadIdx.x == 0) { loss[row] = value; __threadfence(); is_last = atomicAdd(ticket, 1u) == (unsigned)rows - 1u; }
  __syncthreads();
  if (!is_last) return;
  float s = 0.f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) s += __ldcg(loss + i);
  s = block_sum(s, red);
  if (threadIdx.x == 0) { total[0] = s; *ticket = 0u; }
}
// Per-sample loss value and dL/dy.  reference: loss.go:53-68,91-105 (MSE), :120-140,165-178 (CrossEntropy:
// value = -sum y*log(max(p,1e-10)); gradient returned as p - y).
__global__ void loss_rows_kernel(const float* __restrict__ p, const float* __restrict__ y, float* __restrict__ grad,
                                 float* __restrict__ loss, int n, int kind, unsigned* __restrict__ ticket, float* __restrict__ total) {
  __shared__ float red[33];
  const long off = (long)blockIdx.x * n;
  float s = 0.f;
  if (kind == GN_LOSS_MSE) {
    float f = 2.f / (float)n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) { float d = p[off + i] - y[off + i]; s += d * d; grad[off + i] = f * d; }
    s = block_sum(s, red) / (float)n;
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      float pr = p[off + i], yy = y[off + i];
      grad[off + i] = pr - yy;
      if (yy != 0.f) s -= yy * logf(fmaxf(pr, 1e-10f));
    }
    s = block_sum(s, red);
  }
  loss_row_done(s, loss, blockIdx.x, gridDim.x, ticket, total, red);
}
// The whole head of a training step in one pass over the logits: softmax or log-softmax of z, the sample's loss against y, and
// the gradient that reaches z (the loss gradient through the head's Jacobian, see head_jacobian_kernel).  A cluster of `cs`
// blocks holds one row in registers, E values per thread; the four reductions (maximum, exponential sum, and loss and Jacobian
// sum together) meet in distributed shared memory.  Three kernels of one block per row (softmax, loss, Jacobian) read
// the row nine times: 172 us for 64 rows of 32000, against 31 now.
constexpr int HEAD_THREADS = 256, HEAD_MAX_CS = 8, HEAD_MAX_E = 16;
template <int E>
__global__ void __launch_bounds__(HEAD_THREADS) head_loss_kernel(const float* __restrict__ z, const float* __restrict__ y, float* __restrict__ dz, float* __restrict__ loss,
                                                                 int n, int rows, int cs, int log_mode, int kind, unsigned* __restrict__ ticket, float* __restrict__ total) {
  __shared__ float red[33], slot[4];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int row = blockIdx.x / cs, rank = blockIdx.x % cs, i0 = rank * HEAD_THREADS * E + threadIdx.x; const long off = (long)row * n;
  float v[E], t[E];
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int i = i0 + e * HEAD_THREADS; const bool in = i < n;
    v[e] = in ? z[off + i] : -INFINITY; t[e] = in ? y[off + i] : 0.f; mx = fmaxf(mx, v[e]);
  }
  auto gather = [&](int k, float x, bool is_max) -> float {      // over the cluster's blocks, in rank order
    if (cs == 1) return x;
    if (threadIdx.x == 0) slot[k] = x;
    cluster.sync();
    float a = *cluster.map_shared_rank(&slot[k], 0);
    for (int q = 1; q < cs; q++) { const float b = *cluster.map_shared_rank(&slot[k], q); a = is_max ? fmaxf(a, b) : a + b; }
    return a;
  };
  mx = gather(0, block_max(mx, red), true);
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < E; e++) s += i0 + e * HEAD_THREADS < n ? expf(v[e] - mx) : 0.f;
  s = gather(1, block_sum(s, red), false);
  const float ls = logf(s), f = kind == GN_LOSS_MSE ? 2.f / (float)n : 1.f;
  float lv = 0.f, js = 0.f;
#pragma unroll
  for (int e = 0; e < E; e++) {
    if (i0 + e * HEAD_THREADS < n) {
      const float p = log_mode ? v[e] - mx - ls : expf(v[e] - mx) / s, d = p - t[e], g = f * d;
      if (kind == GN_LOSS_MSE) lv += d * d; else if (t[e] != 0.f) lv -= t[e] * logf(fmaxf(p, 1e-10f));
      js += log_mode ? g : g * p;
      v[e] = p; t[e] = g;
    }
  }
  lv = gather(2, block_sum(lv, red), false);
  js = gather(3, block_sum(js, red), false);
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int i = i0 + e * HEAD_THREADS;
    if (i < n) dz[off + i] = log_mode ? t[e] - expf(v[e]) * js : v[e] * (t[e] - js);
  }
  if (cs > 1) cluster.sync();                                 // nobody leaves while its slots are being read
  if (rank == 0) loss_row_done(kind == GN_LOSS_MSE ? lv / (float)n : lv, loss, row, rows, ticket, total, red);
}

// Dense.Backward for a Softmax head (layer.go:516-528):  dz_k = sum_i g_i p_i (delta_ik - p_k) = p_k (g_k - sum_i g_i p_i)
// and for a LogSoftmax head (layer.go:547-559):          dz_k = sum_i g_i (delta_ik - e^{l_k})  = g_k - e^{l_k} sum_i g_i
__global__ void head_jacobian_kernel(const float* __restrict__ g, const float* __restrict__ out, float* __restrict__ dz, int n, int log_mode) {
  __shared__ float red[33];
  const long off = (long)blockIdx.x * n;
  float s = 0.f;
  if (log_mode) for (int i = threadIdx.x; i < n; i += blockDim.x) s += g[off + i];
  else for (int i = threadIdx.x; i < n; i += blockDim.x) s += g[off + i] * out[off + i];
  s = block_sum(s, red);
  if (log_mode) for (int i = threadIdx.x; i < n; i += blockDim.x) dz[off + i] = g[off + i] - expf(out[off + i]) * s;
  else for (int i = threadIdx.x; i < n; i += blockDim.x) dz[off + i] = out[off + i] * (g[off + i] - s);
}

// ---------------------------------------------------------------- reductions
// out[c] (=|+=) sum_r in[r*ld + c], rows in `chunks` slabs, partials reduced in slab order.
__global__ void colsum_partial_kernel(const float* __restrict__ in, long ld, int R, int C, float* __restrict__ part) {
  int c = blockIdx.x * blockDim.x + threadIdx.x; if (c >= C) return;
  int chunks = gridDim.y, per = (R + chunks - 1) / chunks, r0 = blockIdx.y * per, r1 = min(R, r0 + per);
  float s = 0.f;
#pragma unroll 8
  for (int r = r0; r < r1; r++) s += in[(long)r * ld + c];
  part[(long)blockIdx.y * C + c] = s;
}
__global__ void colsum_final_kernel(const float* __restrict__ part, int chunks, int C, float* __restrict__ out, int accumulate) {
  int c = blockIdx.x * blockDim.x + threadIdx.x; if (c >= C) return;
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < chunks; k++) s += part[(long)k * C + c];
  out[c] = accumulate ? out[c] + s : s;
}
// delta[s, c] = sum_t in[s, t, c]   ([B,T,C] -> [B,C]); the reference adds per-token terms one token after another.
__global__ void token_sum_kernel(const float* __restrict__ in, int T, int C, float* __restrict__ out) {
  // block = 128 columns x 4 groups of tokens; each group adds every 4th token, four loads in flight per thread
  __shared__ float part[4][128];
  const int c = blockIdx.x * 128 + threadIdx.x, grp = threadIdx.y;
  float s = 0.f;
  if (c < C) {
    const float* p = in + (long)blockIdx.y * T * C + c;
    int t = grp;
    for (; t + 12 < T; t += 16) {
      float a0 = p[(long)t * C], a1 = p[(long)(t + 4) * C], a2 = p[(long)(t + 8) * C], a3 = p[(long)(t + 12) * C];
      s += (a0 + a1) + (a2 + a3);
    }
    for (; t < T; t += 4) s += p[(long)t * C];
  }
  part[grp][threadIdx.x] = s;
  __syncthreads();
  if (grp == 0 && c < C) out[(long)blockIdx.y * C + c] = (part[0][threadIdx.x] + part[1][threadIdx.x]) + (part[2][threadIdx.x] + part[3][threadIdx.x]);
}

// The same sum with 16-byte loads: block = 32 column groups of 4 x 8 groups of tokens (C a multiple of 4, aligned rows).
__global__ void __launch_bounds__(256) token_sum_vec_kernel(const float* __restrict__ in, int T, int C, float* __restrict__ out) {
  __shared__ float4 part[8][32];
  const int c = (blockIdx.x * 32 + threadIdx.x) * 4, grp = threadIdx.y;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < C) {
    const float* p = in + (long)blockIdx.y * T * C + c;
    int t = grp;
    for (; t + 24 < T; t += 32) {
      const float4 a0 = *reinterpret_cast<const float4*>(p + (long)t * C), a1 = *reinterpret_cast<const float4*>(p + (long)(t + 8) * C);
      const float4 a2 = *reinterpret_cast<const float4*>(p + (long)(t + 16) * C), a3 = *reinterpret_cast<const float4*>(p + (long)(t + 24) * C);
      s.x += (a0.x + a1.x) + (a2.x + a3.x); s.y += (a0.y + a1.y) + (a2.y + a3.y); s.z += (a0.z + a1.z) + (a2.z + a3.z); s.w += (a0.w + a1.w) + (a2.w + a3.w);
    }
    for (; t < T; t += 8) { const float4 a = *reinterpret_cast<const float4*>(p + (long)t * C); s.x += a.x; s.y += a.y; s.z += a.z; s.w += a.w; }
  }
  part[grp][threadIdx.x] = s;
  __syncthreads();
  if (grp == 0 && c < C) {
    float4 r = part[0][threadIdx.x];
#pragma unroll
    for (int g = 1; g < 8; g++) { const float4 q = part[g][threadIdx.x]; r.x += q.x; r.y += q.y; r.z += q.z; r.w += q.w; }
    *reinterpret_cast<float4*>(out + (long)blockIdx.y * C + c) = r;
  }
}

// Token sums from the 32-row partial sums a plane-writing contraction leaves behind (TcParams::rowsum32): T / 32 rows per
// sequence, added in order.
__global__ void __launch_bounds__(128) token_sum_part32_kernel(const float* __restrict__ part, int groups, int C, float* __restrict__ out) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4; if (c >= C) return;
  const float* p = part + (long)blockIdx.y * groups * C + c;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int g = 0; g < groups; g++) { const float4 q = *reinterpret_cast<const float4*>(p + (long)g * C); s.x += q.x; s.y += q.y; s.z += q.z; s.w += q.w; }
  *reinterpret_cast<float4*>(out + (long)blockIdx.y * C + c) = s;
}
// The same sum over a tensor that exists only as operand planes (two fp16 planes and an inverse scale per row, written by a
// contraction's epilogue): element = (p0 + p1) * inv_scale[row].  Same block shape as above: 4 columns per thread.
__global__ void __launch_bounds__(256) token_sum_planes_kernel(const __half* __restrict__ pl, const float* __restrict__ inv, long ldp,
                                                               int T, int C, float* __restrict__ out) {
  __shared__ float4 part[8][32];
  const int c = (blockIdx.x * 32 + threadIdx.x) * 4, grp = threadIdx.y;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < C) {
    const long row0 = (long)blockIdx.y * T;
    for (int t = grp; t < T; t += 8) {
      const __half* o = pl + (row0 + t) * 2 * ldp + pl_off(c); const float is = inv[row0 + t];
      const uint2 a = *reinterpret_cast<const uint2*>(o), b = *reinterpret_cast<const uint2*>(o + PL_LO);
      const float2 a0 = __half22float2(*reinterpret_cast<const __half2*>(&a.x)), a1 = __half22float2(*reinterpret_cast<const __half2*>(&a.y));
      const float2 b0 = __half22float2(*reinterpret_cast<const __half2*>(&b.x)), b1 = __half22float2(*reinterpret_cast<const __half2*>(&b.y));
      s.x += (a0.x + b0.x) * is; s.y += (a0.y + b0.y) * is; s.z += (a1.x + b1.x) * is; s.w += (a1.y + b1.y) * is;
    }
  }
  part[grp][threadIdx.x] = s;
  __syncthreads();
  if (grp == 0 && c < C) {
    float4 r = part[0][threadIdx.x];
#pragma unroll
    for (int g = 1; g < 8; g++) { const float4 q = part[g][threadIdx.x]; r.x += q.x; r.y += q.y; r.z += q.z; r.w += q.w; }
    *reinterpret_cast<float4*>(out + (long)blockIdx.y * C + c) = r;
  }
}

// ---------------------------------------------------------------- LayerNorm
// One warp per row.  reference: layernorm.go:268-301
__global__ void layernorm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                                     float* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ std_out, long rows, int n, float eps) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31;
  const float* xr = x + row * n; float* yr = y + row * n;
  float s = 0.f;
  for (int i = lane; i < n; i += 32) s += xr[i];
  float mean = warp_sum(s) / (float)n;
  float ss = 0.f;
  for (int i = lane; i < n; i += 32) { float d = xr[i] - mean; ss += d * d; }
  float var = warp_sum(ss) / (float)n;
  float sd = sqrtf(var + eps);
  for (int i = lane; i < n; i += 32) yr[i] = gamma[i] * ((xr[i] - mean) / sd) + beta[i];
  if (lane == 0) { mean_out[row] = mean; std_out[row] = sd; }
}
// reference: layernorm.go:389-417 -- the second term is divided by N*std*std (not std^3).
// dx may alias g.
__global__ void layernorm_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ gamma,
                                     const float* __restrict__ mean_in, const float* __restrict__ std_in, float* dx, long rows, int n) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31;
  const float* xr = x + row * n; const float* gr = g + row * n; float* dr = dx + row * n;
  float mean = mean_in[row], sd = std_in[row];
  float sg = 0.f, sgx = 0.f;
  for (int i = lane; i < n; i += 32) { float q = gr[i] * gamma[i]; sg += q; sgx += q * (xr[i] - mean); }
  sg = warp_sum(sg); sgx = warp_sum(sgx);
  float fn = (float)n;
  for (int i = lane; i < n; i += 32) {
    float q = gr[i] * gamma[i], d = xr[i] - mean;
    float v = (q - sg / fn) / sd;
    v -= (d * sgx) / (fn * sd * sd);
    dr[i] = v;
  }
}
// gGamma[c] = sum_r g*(x-mean)/std ; gBeta[c] = sum_r g     (layernorm.go:421-433)
__global__ void layernorm_pgrad_partial_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ mean_in,
                                               const float* __restrict__ std_in, long rows, int n, float* __restrict__ part) {
  int c = blockIdx.x * blockDim.x + threadIdx.x; if (c >= n) return;
  long chunks = gridDim.y, per = (rows + chunks - 1) / chunks, r0 = blockIdx.y * per, r1 = min(rows, r0 + per);
  float sgam = 0.f, sbet = 0.f;
  for (long r = r0; r < r1; r++) { float gg = g[r * n + c]; sgam += gg * ((x[r * n + c] - mean_in[r]) / std_in[r]); sbet += gg; }
  part[((long)blockIdx.y * 2) * n + c] = sgam; part[((long)blockIdx.y * 2 + 1) * n + c] = sbet;
}
// block = 32 columns x 32 groups of chunks (1024 threads); the groups are combined through shared memory in a fixed order
// gBeta may be null (RMSNorm)
__global__ void __launch_bounds__(1024) layernorm_pgrad_final_kernel(const float* __restrict__ part, int chunks, int n, float* __restrict__ gGamma, float* __restrict__ gBeta) {
  __shared__ float sa[32][33], sb[32][33];
  const int tx = threadIdx.x & 31, grp = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float a = 0.f, b = 0.f;
  if (c < n) {
#pragma unroll 4
    for (int k = grp; k < chunks; k += 32) { a += part[((long)k * 2) * n + c]; if (gBeta) b += part[((long)k * 2 + 1) * n + c]; }
  }
  sa[grp][tx] = a; sb[grp][tx] = b;
  __syncthreads();
  if (grp == 0 && c < n) {
    float ta = 0.f, tb = 0.f;
    for (int k = 0; k < 32; k++) { ta += sa[k][tx]; tb += sb[k][tx]; }
    gGamma[c] = ta; if (gBeta) gBeta[c] = tb;
  }
}

// ---------------------------------------------------------------- rows in registers
// LayerNorm (RMS = false) and RMSNorm for rows of up to 1024 columns, a multiple of four, 16-byte aligned: one warp per row, the row
// is read once and kept in registers (NV float4 per lane) between the reductions and the output.  Same arithmetic as the kernels
// above and below, except that LayerNorm takes one reciprocal of the deviation per row instead of a division per element.
// Optional second output: the row as operand planes of the contraction engine (two fp16 planes interleaved in blocks of 32
// columns, row length 2 ldp, zero beyond n; the row's inverse scale, its 2-norm): the row maximum and norm are two warp
// reductions here, and the contraction that consumes the row needs no split pass.
struct RowPlaneOut { __half* p = nullptr; float* inv = nullptr; float* rownorm = nullptr; };
template <int NV>
__device__ __forceinline__ void row_planes_emit(const float4 (&o)[NV], long row, int n, int lane, const RowPlaneOut& po) {
  float mx = 0.f, sq = 0.f; const int ldp = (n + 31) & ~31;
#pragma unroll
  for (int k = 0; k < NV; k++) {                            // (entries beyond n are zero)
    mx = fmaxf(mx, fmaxf(fmaxf(fabsf(o[k].x), fabsf(o[k].y)), fmaxf(fabsf(o[k].z), fabsf(o[k].w))));
    sq += (o[k].x * o[k].x + o[k].y * o[k].y) + (o[k].z * o[k].z + o[k].w * o[k].w);
  }
  mx = warp_max(mx); sq = warp_sum(sq);
  float inv; const float sc = row_scale(mx, &inv);
  if (lane == 0) { po.inv[row] = inv; if (po.rownorm) po.rownorm[row] = sqrtf(sq) * 1.0001f; }
  __half* h = po.p + row * 2 * ldp + pl_off(4 * lane);      // columns 4 lane + 128 k
#pragma unroll
  for (int k = 0; k < NV; k++) {
    if (4 * lane + 128 * k >= ldp) continue;
    uint2 a, b; split2_pair(o[k].x, o[k].y, sc, a.x, b.x); split2_pair(o[k].z, o[k].w, sc, a.y, b.y);
    *reinterpret_cast<uint2*>(h + 256 * k) = a; *reinterpret_cast<uint2*>(h + 256 * k + PL_LO) = b;
  }
}
template <int NV>
__device__ __forceinline__ void row_load(float4 (&v)[NV], const float* __restrict__ p, int n, int lane) {
#pragma unroll
  for (int k = 0; k < NV; k++) v[k] = 4 * lane + 128 * k < n ? *reinterpret_cast<const float4*>(p + 4 * lane + 128 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <int NV>
__device__ __forceinline__ void row_store(const float4 (&v)[NV], float* __restrict__ p, int n, int lane) {
#pragma unroll
  for (int k = 0; k < NV; k++) if (4 * lane + 128 * k < n) *reinterpret_cast<float4*>(p + 4 * lane + 128 * k) = v[k];
}
// stat_a: row means (RMS: row rms), stat_b: row deviations
template <int NV, bool RMS>
__global__ void __launch_bounds__(256) norm_fwd_vec_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ y,
                                                           float* __restrict__ stat_a, float* __restrict__ stat_b, long rows, int n, float eps, const RowPlaneOut po) {
  const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5); if (row >= rows) return;
  const int lane = threadIdx.x & 31; const float fn = (float)n;
  float4 v[NV]; row_load(v, x + row * n, n, lane);
  if (RMS) {
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) ss += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
    const float r = (float)sqrt((double)(warp_sum(ss) / fn + eps));
#pragma unroll
    for (int k = 0; k < NV; k++) if (4 * lane + 128 * k < n) {
      const float4 ga = __ldg(reinterpret_cast<const float4*>(gamma) + lane + 32 * k);
      v[k] = make_float4((v[k].x / r) * ga.x, (v[k].y / r) * ga.y, (v[k].z / r) * ga.z, (v[k].w / r) * ga.w);
    }
    if (lane == 0) stat_a[row] = r;
  } else {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
    const float mean = warp_sum(s) / fn;
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) if (4 * lane + 128 * k < n) { const float a = v[k].x - mean, b = v[k].y - mean, c = v[k].z - mean, d = v[k].w - mean; ss += (a * a + b * b) + (c * c + d * d); }
    const float sd = sqrtf(warp_sum(ss) / fn + eps), isd = 1.f / sd;
#pragma unroll
    for (int k = 0; k < NV; k++) if (4 * lane + 128 * k < n) {
      const float4 ga = __ldg(reinterpret_cast<const float4*>(gamma) + lane + 32 * k), be = __ldg(reinterpret_cast<const float4*>(beta) + lane + 32 * k);
      v[k] = make_float4(ga.x * ((v[k].x - mean) * isd) + be.x, ga.y * ((v[k].y - mean) * isd) + be.y, ga.z * ((v[k].z - mean) * isd) + be.z, ga.w * ((v[k].w - mean) * isd) + be.w);
    }
    if (lane == 0) { stat_a[row] = mean; stat_b[row] = sd; }
  }
  row_store(v, y + row * n, n, lane);
  if (po.p) row_planes_emit(v, row, n, lane, po);
}
// Rows of g and dx are dense, row r of x lies at x + r ldx and its statistics at stat[r lds].
// dx (may alias g), and this block's part of the parameter gradients: part[block][0] = sum g (x - mean) / sd (RMS: sum g x / rms),
// part[block][1] = sum g.  The warps stride over the rows with the sums of their columns in registers, so g and x are read
// once for both outputs (two passes before, the second at 1 TB/s: 18 of 25 us at 3600 rows of 384).
template <int NV, bool RMS>
__global__ void __launch_bounds__(256) norm_bwd_vec_kernel(const float* g, const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ stat_a,
                                                           const float* __restrict__ stat_b, float* dx, float* __restrict__ part, long rows, int n, long ldx, long lds, const RowPlaneOut po) {
  __shared__ float4 red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5; const float fn = (float)n;
  float4 ga[NV], sg_[NV], sb_[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) sg_[k] = sb_[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  row_load(ga, gamma, n, lane);
  for (long row = (long)blockIdx.x * 8 + w; row < rows; row += (long)gridDim.x * 8) {
    float4 q[NV], d[NV]; row_load(q, g + row * n, n, lane); row_load(d, x + row * ldx, n, lane);
    const float a = stat_a[row * lds];
    float s = 0.f, sx = 0.f;
    if (RMS) {
      const float inv = 1.f / a;
#pragma unroll
      for (int k = 0; k < NV; k++) {
        sg_[k].x += q[k].x * (d[k].x * inv); sg_[k].y += q[k].y * (d[k].y * inv); sg_[k].z += q[k].z * (d[k].z * inv); sg_[k].w += q[k].w * (d[k].w * inv);
        sx += (q[k].x * ga[k].x * d[k].x + q[k].y * ga[k].y * d[k].y) + (q[k].z * ga[k].z * d[k].z + q[k].w * ga[k].w * d[k].w);
      }
      const float f = warp_sum(sx) / (fn * a * a);
#pragma unroll
      for (int k = 0; k < NV; k++)
        q[k] = make_float4((ga[k].x * inv) * (q[k].x - d[k].x * f), (ga[k].y * inv) * (q[k].y - d[k].y * f), (ga[k].z * inv) * (q[k].z - d[k].z * f), (ga[k].w * inv) * (q[k].w - d[k].w * f));
    } else {
      const float sd = stat_b[row * lds], isd = 1.f / sd;
#pragma unroll
      for (int k = 0; k < NV; k++) {
        if (4 * lane + 128 * k < n) { d[k].x -= a; d[k].y -= a; d[k].z -= a; d[k].w -= a; }
        sg_[k].x += q[k].x * (d[k].x * isd); sg_[k].y += q[k].y * (d[k].y * isd); sg_[k].z += q[k].z * (d[k].z * isd); sg_[k].w += q[k].w * (d[k].w * isd);
        sb_[k].x += q[k].x; sb_[k].y += q[k].y; sb_[k].z += q[k].z; sb_[k].w += q[k].w;
        q[k].x *= ga[k].x; q[k].y *= ga[k].y; q[k].z *= ga[k].z; q[k].w *= ga[k].w;
        s += (q[k].x + q[k].y) + (q[k].z + q[k].w);
        sx += (q[k].x * d[k].x + q[k].y * d[k].y) + (q[k].z * d[k].z + q[k].w * d[k].w);
      }
      s = warp_sum(s) / fn; const float f = warp_sum(sx) / (fn * sd * sd);
#pragma unroll
      for (int k = 0; k < NV; k++) if (4 * lane + 128 * k < n)
        q[k] = make_float4((q[k].x - s) * isd - d[k].x * f, (q[k].y - s) * isd - d[k].y * f, (q[k].z - s) * isd - d[k].z * f, (q[k].w - s) * isd - d[k].w * f);
    }
    row_store(q, dx + row * n, n, lane);
    if (po.p) row_planes_emit(q, row, n, lane, po);
  }
  float* pb = part + (long)blockIdx.x * 2 * n;
#pragma unroll
  for (int k = 0; k < NV; k++) {
#pragma unroll
    for (int h = 0; h < (RMS ? 1 : 2); h++) {
      __syncthreads();
      red[w][lane] = h ? sb_[k] : sg_[k];
      __syncthreads();
      if (w == 0 && 4 * lane + 128 * k < n) {
        float4 t = red[0][lane];
#pragma unroll
        for (int r = 1; r < 8; r++) { const float4 u = red[r][lane]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
        *reinterpret_cast<float4*>(pb + h * n + 4 * lane + 128 * k) = t;
      }
    }
  }
}
// ---------------------------------------------------------------- RMSNorm
// One warp per row.  reference: rmsnorm.go:222-240 (forward), :301-330 (backward); the row's rms is kept for the backward.
__global__ void rmsnorm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma, float* __restrict__ y, float* __restrict__ rms_out, long rows, int n, float eps) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31;
  const float* xr = x + row * n; float* yr = y + row * n;
  float ss = 0.f;
  for (int i = lane; i < n; i += 32) ss += xr[i] * xr[i];
  const float r = (float)sqrt((double)(warp_sum(ss) / (float)n + eps));
  for (int i = lane; i < n; i += 32) yr[i] = (xr[i] / r) * gamma[i];
  if (lane == 0) rms_out[row] = r;
}
// dx may alias g.
__global__ void rmsnorm_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ rms_in,
                                   float* dx, long rows, int n) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31;
  const float* xr = x + row * n; const float* gr = g + row * n; float* dr = dx + row * n;
  const float r = rms_in[row], inv = 1.f / r;
  float s = 0.f;
  for (int i = lane; i < n; i += 32) s += gr[i] * gamma[i] * xr[i];
  const float factor = warp_sum(s) / ((float)n * r * r);
  for (int i = lane; i < n; i += 32) dr[i] = (gamma[i] * inv) * (gr[i] - xr[i] * factor);
}
// gGamma[c] partial sums over a chunk of rows: sum_r g * (x / rms)    (rmsnorm.go:322-330); part[chunk][n]
__global__ void rmsnorm_pgrad_partial_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ rms_in, long rows, int n, float* __restrict__ part) {
  int c = blockIdx.x * blockDim.x + threadIdx.x; if (c >= n) return;
  long chunks = gridDim.y, per = (rows + chunks - 1) / chunks, r0 = blockIdx.y * per, r1 = min(rows, r0 + per);
  float s = 0.f;
  for (long r = r0; r < r1; r++) s += g[r * n + c] * (x[r * n + c] * (1.f / rms_in[r]));
  part[(long)blockIdx.y * n + c] = s;
}
__global__ void rmsnorm_pgrad_final_kernel(const float* __restrict__ part, int chunks, int n, float* __restrict__ gGamma) {
  int c = blockIdx.x * blockDim.x + threadIdx.x; if (c >= n) return;
  float a = 0.f;
  for (int k = 0; k < chunks; k++) a += part[(long)k * n + c];
  gGamma[c] = a;
}

// Norm backward on a few rows: rows s of g and dx are dense [rows, n], row s of the norm's input lies at x + s * ldx and its
// statistics at mean[s * lds], sd[s * lds] (LayerNorm) or mean[s * lds] = rms (sd = null: RMSNorm).  One warp per row; the
// formulas of the kernels above.
__global__ void __launch_bounds__(128) norm_bwd_rows_kernel(const float* __restrict__ g, const float* __restrict__ x, long ldx, const float* __restrict__ gamma,
                                                            const float* __restrict__ mean_in, const float* __restrict__ sd_in, long lds, float* __restrict__ dx, int rows, int n) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31; if (row >= rows) return;
  const float* xr = x + row * ldx; const float* gr = g + (long)row * n; float* dr = dx + (long)row * n;
  const float c = mean_in[row * lds], fn = (float)n; float sg = 0.f, sgx = 0.f;
  if (sd_in) {
    const float sd = sd_in[row * lds], isd = 1.f / sd;
    for (int i = lane; i < n; i += 32) { const float q = gr[i] * gamma[i]; sg += q; sgx += q * (xr[i] - c); }
    sg = warp_sum(sg) / fn; const float w = warp_sum(sgx) / (fn * sd * sd);
    for (int i = lane; i < n; i += 32) dr[i] = (gr[i] * gamma[i] - sg) * isd - (xr[i] - c) * w;
  } else {
    const float inv = 1.f / c;
    for (int i = lane; i < n; i += 32) sgx += gr[i] * gamma[i] * xr[i];
    const float f = warp_sum(sgx) / (fn * c * c);
    for (int i = lane; i < n; i += 32) dr[i] = (gamma[i] * inv) * (gr[i] - xr[i] * f);
  }
}
// ... and its parameter gradients, written (not added); block = 32 columns x 8 groups of rows, combined in a fixed order
__global__ void __launch_bounds__(256) norm_pgrad_rows_kernel(const float* __restrict__ g, const float* __restrict__ x, long ldx, const float* __restrict__ mean_in,
                                                              const float* __restrict__ sd_in, long lds, int rows, int n, float* __restrict__ gGamma, float* __restrict__ gBeta) {
  __shared__ float sa[8][33], sb[8][33];
  const int tx = threadIdx.x & 31, grp = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float a = 0.f, b = 0.f;
  if (c < n) {
#pragma unroll 4
    for (int r = grp; r < rows; r += 8) {
      const float gg = g[(long)r * n + c], st = mean_in[r * lds];
      a += sd_in ? gg * ((x[r * ldx + c] - st) / sd_in[r * lds]) : gg * (x[r * ldx + c] * (1.f / st)); b += gg;
    }
  }
  sa[grp][tx] = a; sb[grp][tx] = b;
  __syncthreads();
  if (grp == 0 && c < n) {
    for (int k = 1; k < 8; k++) { a += sa[k][tx]; b += sb[k][tx]; }
    gGamma[c] = a; if (gBeta) gBeta[c] = b;
  }
}

// ---------------------------------------------------------------- Dropout
// The reference's generator (layer.go:61-75): s <- s * 6364136223846793005 + 1, value = float32(s >> 33) / 2^31, one
// stream per layer seeded with 42 and consumed element by element, sample by sample (dropout.go:139-152).  Draw k of the
// stream is reached by composing the affine map k times (square and multiply), so every thread can enter the stream at
// its own elements: element i of global sample g of a batch that starts after `count` draws uses draw count + g n + i + 1.
// `cnt` = the two state floats (count mod 2^20, count >> 20).
__device__ __forceinline__ unsigned long long lcg_jump(unsigned long long s0, unsigned long long k) {
  unsigned long long A = 1, C = 0, a = 6364136223846793005ull, c = 1;
  while (k) { if (k & 1) { A = A * a; C = C * a + c; } c = c * (a + 1); a = a * a; k >>= 1; }
  return A * s0 + C;
}
constexpr int DROP_RUN = 8;      // consecutive elements per thread (one jump, then the recurrence)
__global__ void dropout_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, float* __restrict__ mask, const float* __restrict__ cnt,
                                   long total, int n, float p, long first_elem) {
  const unsigned long long count = (unsigned long long)cnt[0] + ((unsigned long long)cnt[1] << 20);
  const float scale = 1.0f / (1.0f - p);
  for (long e0 = (blockIdx.x * (long)blockDim.x + threadIdx.x) * DROP_RUN; e0 < total; e0 += (long)gridDim.x * blockDim.x * DROP_RUN) {
    unsigned long long s = lcg_jump(42ull, count + (unsigned long long)(first_elem + e0));
#pragma unroll
    for (int j = 0; j < DROP_RUN; j++) {
      const long e = e0 + j; if (e >= total) break;
      s = s * 6364136223846793005ull + 1ull;
      const float r = (float)(s >> 33) / 2147483648.0f;
      const bool keep = !(r < p);
      mask[e] = keep ? 1.f : 0.f; y[e] = keep ? x[e] * scale : 0.f;
    }
  }
}
__global__ void dropout_bwd_kernel(const float* __restrict__ g, const float* __restrict__ mask, float* __restrict__ dx, long total, float p) {
  const float scale = 1.0f / (1.0f - p);
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) dx[e] = mask[e] > 0.f ? g[e] * scale : 0.f;
}
// after a training batch: the stream has moved on by `add` draws (global batch x elements per sample)
__global__ void dropout_advance_kernel(float* __restrict__ cnt, unsigned long long add) {
  const unsigned long long c = (unsigned long long)cnt[0] + ((unsigned long long)cnt[1] << 20) + add;
  cnt[0] = (float)(c & 0xfffffull); cnt[1] = (float)(c >> 20);
}

// ---------------------------------------------------------------- embedding / positional / CLS
// out[s,t,:] = E[floor(id)] (+ P[t,:])   reference: embedding.go:120-136, transformer.go:80-82
// A token id outside [0, V) is an error in the reference (embedding.go:124-129): the kernel records it in the status
// word (GN_STATUS_BAD_TOKEN; the host turns it into GN_ERR_INVALID_ARG and the step changes nothing) and carries on
// with a clamped id, so that nothing is read out of bounds.
constexpr int GN_STATUS_BAD_TOKEN = 100;
__global__ void embedding_fwd_kernel(const float* __restrict__ ids, const float* __restrict__ E, const float* __restrict__ P,
                                     float* __restrict__ out, long tokens, int T, int d, int V, int* __restrict__ idx_out, int* __restrict__ status, int row0_only) {
  long tok = blockIdx.x; if (tok >= tokens) return;
  int id = (int)floorf(ids[tok]);
  if (id < 0 || id >= V || !(ids[tok] == ids[tok])) { if (threadIdx.x == 0) atomicCAS(status, 0, GN_STATUS_BAD_TOKEN); id = id < 0 ? 0 : V - 1; }
  if (threadIdx.x == 0 && idx_out) idx_out[tok] = id;
  if (row0_only && tok % T) return;                        // the layers above read token 0 of every sequence: out is [sequences, d]
  const float* e = E + (long)id * d; float* o = out + (row0_only ? tok / T : tok) * d;
  if (P) { const float* p = P + (long)(tok % T) * d; for (int i = threadIdx.x; i < d; i += blockDim.x) o[i] = e[i] + p[i]; }
  else for (int i = threadIdx.x; i < d; i += blockDim.x) o[i] = e[i];
}
// The same with rows in registers (d <= 1024, a multiple of four, 16-byte rows), one warp per token; optionally the row as operand planes
// for the projections of the block above.  Memory-bound; a block of 128 threads per token moved 268 MB in 85 us.
template <int NV>
__global__ void __launch_bounds__(256) embedding_fwd_vec_kernel(const float* __restrict__ ids, const float* __restrict__ E, const float* __restrict__ P, float* __restrict__ out, long tokens, int T, int d,
                                                                int V, int* __restrict__ idx_out, int* __restrict__ status, int row0_only, const RowPlaneOut po) {
  const long tok = (long)blockIdx.x * 8 + (threadIdx.x >> 5); if (tok >= tokens) return;
  const int lane = threadIdx.x & 31; const float fid = ids[tok]; int id = (int)floorf(fid);
  if (id < 0 || id >= V || !(fid == fid)) { if (lane == 0) atomicCAS(status, 0, GN_STATUS_BAD_TOKEN); id = id < 0 ? 0 : V - 1; }
  if (lane == 0 && idx_out) idx_out[tok] = id;
  if (row0_only && tok % T) return;
  float4 v[NV]; row_load(v, E + (long)id * d, d, lane);
  if (P) {
    float4 p[NV]; row_load(p, P + (long)(tok % T) * d, d, lane);
#pragma unroll
    for (int k = 0; k < NV; k++) { v[k].x += p[k].x; v[k].y += p[k].y; v[k].z += p[k].z; v[k].w += p[k].w; }
  }
  const long row = row0_only ? tok / T : tok;
  row_store(v, out + row * d, d, lane);
  if (po.p) row_planes_emit(v, row, d, lane, po);
}
__global__ void posenc_fwd_kernel(const float* __restrict__ x, const float* __restrict__ P, float* __restrict__ out, long total, long per_sample) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) out[i] = x[i] + P[i % per_sample];
}
// Embedding.Backward zeroes its whole gradient at every call (embedding.go:151-154), so only the last
// sample of each worker chunk reaches the table.  Gradient of ONE such sample, added to the table: block t handles
// position t, and only if t is the first position of its token id; it then adds the rows of all positions with that
// id in ascending order, exactly the sum the reference's loop forms for that table row (embedding.go:156-180), and adds
// the result to the row.  No two blocks touch the same row, so there are no atomics and the result does not depend on
// scheduling; the samples of a batch are processed by consecutive launches in sample order (the order in which the
// reference adds its workers' gradients, net.go:694-700).
__global__ void __launch_bounds__(128) embedding_bwd_sample_kernel(const float* __restrict__ g, const int* __restrict__ ids, float* __restrict__ gE, int T, int d) {
  extern __shared__ int same[];                 // positions after t that hold the same id, ascending
  __shared__ int count[5];
  const int t = blockIdx.x, id = ids[t], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int mine = 0;
  for (int u = threadIdx.x; u < t; u += 128) mine |= ids[u] == id;
  if (__syncthreads_or(mine)) return;           // an earlier position of this id adds the row
  int n_same = 0;
  for (int u0 = t + 1; u0 < T; u0 += 128) {     // 128 positions at a time, kept in order (one thread walking the ids took 12 us)
    const int u = u0 + threadIdx.x; const bool hit = u < T && ids[u] == id;
    const unsigned b = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) count[w] = __popc(b);
    __syncthreads();
    int before = n_same;
    for (int q = 0; q < w; q++) before += count[q];
    if (hit) same[before + __popc(b & ((1u << lane) - 1u))] = u;
    n_same += count[0] + count[1] + count[2] + count[3];
    __syncthreads();
  }
  float* dst = gE + (long)id * d;
  for (int i = threadIdx.x; i < d; i += 128) {
    float s = g[(long)t * d + i];
    for (int k = 0; k < n_same; k++) s += g[(long)same[k] * d + i];
    dst[i] += s;
  }
}
// Results of a small inference call and the status word, straight to host memory.
__global__ void finish_kernel(const float* __restrict__ src, float* __restrict__ dst, int n, const int* __restrict__ status, float* __restrict__ ret) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) ret[1] = __int_as_float(*status);
}
// Multi-GPU exchange of the few samples that reach the table: slot q of the buffers belongs to the q-th qualifying
// sample of the global batch; the rank that owns it copies its gradient rows [T, d] and token ids (as floats) there,
// every other rank leaves zeros, and a sum all-reduce of the small buffers gives every rank all of them.
__global__ void embedding_pack_kernel(const float* __restrict__ g, const int* __restrict__ idx, float* __restrict__ rows, float* __restrict__ ids, int T, int d) {
  const int t = blockIdx.x;
  for (int i = threadIdx.x; i < d; i += blockDim.x) rows[(long)t * d + i] = g[(long)t * d + i];
  if (threadIdx.x == 0) ids[t] = (float)idx[t];
}
__global__ void ids_to_int_kernel(const float* __restrict__ f, int* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x; if (i < n) out[i] = (int)f[i];
}
// out [2 B, d] <- tokens 0 and T - 1 of every sequence of x [B, T, d]; one block per row
__global__ void gather_ends_kernel(const float* __restrict__ x, float* __restrict__ out, int T, int d) {
  const long r = blockIdx.x; const float* src = x + ((r >> 1) * T + (r & 1) * (T - 1)) * (long)d; float* dst = out + r * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) dst[i] = src[i];
}
// CLSPooling: y[s,:] = x[s,0,:]; backward: zeros except token 0   transformer.go:1684, :1715-1724
__global__ void cls_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, int T, int d) {
  const float* src = x + (long)blockIdx.x * T * d; float* dst = y + (long)blockIdx.x * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) dst[i] = src[i];
}
__global__ void cls_bwd_kernel(const float* __restrict__ g, float* __restrict__ dx, int T, int d, long total) {
  long per = (long)T * d;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    long s = i / per, r = i % per;
    dx[i] = r < d ? g[s * d + r] : 0.f;
  }
}

// ---------------------------------------------------------------- attention row kernels
// P[i, :] = softmax over j <= i of S[i,j] * inv_scale, zeros for j > i.  reference: transformer.go:470-491
// (masked scores are -1e9 before the softmax, whose exponentials are exactly 0 in fp32).
// One warp per row; rows are [batch*heads*T].
__global__ void attn_softmax_kernel(float* __restrict__ S, int T, float inv_scale, int causal, long rows) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31; int i = (int)(row % T); int lim = causal ? i + 1 : T;
  float* r = S + row * T;
  float mx = -INFINITY;
  for (int j = lane; j < lim; j += 32) mx = fmaxf(mx, r[j] * inv_scale);
  mx = warp_max(mx);
  float s = 0.f;
  for (int j = lane; j < lim; j += 32) s += expf(r[j] * inv_scale - mx);
  s = warp_sum(s);
  for (int j = lane; j < T; j += 32) r[j] = j < lim ? expf(r[j] * inv_scale - mx) / s : 0.f;
}
// dS[i,j] = P[i,j] * (dP[i,j] - sum_k dP[i,k] P[i,k]) * inv_scale for j <= i, else 0.  transformer.go:625-648
__global__ void attn_ds_kernel(const float* __restrict__ P, float* __restrict__ dP, int T, float inv_scale, int causal, long rows) {
  long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); if (row >= rows) return;
  int lane = threadIdx.x & 31; int i = (int)(row % T); int lim = causal ? i + 1 : T;
  const float* p = P + row * T; float* d = dP + row * T;
  float s = 0.f;
  for (int j = lane; j < lim; j += 32) s += d[j] * p[j];
  s = warp_sum(s);
  for (int j = lane; j < T; j += 32) d[j] = j < lim ? p[j] * (d[j] - s) * inv_scale : 0.f;
}

// ---------------------------------------------------------------- TransformerBlock variants
// Rotary embeddings on a [tokens, D] tensor in place (transformer.go:212-236): within every head, element i of the first
// half and element i + hd/2 are rotated by the angle of (position, i); `tab` holds cos | sin per (position, i), computed on
// the host with the reference's float32 / float64 conversions.  sign = -1 applies the conjugate (backward pass).
// Row r of a sequence's T rows is its token r * tstep.  blockIdx.y picks one of two arrays; V neighbouring pairs per thread (4: hd a
// multiple of 8, rows 16-byte aligned).  Memory-bound; with one pair per thread and 64-bit index divisions a pass over 4096 x 512
// took 11 us, twice its traffic's time, and q and k took a launch each.
template <int V>
__global__ void __launch_bounds__(256) rope_kernel(float* __restrict__ x0, float* __restrict__ x1, const float* __restrict__ tab, long tokens, int T, int D, int hd, float sign, int tstep) {
  float* x = blockIdx.y ? x1 : x0;
  const int half = hd >> 1, per = (D >> 1) / V; const long total = tokens * per;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long tok = total < 0x7fffffffL ? (long)((unsigned)e / (unsigned)per) : e / per;
    const int r = (int)(e - tok * per) * V, h = r / half, i = r - h * half;
    const int t = (total < 0x7fffffffL ? (int)((unsigned)tok % (unsigned)T) : (int)(tok % T)) * tstep;
    const float* cs = tab + ((long)t * half + i) * 2; float* p = x + tok * D + (long)h * hd + i;
    float a[V], b[V], c[2 * V];
    if constexpr (V == 4) {
      const float4 u = *reinterpret_cast<const float4*>(p), w = *reinterpret_cast<const float4*>(p + half);
      const float4 c0 = __ldg(reinterpret_cast<const float4*>(cs)), c1 = __ldg(reinterpret_cast<const float4*>(cs) + 1);
      a[0] = u.x; a[1] = u.y; a[2] = u.z; a[3] = u.w; b[0] = w.x; b[1] = w.y; b[2] = w.z; b[3] = w.w;
      c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    } else { a[0] = p[0]; b[0] = p[half]; c[0] = cs[0]; c[1] = cs[1]; }
    float o0[V], o1[V];
#pragma unroll
    for (int j = 0; j < V; j++) { const float sn = sign * c[2 * j + 1]; o0[j] = a[j] * c[2 * j] - b[j] * sn; o1[j] = a[j] * sn + b[j] * c[2 * j]; }
    if constexpr (V == 4) {
      *reinterpret_cast<float4*>(p) = make_float4(o0[0], o0[1], o0[2], o0[3]); *reinterpret_cast<float4*>(p + half) = make_float4(o1[0], o1[1], o1[2], o1[3]);
    } else { p[0] = o0[0]; p[half] = o1[0]; }
  }
}
// rows [B, C] <- the last token's row of every sequence of in [B, T, C]
__global__ void last_token_rows_kernel(const float* __restrict__ in, float* __restrict__ out, int T, int C, long total) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) { const long s = e / C; out[e] = in[(s * T + (T - 1)) * C + (e - s * C)]; }
}
// dz[s,t,:] *= act'(z_last[s,:]): a Dense layer called token by token differentiates at its LAST call's pre-activation (layer.go:563-567)
__global__ void scale_by_last_deriv_kernel(float* __restrict__ dz, const float* __restrict__ z_last, int T, int C, long total, int act) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) { const long row = e / C; dz[e] *= act_der(act, z_last[(row / T) * C + (e - row * C)]); }
}
__global__ void act_deriv_kernel(const float* __restrict__ z, float* __restrict__ out, long n, int act) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) out[e] = act_der(act, z[e]);
}
// SwiGLU (swiglu.go:163-170): out = swish(gate) * up
__global__ void swiglu_fwd_kernel(const float* __restrict__ gate, const float* __restrict__ up, float* __restrict__ out, long n) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) { const float g = gate[e]; out[e] = (g * act_fwd(GN_ACT_SIGMOID, g)) * up[e]; }
}
// SwiGLU backward inside a TransformerBlock (swiglu.go:203-216 with the pairing of transformer.go:1238-1250): the gradient of
// token t meets the saved state of token T-1-t.  Results are written at the PARTNER's row, where the weight-gradient
// contraction with the layer's inputs needs them.
__global__ void swiglu_bwd_paired_kernel(const float* __restrict__ dOut, const float* __restrict__ gate, const float* __restrict__ up,
                                         float* __restrict__ dGateP, float* __restrict__ dUpP, int T, int C, long total) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long row = e / C; const int c = (int)(e - row * C); const long s = row / T; const int t = (int)(row - s * T);
    const long pe = (s * T + (T - 1 - t)) * C + c;            // partner element
    const float g = gate[pe], u = up[pe], sig = act_fwd(GN_ACT_SIGMOID, g), sw = g * sig, go = dOut[e];
    dUpP[pe] = go * sw; dGateP[pe] = go * (sw + sig * (1.f - sw)) * u;
  }
}
// The two passes above for rows of up to 4096 columns (a multiple of 32) whose results feed the tensor-core engine: a block keeps its
// row in registers between the row's maximum and the operand planes, so the separate split passes (the row read once or twice
// more) go.  Memory-bound: 12 and 28 bytes per element.  Forward: mid only as planes, and the last token's rows in fp32 (the
// weight gradient's input).  Backward: planes of [dGate | dUp] rows (the input gradient's operand) and both in fp32 (the weight
// gradients need them transposed).
constexpr int SW_THREADS = 128;
__device__ __forceinline__ float row_block_max(float mx, float* red) {
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  return fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
}
__device__ __forceinline__ float max4(float m, float4 v) { return fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))); }
__device__ __forceinline__ void planes_store4(__half* row, int c, float4 v, float sc) {
  uint2 a, b; split2_pair(v.x, v.y, sc, a.x, b.x); split2_pair(v.z, v.w, sc, a.y, b.y);
  *reinterpret_cast<uint2*>(row + pl_off(c)) = a; *reinterpret_cast<uint2*>(row + pl_off(c) + PL_LO) = b;
}
template <int NV>
__global__ void __launch_bounds__(SW_THREADS) swiglu_fwd_planes_kernel(const float* __restrict__ gate, const float* __restrict__ up, __half* __restrict__ pl, float* __restrict__ inv_scale,
                                                                       float* __restrict__ last, int T, int F) {
  __shared__ float red[4];
  const long row = blockIdx.x; const int c0 = threadIdx.x * 4; float4 o[NV]; float mx = 0.f;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int c = c0 + 512 * k;
    if (c < F) {
      const float4 g = *reinterpret_cast<const float4*>(gate + row * F + c), u = *reinterpret_cast<const float4*>(up + row * F + c);
      o[k] = make_float4((g.x * act_fwd(GN_ACT_SIGMOID, g.x)) * u.x, (g.y * act_fwd(GN_ACT_SIGMOID, g.y)) * u.y, (g.z * act_fwd(GN_ACT_SIGMOID, g.z)) * u.z, (g.w * act_fwd(GN_ACT_SIGMOID, g.w)) * u.w);
      mx = max4(mx, o[k]);
    }
  }
  float inv; const float sc = row_scale(row_block_max(mx, red), &inv);
  if (threadIdx.x == 0) inv_scale[row] = inv;
  const bool is_last = row % T == T - 1;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int c = c0 + 512 * k; if (c >= F) break;
    planes_store4(pl + row * 2 * F, c, o[k], sc);
    if (is_last) *reinterpret_cast<float4*>(last + (row / T) * F + c) = o[k];
  }
}
__device__ __forceinline__ void swiglu_der(float g, float u, float go, float& dg, float& du) {
  const float sig = act_fwd(GN_ACT_SIGMOID, g), sw = g * sig;
  du = go * sw; dg = go * (sw + sig * (1.f - sw)) * u;
}
template <int NV>
__global__ void __launch_bounds__(SW_THREADS) swiglu_bwd_planes_kernel(const float* __restrict__ dOut, const float* __restrict__ gate, const float* __restrict__ up, float* __restrict__ dGateP,
                                                                       float* __restrict__ dUpP, __half* __restrict__ pl, float* __restrict__ inv_scale, int T, int F) {
  __shared__ float red[4];
  const long row = blockIdx.x, s = row / T, src = s * T + (T - 1 - (row - s * T)); const int c0 = threadIdx.x * 4; float4 dg[NV], du[NV]; float mx = 0.f;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int c = c0 + 512 * k;
    if (c < F) {
      const float4 g = *reinterpret_cast<const float4*>(gate + row * F + c), u = *reinterpret_cast<const float4*>(up + row * F + c), go = *reinterpret_cast<const float4*>(dOut + src * F + c);
      swiglu_der(g.x, u.x, go.x, dg[k].x, du[k].x); swiglu_der(g.y, u.y, go.y, dg[k].y, du[k].y); swiglu_der(g.z, u.z, go.z, dg[k].z, du[k].z); swiglu_der(g.w, u.w, go.w, dg[k].w, du[k].w);
      mx = max4(max4(mx, dg[k]), du[k]);
    }
  }
  float inv; const float sc = row_scale(row_block_max(mx, red), &inv);
  if (threadIdx.x == 0) inv_scale[row] = inv;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const int c = c0 + 512 * k; if (c >= F) break;
    *reinterpret_cast<float4*>(dGateP + row * F + c) = dg[k]; *reinterpret_cast<float4*>(dUpP + row * F + c) = du[k];
    planes_store4(pl + row * 4 * F, c, dg[k], sc); planes_store4(pl + row * 4 * F, F + c, du[k], sc);
  }
}
// The same for the gradient of token 0 alone: rows s of dOut, dGate, dUp are dense, the last token's projections lie `ld` apart
__global__ void swiglu_bwd_rows_kernel(const float* __restrict__ dOut, const float* __restrict__ gate, const float* __restrict__ up, long ld,
                                       float* __restrict__ dGate, float* __restrict__ dUp, int C, long total) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long s = e / C, o = s * ld + (e - s * C);
    const float g = gate[o], u = up[o], sig = act_fwd(GN_ACT_SIGMOID, g), sw = g * sig, go = dOut[e];
    dUp[e] = go * sw; dGate[e] = go * (sw + sig * (1.f - sw)) * u;
  }
}
// What a block's backward pass needs when only token 0 has a gradient: token 0's rows of the two norms' inputs and their statistics
// (st: mean 1 | deviation 1 | mean 2 | deviation 2, [B] each), the last token's rows of everything that meets a weight gradient.
struct KeepRows { float *r2, *r1, *n1, *att, *x, *mid, *gate, *up, *st; };
__global__ void __launch_bounds__(256) keep_rows_kernel(const float* __restrict__ r2, const float* __restrict__ r1, const float* __restrict__ n1, const float* __restrict__ att,
                                                        const float* __restrict__ x, const float* __restrict__ mid, const float* __restrict__ gate, const float* __restrict__ up,
                                                        const float* __restrict__ st, const KeepRows k, int T, int D, int F, int B) {
  const long s = blockIdx.x, N = (long)B * T, first = s * T, last = first + T - 1;
  for (int i = threadIdx.x; i < D; i += 256) {
    k.r2[s * D + i] = r2[first * D + i]; k.r1[s * D + i] = r1[first * D + i];
    k.n1[s * D + i] = n1[last * D + i]; k.att[s * D + i] = att[last * D + i]; k.x[s * D + i] = x[last * D + i];
  }
  for (int i = threadIdx.x; i < F; i += 256) {
    if (mid) k.mid[s * F + i] = mid[last * F + i];
    if (gate) { k.gate[s * F + i] = gate[last * F + i]; k.up[s * F + i] = up[last * F + i]; }
  }
  if (threadIdx.x < 4) k.st[threadIdx.x * (long)B + s] = st[threadIdx.x * N + first];
}
// dx[s, 0, :] += r[s, :]; one block per sequence
__global__ void add_row0_kernel(const float* __restrict__ r, float* __restrict__ dx, int T, int d) {
  for (int i = threadIdx.x; i < d; i += blockDim.x) dx[(long)blockIdx.x * T * d + i] += r[(long)blockIdx.x * d + i];
}
// out[s,t,:] = a[s,t,:] + b[s,T-1-t,:]
__global__ void add_token_reversed_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, int T, int C, long total) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long row = e / C; const int c = (int)(e - row * C); const long s = row / T; const int t = (int)(row - s * T);
    out[e] = a[e] + b[(s * T + (T - 1 - t)) * C + c];
  }
}

// ---------------------------------------------------------------- Adam
// reference: opt.go:237-251.  Every operation is rounded separately (no fused multiply-add), as the Go
// code does, so that the update is bit-identical to the CPU path for identical gradients.
//   g' = g * grad_scale (the 1/batch averaging of net.go:702-706, folded into this pass)
//   m = b1*m + (1-b1)*g' ; v = b2*v + (1-b2)*g'*g' ; p -= effLR * m / (sqrt(v) + eps)
// `status` (may be null): the context's status word; when a bounded wait of an earlier kernel of this step gave up, the
// gradients are not trustworthy and the pass leaves the parameters and moments untouched.
// `dargs` (may be null): the coefficients are read from there instead of `a`, so that a recorded launch follows the schedule.
// `ret` (may be null; host memory): receives the step's loss sum and the status word, the caller's one read-back.
struct AdamArgs { float effLR, b1, b2, omb1, omb2, eps, grad_scale; };
// `ranges` (MX): parameter ranges whose largest magnitude after the update is wanted, ascending; mx[j] (zero on entry) receives that of
// range j -- the operand planes of the weight matrices are scaled by it, and finding it here saves a pass over all of them.  A
// warp keeps the maximum of the range it is in in registers and hands it over when it leaves the range.  Memory-bound either way (28 bytes per parameter).
template <bool MX>
__global__ void __launch_bounds__(256) adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, long n, const AdamArgs a, const AdamArgs* __restrict__ dargs,
                                                   const int* __restrict__ status, const float* __restrict__ loss_sum, float* __restrict__ ret, const PlaneRange* __restrict__ ranges, int nr, int* __restrict__ mx) {
  if (ret && blockIdx.x == 0 && threadIdx.x == 0) { ret[0] = *loss_sum; ret[1] = __int_as_float(*status); }
  if (status && *status != 0) return;
  const AdamArgs c = dargs ? *dargs : a;
  const float effLR = c.effLR, b1 = c.b1, b2 = c.b2, omb1 = c.omb1, omb2 = c.omb2, eps = c.eps, grad_scale = c.grad_scale;
  // The four arrays are slices of the flat buffers at the same offset, so they share their position relative to a
  // 16-byte boundary: `head` leading elements are handled one by one, then float4s, then the tail.
  const long head = min(n, (long)((4 - ((reinterpret_cast<uintptr_t>(p) >> 2) & 3)) & 3));
  const long n4 = (n - head) >> 2;
  float4* p4 = reinterpret_cast<float4*>(p + head); const float4* g4 = reinterpret_cast<const float4*>(g + head);
  float4* m4 = reinterpret_cast<float4*>(m + head); float4* v4 = reinterpret_cast<float4*>(v + head);
  auto upd = [&](float& pp, float gg, float& mm, float& vv) {
    float gs = __fmul_rn(gg, grad_scale);
    mm = __fadd_rn(__fmul_rn(b1, mm), __fmul_rn(omb1, gs));
    vv = __fadd_rn(__fmul_rn(b2, vv), __fmul_rn(__fmul_rn(omb2, gs), gs));
    pp = __fsub_rn(pp, __fdiv_rn(__fmul_rn(effLR, mm), __fadd_rn(__fsqrt_rn(vv), eps)));
  };
  int j = 0; const float *js = nullptr, *je = nullptr; float mxv = 0.f; const int lane = threadIdx.x & 31;
  auto one = [&](const float* q, float x, int from) {        // a parameter near a range's edge
    for (int k = from; k < nr && ranges[k].b <= q; k++) if (q < ranges[k].e) atomicMax(mx + k, __float_as_int(fabsf(x)));
  };
  auto flush = [&]() {                                       // (the whole warp)
    const float t = warp_max(mxv); mxv = 0.f;
    if (lane == 0 && t > 0.f && t > __int_as_float(*(volatile int*)(mx + j))) atomicMax(mx + j, __float_as_int(t));
  };
  // (chunks of at most 32 KB per array, block by block: one contiguous run per block was 12 % slower at 134 M parameters)
  const long chunk = max(256L, min(2048L, ((n4 + gridDim.x - 1) / gridDim.x + 255) & ~255L));
  for (long i0 = blockIdx.x * chunk; i0 < n4; i0 += gridDim.x * chunk) {
    const long i1 = min(n4, i0 + chunk);
    for (long base = i0 + (threadIdx.x & ~31); base < i1; base += 256) {
      const long i = base + lane; const bool act = i < i1; float4 P = make_float4(0.f, 0.f, 0.f, 0.f);
      if (act) {
        const float4 G = g4[i]; float4 M = m4[i], V = v4[i]; P = p4[i];
        upd(P.x, G.x, M.x, V.x); upd(P.y, G.y, M.y, V.y); upd(P.z, G.z, M.z, V.z); upd(P.w, G.w, M.w, V.w);
        p4[i] = P; m4[i] = M; v4[i] = V;
      }
      if (MX) {
        const float* w0 = p + head + 4 * base; const float* q = w0 + 4 * lane;
        if (j < nr && w0 >= je) {                            // on to the first range that ends behind the warp's first parameter
          if (je) flush();
          int lo = j, hi = nr;
          while (lo < hi) { const int mid = (lo + hi) >> 1; if (ranges[mid].e > w0) hi = mid; else lo = mid + 1; }
          j = lo; if (j < nr) { js = ranges[j].b; je = ranges[j].e; }
        }
        if (j < nr && act) {
          if (q >= js && q + 4 <= je) mxv = fmaxf(mxv, fmaxf(fmaxf(fabsf(P.x), fabsf(P.y)), fmaxf(fabsf(P.z), fabsf(P.w))));
          else if (q + 4 > js) { one(q, P.x, j); one(q + 1, P.y, j); one(q + 2, P.z, j); one(q + 3, P.w, j); }
        }
      }
    }
  }
  if (MX && j < nr) flush();
  const long tid = blockIdx.x * (long)blockDim.x + threadIdx.x, nthreads = (long)gridDim.x * blockDim.x;
  if (tid < head) { upd(p[tid], g[tid], m[tid], v[tid]); if (MX) one(p + tid, p[tid], 0); }
  for (long i = head + (n4 << 2) + tid; i < n; i += nthreads) { upd(p[i], g[i], m[i], v[i]); if (MX) one(p + i, p[i], 0); }
}


// ---------------------------------------------------------------- BatchNorm2D (NCHW)
// The reference normalises ONE sample at a time, so the statistics of a (sample, channel) pair are taken over that
// sample's S = H*W positions (batchnorm2d.go:336-377).  One block per (sample, channel).
// stat layout: [B*C] mean | [B*C] std | [B*C] variance.
__global__ void bn_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ y,
                              float* __restrict__ stat, int C, int S, long BC, float eps) {
  __shared__ float red[33];
  const long bc = blockIdx.x; const int c = (int)(bc % C);
  const float* xp = x + bc * S; float* yp = y + bc * S;
  float s = 0.f;
  for (int i = threadIdx.x; i < S; i += blockDim.x) s += xp[i];
  const float mean = block_sum(s, red) * (1.f / (float)S);
  float ss = 0.f;
  for (int i = threadIdx.x; i < S; i += blockDim.x) { float d = xp[i] - mean; ss += d * d; }
  const float var = block_sum(ss, red) * (1.f / (float)S);
  const float sd = sqrtf(var + eps), istd = 1.f / sd, g = gamma[c], b = beta[c];
  for (int i = threadIdx.x; i < S; i += blockDim.x) yp[i] = g * ((xp[i] - mean) * istd) + b;
  if (threadIdx.x == 0) { stat[bc] = mean; stat[BC + bc] = sd; stat[2 * BC + bc] = var; }
}
// running = (1 - momentum) * running + momentum * statistic, once per sample in batch order (batchnorm2d.go:352, :376); `mean`, `var`:
// [B, C] per-sample statistics of the whole global batch (with several ranks every replica walks all of them).  A block stages 128
// samples of 32 channels at a time; one warp then walks the means, one the variances (from global memory: 30 us for 50 samples).
__global__ void __launch_bounds__(256) bn_running_kernel(const float* __restrict__ mean, const float* __restrict__ var, float* __restrict__ run, int B, int C, float mom) {
  __shared__ float st[2][128][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x * 32 + lane; const bool in = c < C;
  float r = in && w < 2 ? run[(long)w * C + c] : 0.f;
  for (int b0 = 0; b0 < B; b0 += 128) {
    const int n = min(128, B - b0);
    __syncthreads();
#pragma unroll 4
    for (int b = w; b < n; b += 8) if (in) { st[0][b][lane] = mean[(long)(b0 + b) * C + c]; st[1][b][lane] = var[(long)(b0 + b) * C + c]; }
    __syncthreads();
    if (w < 2) {
#pragma unroll 8
      for (int b = 0; b < n; b++) r = (1.f - mom) * r + mom * st[w][b][lane];
    }
  }
  if (in && w < 2) run[(long)w * C + c] = r;
}
// inference mode: running statistics (batchnorm2d.go:492-509)
__global__ void bn_eval_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ run,
                               float* __restrict__ y, int C, int S, long total, float eps) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int c = (int)((i / S) % C);
    y[i] = gamma[c] * ((x[i] - run[c]) / sqrtf(run[C + c] + eps)) + beta[c];
  }
}
// reference: batchnorm2d.go:626-660, m = S.  pg: per (sample, channel) contributions [B, 2C] = gGamma | gBeta, summed over samples afterwards.
__global__ void bn_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ stat,
                              float* __restrict__ dx, float* __restrict__ pg, int C, int S, long BC, int relu) {
  __shared__ float red[33];
  const long bc = blockIdx.x; const int c = (int)(bc % C); const long b = bc / C;
  const float* xp = x + bc * S; const float* gp = g + bc * S; float* dp = dx + bc * S;
  const float mean = stat[bc], sd = stat[BC + bc], gm = gamma[c], m = (float)S;
  float sg = 0.f, sgx = 0.f;
  for (int i = threadIdx.x; i < S; i += blockDim.x) { float gg = gp[i]; sg += gg; sgx += gg * (xp[i] - mean); }
  sg = block_sum(sg, red); sgx = block_sum(sgx, red);
  for (int i = threadIdx.x; i < S; i += blockDim.x) {
    float d = xp[i] - mean, gi = gp[i] * gm;
    const float v = gi / sd - (sg * gm) / m / sd - d * (sgx * gm) / m / (sd * sd * sd);
    dp[i] = relu && !(xp[i] > 0.f) ? 0.f : v;               // (the derivative of a ReLU right below: its output is this layer's input)
  }
  if (threadIdx.x == 0) { pg[b * 2 * C + c] = sgx / sd; pg[b * 2 * C + C + c] = sg; }     // sum g*(x-mean)/std ; sum g
}

}  // namespace gn
