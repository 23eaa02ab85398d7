// conv_lstm.cuh -- Conv2D / MaxPool2D kernels (NCHW), wide GRUs, and the LSTM clipping recurrence on the gradient matrix itself.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"
#include "rowops.cuh"

namespace gn {
namespace cg = cooperative_groups;

struct ConvShape { int B, inC, outC, k, s, p, H, W, oH, oW; };

// z[b,oc,oh,ow] = bias[oc] + sum_{ic,kh,kw} W[oc,ic,kh,kw] x[b,ic,oh*s+kh-p,ow*s+kw-p]; a = act(z)
// reference: conv2d.go:716-959 (zero padding = out-of-range taps skipped; bias added last)
__global__ void conv2d_fwd_kernel(const float* __restrict__ x, const float* __restrict__ Wt, const float* __restrict__ bias,
                                  float* __restrict__ z, float* __restrict__ a, ConvShape c, int act, float alpha) {
  long total = (long)c.B * c.outC * c.oH * c.oW;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int ow = (int)(i % c.oW); long r = i / c.oW; int oh = (int)(r % c.oH); r /= c.oH; int oc = (int)(r % c.outC); int b = (int)(r / c.outC);
    const float* xb = x + (long)b * c.inC * c.H * c.W;
    const float* w = Wt + (long)oc * c.inC * c.k * c.k;
    float acc = 0.f;
    for (int ic = 0; ic < c.inC; ic++)
      for (int kh = 0; kh < c.k; kh++) {
        int ih = oh * c.s + kh - c.p; if (ih < 0 || ih >= c.H) continue;
        for (int kw = 0; kw < c.k; kw++) {
          int iw = ow * c.s + kw - c.p; if (iw < 0 || iw >= c.W) continue;
          acc = fmaf(__ldg(w + (ic * c.k + kh) * c.k + kw), xb[((long)ic * c.H + ih) * c.W + iw], acc);
        }
      }
    acc += bias[oc];
    z[i] = acc; a[i] = act_fwd(act, acc, alpha);
  }
}
// dx[b,ic,ih,iw] = sum_{oc,kh,kw} g[b,oc,oh,ow] W[oc,ic,kh,kw] with oh*s+kh-p = ih   (conv2d.go:1151-1162)
__global__ void conv2d_dgrad_kernel(const float* __restrict__ g, const float* __restrict__ Wt, float* __restrict__ dx, ConvShape c) {
  long total = (long)c.B * c.inC * c.H * c.W;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int iw = (int)(i % c.W); long r = i / c.W; int ih = (int)(r % c.H); r /= c.H; int ic = (int)(r % c.inC); int b = (int)(r / c.inC);
    const float* gb = g + (long)b * c.outC * c.oH * c.oW;
    float acc = 0.f;
    for (int oc = 0; oc < c.outC; oc++)
      for (int kh = 0; kh < c.k; kh++) {
        int th = ih + c.p - kh; if (th < 0 || th % c.s) continue; int oh = th / c.s; if (oh >= c.oH) continue;
        for (int kw = 0; kw < c.k; kw++) {
          int tw = iw + c.p - kw; if (tw < 0 || tw % c.s) continue; int ow = tw / c.s; if (ow >= c.oW) continue;
          acc = fmaf(gb[((long)oc * c.oH + oh) * c.oW + ow], __ldg(Wt + (((long)oc * c.inC + ic) * c.k + kh) * c.k + kw), acc);
        }
      }
    dx[i] = acc;
  }
}
// The same for stride 1 (no divisions in the tap loops, which are unrolled): images that the register-tiled kernels do not take.  Four
// images of 640 x 640, 8 -> 16 channels: 4.3 ms less than above with a 3 x 3 window, 10 with 5 x 5.
template <int K>
__global__ void __launch_bounds__(256) conv2d_dgrad_s1_kernel(const float* __restrict__ g, const float* __restrict__ Wt, float* __restrict__ dx, ConvShape c) {
  const long total = (long)c.B * c.inC * c.H * c.W;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int iw = (int)(i % c.W); long r = i / c.W; const int ih = (int)(r % c.H); r /= c.H; const int ic = (int)(r % c.inC), b = (int)(r / c.inC);
    const float* gb = g + (long)b * c.outC * c.oH * c.oW;
    float acc = 0.f;
    for (int oc = 0; oc < c.outC; oc++) {
      const float* gp = gb + (long)oc * c.oH * c.oW; const float* wp = Wt + ((long)oc * c.inC + ic) * K * K;
#pragma unroll
      for (int kh = 0; kh < K; kh++) {
        const int oh = ih + c.p - kh; if (oh < 0 || oh >= c.oH) continue;
#pragma unroll
        for (int kw = 0; kw < K; kw++) {
          const int ow = iw + c.p - kw; if (ow < 0 || ow >= c.oW) continue;
          acc = fmaf(gp[oh * c.oW + ow], __ldg(wp + kh * K + kw), acc);
        }
      }
    }
    dx[i] = acc;
  }
}
// One block per weight: dW[oc,ic,kh,kw] = sum_{b,oh,ow} g * x ; blocks >= nW reduce one bias each.
__global__ void conv2d_wgrad_kernel(const float* __restrict__ g, const float* __restrict__ x, float* __restrict__ dW, float* __restrict__ db, ConvShape c) {
  __shared__ float red[33];
  int nW = c.outC * c.inC * c.k * c.k;
  int wi = blockIdx.x;
  long span = (long)c.B * c.oH * c.oW;
  float s = 0.f;
  if (wi < nW) {
    int kw = wi % c.k; int r = wi / c.k; int kh = r % c.k; r /= c.k; int ic = r % c.inC; int oc = r / c.inC;
    for (long i = threadIdx.x; i < span; i += blockDim.x) {
      int ow = (int)(i % c.oW); long q = i / c.oW; int oh = (int)(q % c.oH); int b = (int)(q / c.oH);
      int ih = oh * c.s + kh - c.p, iw = ow * c.s + kw - c.p;
      if (ih < 0 || ih >= c.H || iw < 0 || iw >= c.W) continue;
      s = fmaf(g[(((long)b * c.outC + oc) * c.oH + oh) * c.oW + ow], x[(((long)b * c.inC + ic) * c.H + ih) * c.W + iw], s);
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) dW[wi] = s;
  } else {
    int oc = wi - nW;
    for (long i = threadIdx.x; i < span; i += blockDim.x) {
      long q = i / ((long)c.oH * c.oW); long rem = i % ((long)c.oH * c.oW);
      s += g[((long)q * c.outC + oc) * c.oH * c.oW + rem];
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) db[oc] = s;
  }
}

// Weight gradient, tiled: one block per (oc, ic) pair and batch slice, so the K*K taps of the pair share every load of
// g and the input plane is read from L1; partial sums go to part[slice][nW + outC] (bias partials from the ic == 0
// blocks) and conv_wgrad_final_kernel adds the slices in order.  Same sums as conv2d_wgrad_kernel.
template <int K>
__global__ void __launch_bounds__(256) conv2d_wgrad_tile_kernel(const float* __restrict__ g, const float* __restrict__ x, float* __restrict__ part, ConvShape c, int slices) {
  __shared__ float red[8][K * K + 1];
  const int pair = blockIdx.x, oc = pair / c.inC, ic = pair % c.inC, sl = blockIdx.y;
  const int bper = (c.B + slices - 1) / slices, b0 = sl * bper, b1 = min(c.B, b0 + bper);
  const int npos = c.oH * c.oW, nW = c.outC * c.inC * K * K;
  float acc[K * K], sb = 0.f;
#pragma unroll
  for (int t = 0; t < K * K; t++) acc[t] = 0.f;
  const long span = (long)max(0, b1 - b0) * npos;
  for (long i = threadIdx.x; i < span; i += 256) {
    const int b = b0 + (int)(i / npos), pos = (int)(i % npos), oh = pos / c.oW, ow = pos - oh * c.oW;
    const float gv = g[(((long)b * c.outC + oc) * c.oH + oh) * c.oW + ow];
    sb += gv;
    const float* xb = x + ((long)b * c.inC + ic) * c.H * c.W;
#pragma unroll
    for (int kh = 0; kh < K; kh++) {
      const int ih = oh * c.s + kh - c.p; if (ih < 0 || ih >= c.H) continue;
#pragma unroll
      for (int kw = 0; kw < K; kw++) {
        const int iw = ow * c.s + kw - c.p; if (iw < 0 || iw >= c.W) continue;
        acc[kh * K + kw] = fmaf(gv, xb[ih * c.W + iw], acc[kh * K + kw]);
      }
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int t = 0; t < K * K; t++) { const float v = warp_sum(acc[t]); if (lane == 0) red[w][t] = v; }
  sb = warp_sum(sb); if (lane == 0) red[w][K * K] = sb;
  __syncthreads();
  if (threadIdx.x <= K * K) {
    float v = 0.f;
    for (int q = 0; q < 8; q++) v += red[q][threadIdx.x];
    float* prow = part + (long)sl * (nW + c.outC);
    if (threadIdx.x < K * K) prow[(long)pair * K * K + threadIdx.x] = v;
    else if (ic == 0) prow[nW + oc] = v;
  }
}
// ---------------------------------------------------------------- Conv1D
// Input [B, inC, L], output [B, outC, oL], weights [outC, inC, k].  reference: conv1d.go:178-216 (the sum starts from the
// bias), :254-288 (the backward pass uses the incoming gradient as it is: no activation derivative).
struct Conv1Shape { int B, inC, outC, k, s, p, L, oL; };
__global__ void conv1d_fwd_kernel(const float* __restrict__ x, const float* __restrict__ Wt, const float* __restrict__ bias, float* __restrict__ y,
                                  Conv1Shape c, int act, float alpha) {
  long total = (long)c.B * c.outC * c.oL;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int ol = (int)(i % c.oL); long r = i / c.oL; int oc = (int)(r % c.outC); int b = (int)(r / c.outC);
    const float* xb = x + (long)b * c.inC * c.L; const float* w = Wt + (long)oc * c.inC * c.k;
    float sum = bias[oc];
    for (int ic = 0; ic < c.inC; ic++) for (int k = 0; k < c.k; k++) {
      int pos = ol * c.s + k - c.p;
      if (pos >= 0 && pos < c.L) sum = fmaf(xb[(long)ic * c.L + pos], __ldg(w + ic * c.k + k), sum);
    }
    y[i] = act_fwd(act, sum, alpha);
  }
}
__global__ void conv1d_dgrad_kernel(const float* __restrict__ g, const float* __restrict__ Wt, float* __restrict__ dx, Conv1Shape c) {
  long total = (long)c.B * c.inC * c.L;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int pos = (int)(i % c.L); long r = i / c.L; int ic = (int)(r % c.inC); int b = (int)(r / c.inC);
    const float* gb = g + (long)b * c.outC * c.oL;
    float acc = 0.f;
    for (int oc = 0; oc < c.outC; oc++) for (int k = 0; k < c.k; k++) {
      int t = pos + c.p - k; if (t < 0 || t % c.s) continue; int ol = t / c.s; if (ol >= c.oL) continue;
      acc = fmaf(gb[(long)oc * c.oL + ol], __ldg(Wt + ((long)oc * c.inC + ic) * c.k + k), acc);
    }
    dx[i] = acc;
  }
}
// One block per weight: dW[oc,ic,k] = sum_{b,ol} g x ; blocks >= nW reduce one bias each.
__global__ void conv1d_wgrad_kernel(const float* __restrict__ g, const float* __restrict__ x, float* __restrict__ dW, float* __restrict__ db, Conv1Shape c) {
  __shared__ float red[33];
  const int nW = c.outC * c.inC * c.k, wi = blockIdx.x; const long span = (long)c.B * c.oL;
  float s = 0.f;
  if (wi < nW) {
    const int k = wi % c.k; int r = wi / c.k; const int ic = r % c.inC, oc = r / c.inC;
    for (long i = threadIdx.x; i < span; i += blockDim.x) {
      const int ol = (int)(i % c.oL), b = (int)(i / c.oL), pos = ol * c.s + k - c.p;
      if (pos < 0 || pos >= c.L) continue;
      s = fmaf(g[((long)b * c.outC + oc) * c.oL + ol], x[((long)b * c.inC + ic) * c.L + pos], s);
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) dW[wi] = s;
  } else {
    const int oc = wi - nW;
    for (long i = threadIdx.x; i < span; i += blockDim.x) s += g[((long)(i / c.oL) * c.outC + oc) * c.oL + i % c.oL];
    s = block_sum(s, red);
    if (threadIdx.x == 0) db[oc] = s;
  }
}

struct PoolShape { int B, C, k, s, p, H, W, oH, oW; };
// reference: maxpool2d.go:192-221 (init -inf, strict '>', first maximum wins, argmax = flat CHW index).  A block takes pieces of one
// (sample, channel) plane: the index arithmetic is 32-bit and per pixel of the plane.
__global__ void __launch_bounds__(256) maxpool_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, int* __restrict__ arg, PoolShape c) {
  const long pl = blockIdx.x; const int ch = (int)(pl % c.C); const float* xp = x + pl * c.H * c.W;
  for (unsigned at = blockIdx.y * 256 + threadIdx.x; at < (unsigned)(c.oH * c.oW); at += gridDim.y * 256) {
    const int i = (int)at, oh = i / c.oW, ow = i - oh * c.oW, h0 = oh * c.s - c.p, w0 = ow * c.s - c.p;
    float mv = -INFINITY; int mi = -1;
    if (c.k == 2 && c.p == 0) {                              // whole windows: both rows in flight
      const float* q = xp + h0 * c.W + w0; const float a = q[0], b = q[1], d = q[c.W], e = q[c.W + 1]; const int first = (ch * c.H + h0) * c.W + w0;
      if (a > mv) { mv = a; mi = first; } if (b > mv) { mv = b; mi = first + 1; } if (d > mv) { mv = d; mi = first + c.W; } if (e > mv) { mv = e; mi = first + c.W + 1; }
    } else for (int kh = 0; kh < c.k; kh++) for (int kw = 0; kw < c.k; kw++) {
      const int ih = h0 + kh, iw = w0 + kw;
      if (ih >= 0 && ih < c.H && iw >= 0 && iw < c.W) { const float v = xp[ih * c.W + iw]; if (v > mv) { mv = v; mi = (ch * c.H + ih) * c.W + iw; } }
    }
    y[pl * c.oH * c.oW + i] = mv; arg[pl * c.oH * c.oW + i] = mi;
  }
}
// Windows that do not overlap: every input element looks its one window up (no zero fill, no atomics).  `relu`: the derivative of a
// ReLU right below is applied as well -- the element that won its window passes the gradient on only if it is positive (y > 0).
__global__ void __launch_bounds__(256) maxpool_bwd_gather_kernel(const float* __restrict__ g, const int* __restrict__ arg, const float* __restrict__ y, float* __restrict__ dx, PoolShape c, int relu) {
  const long pl = blockIdx.x; const int ch = (int)(pl % c.C);
  for (unsigned at = blockIdx.y * 256 + threadIdx.x; at < (unsigned)(c.H * c.W); at += gridDim.y * 256) {
    const int i = (int)at, ih = i / c.W, iw = i - ih * c.W, oh = (ih + c.p) / c.s, ow = (iw + c.p) / c.s; float v = 0.f;
    if (oh < c.oH && ow < c.oW) { const long o = pl * c.oH * c.oW + oh * c.oW + ow; if (arg[o] == ch * c.H * c.W + i && (!relu || y[o] > 0.f)) v = g[o]; }
    dx[pl * c.H * c.W + i] = v;
  }
}
// 2 x 2 windows that tile the plane (W even, 8-byte aligned rows): a thread per window
__global__ void __launch_bounds__(256) maxpool_bwd_2x2_kernel(const float* __restrict__ g, const int* __restrict__ arg, const float* __restrict__ y, float* __restrict__ dx, PoolShape c, int relu) {
  const long pl = blockIdx.x;
  for (unsigned at = blockIdx.y * 256 + threadIdx.x; at < (unsigned)(c.oH * c.oW); at += gridDim.y * 256) {
    const int i = (int)at, oh = i / c.oW, ow = i - oh * c.oW; const long o = pl * c.oH * c.oW + i;
    const float v = relu && !(y[o] > 0.f) ? 0.f : g[o]; const int d = arg[o] - (((int)(pl % c.C) * c.H + 2 * oh) * c.W + 2 * ow);
    float* q = dx + (pl * c.H + 2 * oh) * c.W + 2 * ow;
    *reinterpret_cast<float2*>(q) = make_float2(d == 0 ? v : 0.f, d == 1 ? v : 0.f);
    *reinterpret_cast<float2*>(q + c.W) = make_float2(d == c.W ? v : 0.f, d == c.W + 1 ? v : 0.f);
  }
}
// dx zero-filled beforehand; windows may overlap when stride < kernel, hence the atomic add (maxpool2d.go:395-406)
__global__ void maxpool_bwd_kernel(const float* __restrict__ g, const int* __restrict__ arg, float* __restrict__ dx, PoolShape c) {
  long total = (long)c.B * c.C * c.oH * c.oW; long per_out = (long)c.C * c.oH * c.oW, per_in = (long)c.C * c.H * c.W;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int a = arg[i]; if (a >= 0) atomicAdd(dx + (i / per_out) * per_in + a, g[i]);
  }
}

// Average pooling: mean over the taps inside the input (padded taps are not counted; a window with no valid tap
// gives 0).  reference: avgpool2d.go:172-228
__global__ void avgpool_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, PoolShape c) {
  long total = (long)c.B * c.C * c.oH * c.oW;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int ow = (int)(i % c.oW); long r = i / c.oW; int oh = (int)(r % c.oH); r /= c.oH;      // r = b * C + ch
    const float* xp = x + r * c.H * c.W;
    float sum = 0.f; int cnt = 0;
    for (int kh = 0; kh < c.k; kh++) for (int kw = 0; kw < c.k; kw++) {
      int ih = oh * c.s + kh - c.p, iw = ow * c.s + kw - c.p;
      if (ih >= 0 && ih < c.H && iw >= 0 && iw < c.W) { sum += xp[ih * c.W + iw]; cnt++; }
    }
    y[i] = cnt > 0 ? sum * (1.f / (float)cnt) : 0.f;
  }
}
// Backward in gather form (one thread per input element, no atomics): dx = sum over the windows that contain the element
// of g / count(window), windows visited in the reference's (oh, ow) order.  reference: avgpool2d.go:441-468
__global__ void avgpool_bwd_kernel(const float* __restrict__ g, float* __restrict__ dx, PoolShape c) {
  long total = (long)c.B * c.C * c.H * c.W;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    int iw = (int)(i % c.W); long r = i / c.W; int ih = (int)(r % c.H); r /= c.H;          // r = b * C + ch
    const float* gp = g + r * c.oH * c.oW;
    float acc = 0.f;
    for (int oh = 0; oh < c.oH; oh++) {
      int kh = ih - oh * c.s + c.p; if (kh < 0 || kh >= c.k) continue;
      for (int ow = 0; ow < c.oW; ow++) {
        int kw = iw - ow * c.s + c.p; if (kw < 0 || kw >= c.k) continue;
        int cnt = 0;
        for (int a = 0; a < c.k; a++) for (int b = 0; b < c.k; b++) {
          int h2 = oh * c.s + a - c.p, w2 = ow * c.s + b - c.p;
          if (h2 >= 0 && h2 < c.H && w2 >= 0 && w2 < c.W) cnt++;
        }
        acc += gp[oh * c.oW + ow] * (1.f / (float)cnt);
      }
    }
    dx[i] = acc;
  }
}

// ---------------------------------------------------------------- GRU with more than 128 units (smaller ones: recurrent.cuh)
// Forward recurrence of one sample per block, thread i = hidden unit i.  reference: gru.go:192-288.
// `pre` [B, T, 3H] holds b + Wx x_t of every step on entry (one contraction over all B*T rows, issued before) and the
// complete pre-activations (update | reset | candidate) on exit.  The layer has 2H recurrent rows: the candidate's
// recurrent product uses the reset gate's rows on r (.) h_prev (gru.go:247-258).
__global__ void gru_fwd_kernel(const float* __restrict__ Wh, float* __restrict__ pre, float* __restrict__ h_all, float* __restrict__ out, int T, int H, int return_seq) {
  extern __shared__ float sm[];
  float* WzT = sm;                   // [H][H]  WzT[j*H+i] = Wh[i, j]        (update rows)
  float* WrT = WzT + (long)H * H;    // [H][H]  WrT[j*H+i] = Wh[H + i, j]    (reset rows)
  float* hbuf = WrT + (long)H * H;   // [2][H]
  float* rh = hbuf + 2 * H;          // [H]  r (.) h_prev
  const int s = blockIdx.x, i = threadIdx.x;
  for (int e = threadIdx.x; e < H * H; e += blockDim.x) { const int r = e / H, j = e % H; WzT[j * H + r] = Wh[e]; WrT[j * H + r] = Wh[(long)H * H + e]; }
  if (i < H) { hbuf[i] = 0.f; hbuf[H + i] = 0.f; }
  __syncthreads();
  for (int t = 0; t < T; t++) {
    const float* hp = hbuf + (t & 1) * H; float* hn = hbuf + ((t + 1) & 1) * H;
    float* pr = pre + ((long)s * T + t) * 3 * H;
    float pz = 0.f, prr = 0.f, z = 0.f, hprev = 0.f;
    if (i < H) {
      pz = pr[i]; prr = pr[H + i]; hprev = hp[i];
      for (int j = 0; j < H; j++) { const float hj = hp[j]; pz = fmaf(WzT[j * H + i], hj, pz); prr = fmaf(WrT[j * H + i], hj, prr); }
      z = act_fwd(GN_ACT_SIGMOID, pz);
      rh[i] = act_fwd(GN_ACT_SIGMOID, prr) * hprev;
    }
    __syncthreads();
    if (i < H) {
      float pc = pr[2 * H + i];
      for (int j = 0; j < H; j++) pc = fmaf(WrT[j * H + i], rh[j], pc);
      const float c = act_fwd(GN_ACT_TANH, pc);
      const float h = hprev + z * (c - hprev);
      pr[i] = pz; pr[H + i] = prr; pr[2 * H + i] = pc;
      const long o = ((long)s * T + t) * H + i;
      h_all[o] = h; hn[i] = h;
      if (return_seq) out[o] = h; else if (t == T - 1) out[(long)s * H + i] = h;
    }
    __syncthreads();
  }
}
// Back-propagation through time of one sample per block.  reference: gru.go:360-534 with unroller.go:190-209, literal:
// the reset gate's delta is never formed (stays zero), the candidate's gradient is scaled by (1 - z) and the
// hidden-state pass-through by z, the candidate's contribution to dh_prev is indexed by the output unit's reset gate,
// and dh_prev is ADDED to the incoming gradient before it is handed to the previous step.
// Writes the gate deltas D [B,T,3H] (update | zero | candidate), h_{t-1} [B,T,H] and r (.) h_{t-1} [B,T,H] for the
// weight-gradient contractions.
__global__ void gru_bwd_kernel(const float* __restrict__ gout, const float* __restrict__ Wh, const float* __restrict__ pre, const float* __restrict__ h_all,
                               float* __restrict__ D, float* __restrict__ hprev_all, float* __restrict__ rh_all, int T, int H, int return_seq) {
  extern __shared__ float sm[];
  float* dU = sm; float* dCr = sm + H;
  const int s = blockIdx.x, i = threadIdx.x;
  float cur = 0.f;
  for (int t = T - 1; t >= 0; t--) {
    float z = 0.f;
    if (i < H) {
      if (return_seq) cur += gout[((long)s * T + t) * H + i]; else if (t == T - 1) cur += gout[(long)s * H + i];
      const float* pr = pre + ((long)s * T + t) * 3 * H;
      z = act_fwd(GN_ACT_SIGMOID, pr[i]);
      const float r = act_fwd(GN_ACT_SIGMOID, pr[H + i]), c = act_fwd(GN_ACT_TANH, pr[2 * H + i]);
      const long o = ((long)s * T + t) * H + i;
      const float hprev = t > 0 ? h_all[o - H] : 0.f;
      const float du = cur * (c - hprev) * z * (1.f - z);
      const float dc = cur * (1.f - z) * (1.f - c * c);
      float* Dr = D + ((long)s * T + t) * 3 * H;
      Dr[i] = du; Dr[H + i] = 0.f; Dr[2 * H + i] = dc;
      hprev_all[o] = hprev; rh_all[o] = r * hprev;
      dU[i] = du; dCr[i] = dc * r;
    }
    __syncthreads();
    if (i < H) {
      float sum = 0.f;
      for (int j = 0; j < H; j++) sum = fmaf(Wh[(long)j * H + i], dU[j], sum);
      for (int j = 0; j < H; j++) sum = fmaf(Wh[((long)H + j) * H + i], dCr[j], sum);
      cur = cur + (sum + cur * z);
    }
    __syncthreads();
  }
}
// The reference clips the WHOLE accumulated LSTM gradient to L2 norm <= 1 after every time-step of every
// sample (lstm.go:694, :725-751), so the gradient of a worker chunk is a sequential recurrence over its
// (sample, t) updates  g <- clip(g + d_k (x) [x_last ; h_{t-1} ; 1]).  One thread-block cluster runs one
// chunk: the 4H gradient rows are split over the cluster's CTAs, each keeps its rows in shared memory,
// and the squared norm is exchanged through distributed shared memory once per update.
// Row r of the running gradient is [gWx[r,:] | gWh[r,:] | gb[r]].
constexpr int SCAN_CLUSTER = 8, SCAN_THREADS = 256;
__global__ void __launch_bounds__(SCAN_THREADS) lstm_grad_scan_kernel(
    const float* __restrict__ D, const float* __restrict__ x, const float* __restrict__ h_all, float* __restrict__ out,
    int T, int in, int H, int n_samples_total, int chunk, int first_sample_offset) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cluster.block_rank();
  const int cl = blockIdx.x / SCAN_CLUSTER;                    // which worker chunk
  const int R4 = 4 * H, ZW = in + H + 1;
  const int rpc = (R4 + SCAN_CLUSTER - 1) / SCAN_CLUSTER, row0 = rank * rpc, nrows = max(0, min(rpc, R4 - row0));
  extern __shared__ float sm[];
  float* acc = sm;                         // [rpc][ZW]
  float* dsh = acc + (long)rpc * ZW;       // [rpc]
  float* zsh = dsh + rpc;                  // [ZW]
  float* red = zsh + ZW;                   // [33]
  __shared__ float part[2][SCAN_CLUSTER];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = SCAN_THREADS >> 5;
  for (int e = tid; e < rpc * ZW; e += SCAN_THREADS) acc[e] = 0.f;
  cluster.sync();
  // samples of this chunk, relative to the tensors passed in
  int s_begin = cl * chunk - first_sample_offset, s_end = min(n_samples_total, s_begin + chunk);
  s_begin = max(s_begin, 0);
  long step = 0;
  for (int s = s_begin; s < s_end; s++) {
    for (int t = T - 1; t >= 0; t--, step++) {
      const int buf = (int)(step & 1);
      const float* Dr = D + ((long)s * T + t) * R4 + row0;
      for (int e = tid; e < nrows; e += SCAN_THREADS) dsh[e] = Dr[e];
      for (int e = tid; e < ZW; e += SCAN_THREADS) {
        float v;
        if (e < in) v = x[(long)s * T * in + (long)(T - 1) * in + e];           // lstm.go:592-621: input of the LAST forward call
        else if (e < in + H) v = t > 0 ? h_all[((long)s * T + (t - 1)) * H + (e - in)] : 0.f;
        else v = 1.f;
        zsh[e] = v;
      }
      __syncthreads();
      float sq = 0.f;
      for (int r = warp; r < nrows; r += nwarps) {
        float dr = dsh[r]; float* a = acc + (long)r * ZW;
        for (int c = lane; c < ZW; c += 32) { float v = fmaf(dr, zsh[c], a[c]); a[c] = v; sq = fmaf(v, v, sq); }
      }
      sq = block_sum(sq, red);
      if (tid < SCAN_CLUSTER) { float* remote = cluster.map_shared_rank(&part[buf][rank], tid); *remote = sq; }
      cluster.sync();
      float total = 0.f;
#pragma unroll
      for (int q = 0; q < SCAN_CLUSTER; q++) total += part[buf][q];
      float norm = sqrtf(total);
      if (norm > 1.f) {
        float sc = 1.f / norm;
        for (int r = warp; r < nrows; r += nwarps) { float* a = acc + (long)r * ZW; for (int c = lane; c < ZW; c += 32) a[c] *= sc; }
      }
    }
  }
  __syncthreads();
  // write out in the flat layout: gWx[4H,in] | gWh[4H,H] | gb[4H]
  float* o = out + (long)cl * ((long)R4 * ZW);
  for (int e = tid; e < nrows * ZW; e += SCAN_THREADS) {
    int r = e / ZW, c = e % ZW, gr = row0 + r; float v = acc[(long)r * ZW + c];
    if (c < in) o[(long)gr * in + c] = v;
    else if (c < in + H) o[(long)R4 * in + (long)gr * H + (c - in)] = v;
    else o[(long)R4 * in + (long)R4 * H + gr] = v;
  }
  cluster.sync();
}

}  // namespace gn
