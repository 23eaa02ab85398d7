// recurrent.cuh -- LSTM and GRU recurrences, forward and back-propagation through time, and the LSTM gradient-clipping recurrence.
#pragma once
#include <cooperative_groups.h>
#include <type_traits>
#include "common.cuh"
#include "rowops.cuh"
#include "update_rows.cuh"

namespace gn {

// ------------------------------------------------------------------ recurrence kernels
// A recurrence is a chain of T small matrix-vector products, bound by the latency of one step.  A block owns NS samples (two when
// there are more samples than SMs).  For up to 128 hidden units (HB blocks of 32) a thread has C columns of the matrix and a 2 C-th
// of the contraction, and keeps their weights for the whole sequence.  The 2 C threads of a column group are
// neighbours in a warp: every 16 bytes of the vector that a lane fetches are used for C columns, and rounds of shuffles that halve what a lane
// still holds leave every lane with the sum of ONE unit of ONE sample, the unit whose element-wise part it does.  A step is
// that, and one barrier behind the new vector.
// Four threads per unit, a column each, fetched four times as much of the vector (shared memory delivers 128 bytes per clock to
// registers, broadcast or not: 4096 of the 5000 cycles of a backward step of the LSTM), and passed partial sums through shared memory behind a second
// barrier.  us before -> now, 64 steps of 128 units, 256 samples: LSTM 65.6 -> 49 forward, 166 -> 80 backward, GRU 210 -> 94 and 122 -> 53; 100
// samples: 49 -> 44, 123 -> 57, 143 -> 80 and 74 -> 49.  What is left of a step is its chain: 0.46 us for 32 units.
// (fma.rn.f32x2, two rows at a time, is no faster here: LSTM backward, 96 units, 71.8 us against 63.5.)
struct RecShape { int T, in, H, return_seq, B; };
__host__ __device__ __forceinline__ int rec_hp(int H) { return (H + 31) & ~31; }
__host__ __device__ __forceinline__ int rec_jq(int H) { return (((H + 3) / 4) + 3) & ~3; }        // length of a quarter, a multiple of 4
constexpr int REC_REG_H = 128;                               // units up to which the register kernels go
// Floats between the pieces (of ks values, a multiple of four) of a vector: an odd number of 16-byte units, so that they lie in different banks
__host__ __device__ constexpr int rec_vs(int ks) { return ks | 4; }

// acc[s][c] += w[.][c] . v_s over R values; the samples' vectors are `vs` floats apart
template <int NS, int R, int C>
__device__ __forceinline__ void rec_fma(float (&acc)[NS][C], const float (&w)[R][C], const float* __restrict__ v, int vs) {
#pragma unroll
  for (int r = 0; r < R; r += 4) {
#pragma unroll
    for (int s = 0; s < NS; s++) {
      const float4 x = *reinterpret_cast<const float4*>(v + s * vs + r);
#pragma unroll
      for (int c = 0; c < C; c++) acc[s][c] = fmaf(w[r + 3][c], x.w, fmaf(w[r + 2][c], x.z, fmaf(w[r + 1][c], x.y, fmaf(w[r][c], x.x, acc[s][c]))));
    }
  }
}
// The sums over the 2 C threads of a column group; lane C s + c of the group receives column c of sample s (NS = 1: so do lanes C + c)
template <int NS, int C>
__device__ __forceinline__ float rec_reduce(const float (&acc)[NS][C], int lane) {
  float v[NS * C];
#pragma unroll
  for (int s = 0; s < NS; s++)
#pragma unroll
    for (int c = 0; c < C; c++) v[C * s + c] = acc[s][c];
  if (NS == 1) {                               // (the order of a sample's sums does not depend on NS)
#pragma unroll
    for (int c = 0; c < C; c++) v[c] += __shfl_xor_sync(0xffffffffu, v[c], C);
  }
#pragma unroll
  for (int h = NS * C / 2; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int k = 0; k < h; k++) { const float give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k]; v[k] = keep + __shfl_xor_sync(0xffffffffu, give, h); }
  }
  return v[0];
}
template <int NS, int C> __device__ __forceinline__ void rec_clear(float (&acc)[NS][C]) {
#pragma unroll
  for (int s = 0; s < NS; s++)
#pragma unroll
    for (int c = 0; c < C; c++) acc[s][c] = 0.f;
}
// Rows k .. k + 3 (k a multiple of four) of columns col0 .. col0 + C - 1 of a matrix [H, H], zero outside.  KFAST: element (row k, column c)
// lies at m[c * H + k], else at m[k * H + c].  `vec`: H is a multiple of four and m 16-byte aligned.
template <bool KFAST, int C>
__device__ __forceinline__ void rec_weights(float (*w)[C], const float* __restrict__ m, int H, int k, int col0, bool vec) {
#pragma unroll
  for (int c4 = 0; c4 < C; c4 += 4)
#pragma unroll
    for (int a = 0; a < 4; a++) {
      const int slow = KFAST ? col0 + c4 + a : k + a, fast = KFAST ? k : col0 + c4; const float* q = m + (long)slow * H + fast; float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (slow < H && fast < H) {
        if (vec) { const float4 y = *reinterpret_cast<const float4*>(q); x[0] = y.x; x[1] = y.y; x[2] = y.z; x[3] = y.w; }
        else { x[0] = q[0]; if (fast + 1 < H) x[1] = q[1]; if (fast + 2 < H) x[2] = q[2]; if (fast + 3 < H) x[3] = q[3]; }
      }
#pragma unroll
      for (int b = 0; b < 4; b++) w[KFAST ? b : a][c4 + (KFAST ? a : b)] = x[b];
    }
}
__device__ __forceinline__ bool rec_vec(const float* m, int H) { return ((reinterpret_cast<uintptr_t>(m) | (uintptr_t)(H * 4)) & 15) == 0; }
// This thread's part of the recurrence: column group, piece of the contraction, and the (sample, unit) whose element-wise part it does
template <int NS, int C> struct RecLane {
  int lane, sp, col0, unit, es; long s; bool el;
  __device__ __forceinline__ RecLane(int H, int B) {
    lane = threadIdx.x & 31; sp = lane & (2 * C - 1); col0 = (threadIdx.x >> 5) * 16 + lane / (2 * C) * C; unit = col0 + (sp & (C - 1)); es = sp / C;
    s = (long)blockIdx.x * NS + es; el = es < NS && unit < H && s < B;
  }
};

// LSTM forward.  reference: lstm.go:276-407.  The reference's gate helpers (lstm.go:1065-1101) run over the first H of the 4H
// pre-activation rows, so only the input gate receives Wx x + Wh h; forget, cell and output gates see their biases alone and
// are constant over time.  `ig` holds the input projections Wx[0:H] x_t of every (sample, step) on entry (one contraction, issued
// before) and the input gate on exit; cell, tanh(cell) and hidden states are kept too.
template <int NS, int HB>
__global__ void __launch_bounds__(64 * HB) lstm_fwd_reg_kernel(const float* __restrict__ Wh, const float* __restrict__ bias, float* __restrict__ ig_all, float* __restrict__ c_all,
                                                               float* __restrict__ tc_all, float* __restrict__ h_all, float* __restrict__ out, const RecShape q_) {
  constexpr int KS = 4 * HB, VS = rec_vs(KS);
  __shared__ __align__(16) float hb[2][NS][8 * VS];
  const int H = q_.H, T = q_.T; const RecLane<NS, 4> L(H, q_.B); const int i = L.unit;
  float w[KS][4]; const bool vec = rec_vec(Wh, H);
#pragma unroll
  for (int k = 0; k < KS; k += 4) rec_weights<true, 4>(w + k, Wh, H, L.sp * KS + k, L.col0, vec);
  for (int e = threadIdx.x; e < 2 * NS * 8 * VS; e += blockDim.x) hb[0][0][e] = 0.f;
  float bi = 0.f, fg = 0.f, cg = 0.f, og = 0.f, c = 0.f, x = 0.f, x1 = 0.f;
  const long base = L.s * T * H + i; const int at = i / KS * VS + i % KS;
  if (L.el) {
    bi = bias[i]; fg = act_fwd(GN_ACT_SIGMOID, bias[H + i]); cg = act_fwd(GN_ACT_TANH, bias[2 * H + i]); og = act_fwd(GN_ACT_SIGMOID, bias[3 * H + i]);
    x = ig_all[base]; if (T > 1) x1 = ig_all[base + H];
  }
  __syncthreads();
  for (int t = 0; t < T; t++) {
    float acc[NS][4]; rec_clear(acc);
    rec_fma(acc, w, &hb[t & 1][0][L.sp * VS], 8 * VS);
    const float sum = rec_reduce(acc, L.lane);
    if (L.el) {
      const long o = base + (long)t * H;
      const float pre = bi + x + sum;
      x = x1; if (t + 2 < T) x1 = ig_all[o + 2 * H];               // two steps ahead: a step is about as long as a load
      const float ig = act_fwd(GN_ACT_SIGMOID, pre);
      c = fg * c + ig * cg;
      const float tc = act_fwd(GN_ACT_TANH, c), h = og * tc;
      hb[(t + 1) & 1][L.es][at] = h;
      ig_all[o] = ig; c_all[o] = c; tc_all[o] = tc; h_all[o] = h;
      if (q_.return_seq) out[o] = h; else if (t == T - 1) out[L.s * H + i] = h;
    }
    __syncthreads();
  }
}
// ... of wider layers: four threads per unit, each with a quarter of its dot product, weights in shared memory
template <int NS>
__global__ void __launch_bounds__(1024) lstm_fwd_kernel(const float* __restrict__ Wh, const float* __restrict__ bias, float* __restrict__ ig_all, float* __restrict__ c_all,
                                                        float* __restrict__ tc_all, float* __restrict__ h_all, float* __restrict__ out, const RecShape q_) {
  extern __shared__ __align__(16) float sm[];
  const int H = q_.H, T = q_.T, Hp = rec_hp(H), jq = rec_jq(H), q = threadIdx.x / Hp, i = threadIdx.x - q * Hp;
  float* hb = sm;                              // [2][NS][4 jq]
  float* part = hb + 2 * NS * 4 * jq;          // [4][NS][Hp]
  float* ws = part + 4 * NS * Hp;              // [4 jq][Hp]
  for (int e = threadIdx.x; e < 4 * jq * Hp; e += blockDim.x) { const int k = e / Hp, r = e - k * Hp; ws[e] = (r < H && k < H) ? Wh[(long)r * H + k] : 0.f; }
  for (int e = threadIdx.x; e < 2 * NS * 4 * jq; e += blockDim.x) hb[e] = 0.f;
  // the elementwise part of (sample, unit): the first NS * Hp threads
  const int es = threadIdx.x / Hp, s = blockIdx.x * NS + es; const bool el = es < NS && i < H && s < q_.B;
  float bi = 0.f, fg = 0.f, cg = 0.f, og = 0.f, c = 0.f, x = 0.f;
  const long base = ((long)s * T) * H + i;
  if (el) {
    bi = bias[i]; fg = act_fwd(GN_ACT_SIGMOID, bias[H + i]); cg = act_fwd(GN_ACT_TANH, bias[2 * H + i]); og = act_fwd(GN_ACT_SIGMOID, bias[3 * H + i]);
    x = ig_all[base];
  }
  __syncthreads();
  for (int t = 0; t < T; t++) {
    const float* hp = hb + (t & 1) * NS * 4 * jq; float* hn = hb + ((t + 1) & 1) * NS * 4 * jq;
    const float* wq = ws + (q * jq) * Hp + i;
#pragma unroll
    for (int k = 0; k < NS; k++) {
      const float* v = hp + k * 4 * jq + q * jq; float a = 0.f, b = 0.f;
#pragma unroll 4
      for (int j = 0; j < jq; j += 2) { a = fmaf(wq[j * Hp], v[j], a); b = fmaf(wq[(j + 1) * Hp], v[j + 1], b); }
      part[(q * NS + k) * Hp + i] = a + b;
    }
    __syncthreads();
    if (el) {
      const long o = base + (long)t * H;
      float pre = bi + x;
      if (t + 1 < T) x = ig_all[o + H];
#pragma unroll
      for (int k = 0; k < 4; k++) pre += part[(k * NS + es) * Hp + i];
      const float ig = act_fwd(GN_ACT_SIGMOID, pre);
      c = fg * c + ig * cg;
      const float tc = act_fwd(GN_ACT_TANH, c), h = og * tc;
      hn[es * 4 * jq + i] = h;
      ig_all[o] = ig; c_all[o] = c; tc_all[o] = tc; h_all[o] = h;
      if (q_.return_seq) out[o] = h; else if (t == T - 1) out[(long)s * H + i] = h;
    }
    __syncthreads();
  }
}

// LSTM back-propagation through time; writes the gate deltas D[s, t, 4H].  reference: lstm.go:476-698 + unroller.go:190-209: the
// hidden-state gradient handed to step t-1 is the gradient of step t PLUS Wh^T d (a running sum), because LSTM.Backward adds
// dhPrev into its argument.
// Element-wise part, for one (sample, unit)
struct LstmBwdUnit {
  float cur = 0.f, dcn = 0.f, fg = 0.f, cg = 0.f, og = 0.f, kf = 0.f, kg = 0.f, ko = 0.f, ig = 0.f, tc = 0.f, cp = 0.f;
  __device__ __forceinline__ void init(const float* bias, const float* gout, const float* ig_all, const float* c_all, const float* tc_all, const RecShape& q, long s, int i, long base) {
    const int H = q.H, T = q.T; const float bf = bias[H + i], bg = bias[2 * H + i], bo = bias[3 * H + i];
    fg = act_fwd(GN_ACT_SIGMOID, bf); cg = act_fwd(GN_ACT_TANH, bg); og = act_fwd(GN_ACT_SIGMOID, bo);
    kf = act_der(GN_ACT_SIGMOID, bf); kg = act_der(GN_ACT_TANH, bg); ko = act_der(GN_ACT_SIGMOID, bo);
    const long o = base + (long)(T - 1) * H;
    ig = ig_all[o]; tc = tc_all[o]; cp = T > 1 ? c_all[o - H] : 0.f;
    if (!q.return_seq) cur = gout[s * H + i];
  }
  __device__ __forceinline__ void step(float& di, float& df, float& dg, float& dq) {
    const float dc = cur * og * (1.f - tc * tc) + dcn;
    di = dc * cg * (ig * (1.f - ig)); df = dc * cp * kf; dg = dc * ig * kg; dq = cur * tc * ko;
    dcn = dc * fg;
  }
};
// Up to 128 units, the matrix [4 Hp, H]: two columns out of 16 per piece of 8 HB rows.  Beyond 96 units a thread's 256 weights do not fit its
// registers: the last 12 of its 32 rows lie in tensor memory, from where they come four rows at a time while rows from registers
// are multiplied (from shared memory, which the vectors keep busy already: 96 us instead of 80, 100 samples 80 instead of 57).
constexpr int LB_TM_ROWS = 12, LB_TM_COLS = 256;             // columns: 2 x 12 x 8 (two warps share a quarter of the lanes), a power of two
__device__ __forceinline__ void rec_tm_load(float (&w)[4][8], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=f"(w[0][0]), "=f"(w[0][1]), "=f"(w[0][2]), "=f"(w[0][3]), "=f"(w[0][4]), "=f"(w[0][5]), "=f"(w[0][6]), "=f"(w[0][7]),
        "=f"(w[1][0]), "=f"(w[1][1]), "=f"(w[1][2]), "=f"(w[1][3]), "=f"(w[1][4]), "=f"(w[1][5]), "=f"(w[1][6]), "=f"(w[1][7]),
        "=f"(w[2][0]), "=f"(w[2][1]), "=f"(w[2][2]), "=f"(w[2][3]), "=f"(w[2][4]), "=f"(w[2][5]), "=f"(w[2][6]), "=f"(w[2][7]),
        "=f"(w[3][0]), "=f"(w[3][1]), "=f"(w[3][2]), "=f"(w[3][3]), "=f"(w[3][4]), "=f"(w[3][5]), "=f"(w[3][6]), "=f"(w[3][7])
      : "r"(addr) : "memory");
}
// (the registers are operands: nothing that uses them moves ahead of the wait)
__device__ __forceinline__ void rec_tm_wait(float (&w)[4][8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+f"(w[0][0]), "+f"(w[0][1]), "+f"(w[0][2]), "+f"(w[0][3]), "+f"(w[0][4]), "+f"(w[0][5]), "+f"(w[0][6]), "+f"(w[0][7]),
        "+f"(w[1][0]), "+f"(w[1][1]), "+f"(w[1][2]), "+f"(w[1][3]), "+f"(w[1][4]), "+f"(w[1][5]), "+f"(w[1][6]), "+f"(w[1][7]),
        "+f"(w[2][0]), "+f"(w[2][1]), "+f"(w[2][2]), "+f"(w[2][3]), "+f"(w[2][4]), "+f"(w[2][5]), "+f"(w[2][6]), "+f"(w[2][7]),
        "+f"(w[3][0]), "+f"(w[3][1]), "+f"(w[3][2]), "+f"(w[3][3]), "+f"(w[3][4]), "+f"(w[3][5]), "+f"(w[3][6]), "+f"(w[3][7])
      :: "memory");
}
__device__ __forceinline__ void rec_tm_store(const float (&w)[4][8], uint32_t addr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
      :: "f"(w[0][0]), "f"(w[0][1]), "f"(w[0][2]), "f"(w[0][3]), "f"(w[0][4]), "f"(w[0][5]), "f"(w[0][6]), "f"(w[0][7]),
         "f"(w[1][0]), "f"(w[1][1]), "f"(w[1][2]), "f"(w[1][3]), "f"(w[1][4]), "f"(w[1][5]), "f"(w[1][6]), "f"(w[1][7]),
         "f"(w[2][0]), "f"(w[2][1]), "f"(w[2][2]), "f"(w[2][3]), "f"(w[2][4]), "f"(w[2][5]), "f"(w[2][6]), "f"(w[2][7]),
         "f"(w[3][0]), "f"(w[3][1]), "f"(w[3][2]), "f"(w[3][3]), "f"(w[3][4]), "f"(w[3][5]), "f"(w[3][6]), "f"(w[3][7]), "r"(addr) : "memory");
}
template <int NS, int HB>
__global__ void __launch_bounds__(64 * HB) lstm_bwd_reg_kernel(const float* __restrict__ gout, const float* __restrict__ Wh, const float* __restrict__ bias, const float* __restrict__ ig_all,
                                                               const float* __restrict__ c_all, const float* __restrict__ tc_all, float* __restrict__ D, const RecShape q_) {
  constexpr int C = 8, KS = 8 * HB, VS = rec_vs(KS), TR = HB == 4 ? LB_TM_ROWS : 0, RR = KS - TR, HALF = RR / 8 * 4;
  __shared__ __align__(16) float db[2][NS][2 * C * VS];
  __shared__ uint32_t tm_slot;
  const int H = q_.H, T = q_.T, warp = threadIdx.x >> 5; const RecLane<NS, C> L(H, q_.B); const int i = L.unit;
  if (TR > 0 && warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&tm_slot)), "r"(LB_TM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const float* wg = Wh + (long)(L.sp >> 2) * H * H; const int k0 = (L.sp & 3) * KS; const bool vec = rec_vec(wg, H);      // (four pieces per gate)
  float w1[HALF][C], w2[RR - HALF][C], wt[4][C];
#pragma unroll
  for (int k = 0; k < HALF; k += 4) rec_weights<false, C>(w1 + k, wg, H, k0 + k, L.col0, vec);
#pragma unroll
  for (int k = HALF; k < RR; k += 4) rec_weights<false, C>(w2 + (k - HALF), wg, H, k0 + k, L.col0, vec);
  for (int e = threadIdx.x; e < 2 * NS * 2 * C * VS; e += 64 * HB) db[0][0][e] = 0.f;
  LstmBwdUnit u; const long base = L.s * T * H + i;
  if (L.el) u.init(bias, gout, ig_all, c_all, tc_all, q_, L.s, i, base);
  float n_ig = 0.f, n_tc = 0.f, n_cp = 0.f;                  // the next step's: loaded two steps ahead, a load takes about as long as a short step
  auto ahead = [&](int t) { const long o = base + (long)t * H; n_ig = ig_all[o]; n_tc = tc_all[o]; n_cp = t > 0 ? c_all[o - H] : 0.f; };
  if (L.el && T > 1) ahead(T - 2);
  if (TR > 0) tc_fence_before();
  __syncthreads();
  if (TR > 0) tc_fence_after();
  const uint32_t tm = TR > 0 ? tm_slot + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * TR * C : 0;
  if constexpr (TR > 0) {
#pragma unroll
    for (int k = 0; k < TR; k += 4) { rec_weights<false, C>(wt, wg, H, k0 + RR + k, L.col0, vec); rec_tm_store(wt, tm + k * C); }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  auto unit_step = [&](int t) {
    if (!L.el) return;
    if (q_.return_seq) u.cur += gout[base + (long)t * H];
    float di, df, dg, dq; u.step(di, df, dg, dq);
    float* e = db[t & 1][L.es] + i / KS * VS + i % KS; e[0] = di; e[4 * VS] = df; e[8 * VS] = dg; e[12 * VS] = dq;
    float* Dr = D + (L.s * T + t) * 4 * H + i; Dr[0] = di; Dr[H] = df; Dr[2 * H] = dg; Dr[3 * H] = dq;
    u.ig = n_ig; u.tc = n_tc; u.cp = n_cp;
    if (t > 1) ahead(t - 2);
  };
  for (int t = T - 1; t > 0; t--) {
    if constexpr (TR > 0) rec_tm_load(wt, tm);               // (loads never reach across iterations: their registers are not to be moved before the wait)
    unit_step(t);
    __syncthreads();
    float acc[NS][C]; rec_clear(acc);
    const float* v = db[t & 1][0] + L.sp * VS; constexpr int vs = 2 * C * VS;
    if constexpr (TR > 0) {
      rec_tm_wait(wt); rec_fma(acc, wt, v + RR, vs); rec_tm_load(wt, tm + 4 * C);
      rec_fma(acc, w1, v, vs);
      rec_tm_wait(wt); rec_fma(acc, wt, v + RR + 4, vs); rec_tm_load(wt, tm + 8 * C);
      rec_fma(acc, w2, v + HALF, vs);
      rec_tm_wait(wt); rec_fma(acc, wt, v + RR + 8, vs);
    } else { rec_fma(acc, w1, v, vs); rec_fma(acc, w2, v + HALF, vs); }
    const float sum = rec_reduce(acc, L.lane);
    if (L.el) u.cur += sum;
  }
  unit_step(0);
  if constexpr (TR > 0) {
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_slot), "r"(LB_TM_COLS) : "memory");
  }
}
// ... of wider layers.  Thread (gate q, unit i) sums over gate q's H rows of column i: the first `rs` rows (a multiple of four) from
// shared memory, the next RR from registers, the rest from global memory.
template <int NS, int RR>
__global__ void __launch_bounds__(1024) lstm_bwd_kernel(const float* __restrict__ gout, const float* __restrict__ Wh, const float* __restrict__ bias, const float* __restrict__ ig_all,
                                                        const float* __restrict__ c_all, const float* __restrict__ tc_all, float* __restrict__ D, const RecShape q_, int rs) {
  extern __shared__ __align__(16) float sm[];
  const int H = q_.H, T = q_.T, Hp = rec_hp(H), q = threadIdx.x / Hp, i = threadIdx.x - q * Hp;
  float* db = sm;                              // [NS][4][Hp]
  float* part = db + NS * 4 * Hp;              // [4][NS][Hp]
  float* ws = part + 4 * NS * Hp;              // [rs][4][Hp]
  for (int e = threadIdx.x; e < rs * 4 * Hp; e += blockDim.x) { const int r = e / (4 * Hp), gq = (e / Hp) & 3, c = e % Hp; ws[e] = c < H ? Wh[((long)gq * H + r) * H + c] : 0.f; }
  float w[RR];
#pragma unroll
  for (int j = 0; j < RR; j++) w[j] = (i < H && rs + j < H) ? Wh[((long)q * H + rs + j) * H + i] : 0.f;
  for (int e = threadIdx.x; e < NS * 4 * Hp; e += blockDim.x) db[e] = 0.f;
  const int es = threadIdx.x / Hp, s = blockIdx.x * NS + es; const bool el = es < NS && i < H && s < q_.B;
  LstmBwdUnit u; const long base = ((long)s * T) * H + i;
  if (el) u.init(bias, gout, ig_all, c_all, tc_all, q_, s, i, base);
  __syncthreads();
  for (int t = T - 1; t >= 0; t--) {
    if (el) {
      const long o = base + (long)t * H;
      if (q_.return_seq) u.cur += gout[o];
      float di, df, dg, dq; u.step(di, df, dg, dq);
      float* d = db + es * 4 * Hp + i; d[0] = di; d[Hp] = df; d[2 * Hp] = dg; d[3 * Hp] = dq;
      float* Dr = D + ((long)s * T + t) * 4 * H + i; Dr[0] = di; Dr[H] = df; Dr[2 * H] = dg; Dr[3 * H] = dq;
      if (t > 0) { u.ig = ig_all[o - H]; u.tc = tc_all[o - H]; u.cp = t > 1 ? c_all[o - 2 * H] : 0.f; }
    }
    if (t == 0) break;
    __syncthreads();
    float acc[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) acc[k] = 0.f;
    const float* d0 = db + q * Hp; const float* wq = ws + q * Hp + i;
#pragma unroll 4
    for (int r = 0; r < rs; r += 4) {
      const float w0 = wq[r * 4 * Hp], w1 = wq[(r + 1) * 4 * Hp], w2 = wq[(r + 2) * 4 * Hp], w3 = wq[(r + 3) * 4 * Hp];
#pragma unroll
      for (int k = 0; k < NS; k++) { const float4 x = *reinterpret_cast<const float4*>(d0 + k * 4 * Hp + r); acc[k] = fmaf(w0, x.x, fmaf(w1, x.y, fmaf(w2, x.z, fmaf(w3, x.w, acc[k])))); }
    }
#pragma unroll
    for (int j = 0; j < RR; j += 4) {
      if (rs + j < Hp) {                       // (rows H .. Hp - 1 of d are zero; Hp and rs are multiples of four)
#pragma unroll
        for (int k = 0; k < NS; k++) {
          const float4 x = *reinterpret_cast<const float4*>(d0 + k * 4 * Hp + rs + j);
          acc[k] = fmaf(w[j], x.x, fmaf(w[j + 1], x.y, fmaf(w[j + 2], x.z, fmaf(w[j + 3], x.w, acc[k]))));
        }
      }
    }
    if (i < H) for (int r = rs + RR; r < H; r++) {
      const float wv = __ldg(Wh + ((long)q * H + r) * H + i);
#pragma unroll
      for (int k = 0; k < NS; k++) acc[k] = fmaf(wv, d0[k * 4 * Hp + r], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < NS; k++) part[(q * NS + k) * Hp + i] = acc[k];
    __syncthreads();
    if (el) u.cur += (part[es * Hp + i] + part[(NS + es) * Hp + i]) + (part[(2 * NS + es) * Hp + i] + part[(3 * NS + es) * Hp + i]);
  }
}

// GRU forward for up to 128 units.  reference: gru.go:192-288.  `gates` [B, T, 3H] holds b + Wx x_t of every step on entry (one
// contraction over all rows, issued before) and the gate values z | r | candidate on exit.  The layer has 2H recurrent rows: the
// candidate's recurrent product uses the reset gate's rows on r (.) h_prev (gru.go:247-258).
template <int NS, int HB>
__global__ void __launch_bounds__(64 * HB) gru_fwd_reg_kernel(const float* __restrict__ Wh, float* __restrict__ gates, float* __restrict__ h_all, float* __restrict__ out, const RecShape q_) {
  constexpr int KS = 4 * HB, VS = rec_vs(KS);
  __shared__ __align__(16) float hb[NS][8 * VS], rb[NS][8 * VS];      // h_prev, r (.) h_prev
  const int H = q_.H, T = q_.T; const RecLane<NS, 4> L(H, q_.B); const int i = L.unit;
  float wz[KS][4], wr[KS][4]; const bool vec = rec_vec(Wh, H);
#pragma unroll
  for (int k = 0; k < KS; k += 4) {
    rec_weights<true, 4>(wz + k, Wh, H, L.sp * KS + k, L.col0, vec);
    rec_weights<true, 4>(wr + k, Wh + (long)H * H, H, L.sp * KS + k, L.col0, vec);
  }
  for (int e = threadIdx.x; e < NS * 8 * VS; e += blockDim.x) { hb[0][e] = 0.f; rb[0][e] = 0.f; }
  float* gp = gates + L.s * T * 3 * H + i; const int at = i / KS * VS + i % KS;
  float h = 0.f, az = 0.f, ar = 0.f, ac = 0.f, nz = 0.f, nr = 0.f, nc = 0.f;      // this step's and the next one's
  if (L.el) { az = gp[0]; ar = gp[H]; ac = gp[2 * H]; if (T > 1) { const float* g = gp + 3 * H; nz = g[0]; nr = g[H]; nc = g[2 * H]; } }
  __syncthreads();
  for (int t = 0; t < T; t++) {
    float a[NS][4], b[NS][4]; rec_clear(a); rec_clear(b);
    rec_fma(a, wr, &hb[0][L.sp * VS], 8 * VS);
    const float sr = rec_reduce(a, L.lane); float r = 0.f;
    if (L.el) { r = act_fwd(GN_ACT_SIGMOID, ar + sr); rb[L.es][at] = r * h; }
    rec_fma(b, wz, &hb[0][L.sp * VS], 8 * VS);
    const float sz = rec_reduce(b, L.lane);
    __syncthreads();
    rec_clear(a);
    rec_fma(a, wr, &rb[0][L.sp * VS], 8 * VS);
    const float sc = rec_reduce(a, L.lane);
    if (L.el) {
      const float z = act_fwd(GN_ACT_SIGMOID, az + sz), c = act_fwd(GN_ACT_TANH, ac + sc);
      h = h + z * (c - h);
      hb[L.es][at] = h;
      float* g = gp + (long)t * 3 * H; g[0] = z; g[H] = r; g[2 * H] = c;
      const long o = (L.s * T + t) * H + i;
      h_all[o] = h;
      if (q_.return_seq) out[o] = h; else if (t == T - 1) out[L.s * H + i] = h;
      az = nz; ar = nr; ac = nc;
      if (t + 2 < T) { g += 6 * H; nz = g[0]; nr = g[H]; nc = g[2 * H]; }
    }
    __syncthreads();
  }
}
// GRU back-propagation through time for up to 128 units.  reference: gru.go:360-534 with unroller.go:190-209, literal: the reset
// gate's delta is never formed (stays zero), the candidate's gradient is scaled by (1 - z) and the hidden-state pass-through by
// z, the candidate's contribution to dh_prev is indexed by the output unit's reset gate, and dh_prev is ADDED to the incoming
// gradient before it is handed to the previous step.  Writes the gate deltas D [B,T,3H] (update | zero | candidate), h_{t-1} [B,T,H]
// and r (.) h_{t-1} [B,T,H] for the weight-gradient contractions.
template <int NS, int HB>
__global__ void __launch_bounds__(64 * HB) gru_bwd_reg_kernel(const float* __restrict__ gout, const float* __restrict__ Wh, const float* __restrict__ gates, const float* __restrict__ h_all,
                                                              float* __restrict__ D, float* __restrict__ hprev_all, float* __restrict__ rh_all, const RecShape q_) {
  constexpr int KS = 4 * HB, VS = rec_vs(KS);
  __shared__ __align__(16) float vb[2][2][NS][8 * VS];      // by parity of the step: update deltas | candidate deltas times r
  const int H = q_.H, T = q_.T; const RecLane<NS, 4> L(H, q_.B); const int i = L.unit;
  float wz[KS][4], wr[KS][4]; const bool vec = rec_vec(Wh, H);
#pragma unroll
  for (int k = 0; k < KS; k += 4) {
    rec_weights<false, 4>(wz + k, Wh, H, L.sp * KS + k, L.col0, vec);
    rec_weights<false, 4>(wr + k, Wh + (long)H * H, H, L.sp * KS + k, L.col0, vec);
  }
  for (int e = threadIdx.x; e < 4 * NS * 8 * VS; e += blockDim.x) vb[0][0][0][e] = 0.f;
  const float* gp = gates + L.s * T * 3 * H + i; const long base = L.s * T * H + i; const int at = i / KS * VS + i % KS;
  float cur = 0.f, z = 0.f, r = 0.f, c = 0.f, hp = 0.f;
  if (L.el) {
    const float* g = gp + (long)(T - 1) * 3 * H; z = g[0]; r = g[H]; c = g[2 * H]; hp = T > 1 ? h_all[base + (long)(T - 2) * H] : 0.f;
    if (!q_.return_seq) cur = gout[L.s * H + i];
  }
  __syncthreads();
  for (int t = T - 1; t >= 0; t--) {
    const float zt = z;
    if (L.el) {
      const long o = base + (long)t * H;
      if (q_.return_seq) cur += gout[o];
      const float du = cur * (c - hp) * z * (1.f - z), dc = cur * (1.f - z) * (1.f - c * c);
      float* Dr = D + (L.s * T + t) * 3 * H + i; Dr[0] = du; Dr[H] = 0.f; Dr[2 * H] = dc;
      hprev_all[o] = hp; rh_all[o] = r * hp;
      vb[t & 1][0][L.es][at] = du; vb[t & 1][1][L.es][at] = dc * r;
      if (t > 0) { const float* g = gp + (long)(t - 1) * 3 * H; z = g[0]; r = g[H]; c = g[2 * H]; hp = t > 1 ? h_all[o - 2 * H] : 0.f; }
    }
    if (t == 0) break;
    __syncthreads();
    float acc[NS][4]; rec_clear(acc);
    rec_fma(acc, wz, &vb[t & 1][0][0][L.sp * VS], 8 * VS);
    rec_fma(acc, wr, &vb[t & 1][1][0][L.sp * VS], 8 * VS);
    const float sum = rec_reduce(acc, L.lane);
    if (L.el) cur = cur + (sum + cur * zt);
  }
}

// ------------------------------------------------------------------ launchers
// f<NS, HB>() for the number of samples per block and of blocks of 32 units
template <class F> inline int rec_dispatch(const Ctx* ctx, const RecShape& q, F&& f) {
  const bool two = q.B > ctx->sm_count;
  auto by_hb = [&](auto ns) -> int {
    switch ((q.H + 31) / 32) {
      case 1: return f(ns, std::integral_constant<int, 1>{});
      case 2: return f(ns, std::integral_constant<int, 2>{});
      case 3: return f(ns, std::integral_constant<int, 3>{});
      default: return f(ns, std::integral_constant<int, 4>{});
    }
  };
  return two ? by_hb(std::integral_constant<int, 2>{}) : by_hb(std::integral_constant<int, 1>{});
}
inline int lstm_fwd(Ctx* ctx, const float* Wh, const float* bias, float* ig, float* c, float* tc, float* h, float* out, const RecShape& q) {
  if (q.H <= REC_REG_H) return rec_dispatch(ctx, q, [&](auto ns, auto hb) -> int {
    GN_LAUNCH(ctx, (lstm_fwd_reg_kernel<ns(), hb()>), cdiv(q.B, ns()), 64 * hb(), 0, Wh, bias, ig, c, tc, h, out, q);
    return check_launch("lstm_fwd");
  });
  const int Hp = rec_hp(q.H), jq = rec_jq(q.H), ns = q.B > ctx->sm_count ? 2 : 1;
  const size_t smem = ((size_t)2 * ns * 4 * jq + 4 * ns * Hp + (size_t)4 * jq * Hp) * sizeof(float);
  auto* K = ns == 2 ? lstm_fwd_kernel<2> : lstm_fwd_kernel<1>;
  if (4 * Hp > 1024 || smem > 220 * 1024) return fail(GN_ERR_UNSUPPORTED, "LSTM of hidden size %d needs %zu bytes of shared memory", q.H, smem);
  GN_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, K, cdiv(q.B, ns), 4 * Hp, smem, Wh, bias, ig, c, tc, h, out, q);
  return check_launch("lstm_fwd");
}
inline int lstm_bwd(Ctx* ctx, const float* gout, const float* Wh, const float* bias, const float* ig, const float* c, const float* tc, float* D, const RecShape& q) {
  if (q.H <= REC_REG_H) return rec_dispatch(ctx, q, [&](auto ns, auto hb) -> int {
    GN_LAUNCH(ctx, (lstm_bwd_reg_kernel<ns(), hb()>), cdiv(q.B, ns()), 64 * hb(), 0, gout, Wh, bias, ig, c, tc, D, q);
    return check_launch("lstm_bwd");
  });
  const int Hp = rec_hp(q.H), ns = q.B > ctx->sm_count ? 2 : 1;
  const size_t fixed = (size_t)8 * ns * Hp * sizeof(float), row = (size_t)4 * Hp * sizeof(float);
  // registers hold 24 rows of each gate's column, shared memory as many of the others as fit, in fours
  const int rs = (int)std::min<size_t>((q.H - 24 + 3) & ~3, ((200 * 1024 - fixed) / row) & ~(size_t)3); const size_t smem = fixed + rs * row;
  auto* K = ns == 2 ? lstm_bwd_kernel<2, 24> : lstm_bwd_kernel<1, 24>;
  GN_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GN_LAUNCH(ctx, K, cdiv(q.B, ns), 4 * Hp, smem, gout, Wh, bias, ig, c, tc, D, q, rs);
  return check_launch("lstm_bwd");
}
inline bool gru_reg_ok(int H) { return H <= REC_REG_H; }
inline int gru_fwd_reg(Ctx* ctx, const float* Wh, float* gates, float* h, float* out, const RecShape& q) {
  return rec_dispatch(ctx, q, [&](auto ns, auto hb) -> int {
    GN_LAUNCH(ctx, (gru_fwd_reg_kernel<ns(), hb()>), cdiv(q.B, ns()), 64 * hb(), 0, Wh, gates, h, out, q);
    return check_launch("gru_fwd");
  });
}
inline int gru_bwd_reg(Ctx* ctx, const float* gout, const float* Wh, const float* gates, const float* h, float* D, float* hprev, float* rh, const RecShape& q) {
  return rec_dispatch(ctx, q, [&](auto ns, auto hb) -> int {
    GN_LAUNCH(ctx, (gru_bwd_reg_kernel<ns(), hb()>), cdiv(q.B, ns()), 64 * hb(), 0, gout, Wh, gates, h, D, hprev, rh, q);
    return check_launch("gru_bwd");
  });
}

// ------------------------------------------------------------------ LSTM gradient clipping
// The reference clips the WHOLE accumulated LSTM gradient to L2 norm <= 1 after every time-step of every sample (lstm.go:694,
// :725-751): g <- clip(g + u_k) over the rank-one updates u_k = d_k z_k^T of a worker chunk, z_k = [x_last ; h_{t-1} ; 1], samples
// ascending, time descending.  The clipping needs only the norm, |g + u_k|^2 = |g|^2 + 2 <g, u_k> + |u_k|^2, so the walk is over
// scalars; it goes in groups of CG updates.  Within a group the inner products come from the group's own Gram block, <u_q, u_r>
// = <d_q, d_r> <z_q, z_r>; across groups <g, u_r> = d_r^T g z_r comes from the gradient matrix itself, formed one group ahead, and
// the Gram block against the group before.  One launch per group (all inputs come from earlier launches: nothing waits inside
// one; g_j is the gradient before group j):
//   block 0     walks group j: v = s_{j-1} p_j + X_j om_{j-1}, then CG dependent steps; leaves om_j[r], the weight of u_r in the
//               gradient after the group, and s_j, the weight of what was there before
//   the others  eight rows of the matrix each: g_j = s_{j-1} g_{j-1} + sum_r om_{j-1}[r] d_r z_r^T, and that slab's part of
//               p_{j+1}[r] = d_r^T g_j z_r for the updates of group j+1
// (The full Gram matrix of all updates, 16384^2 for 256 samples of 64 steps, took two products of 137 GFLOP, 1 GB, and a pass over
// all earlier updates per group: 7.1 ms.  This takes 1.3.)
// Norms, factors and the sums over updates are kept in double.
//
// Where the walk starts.  |g| <= 1, so an update with |u| > 2 is always clipped, by a factor of at most 1 / (|u| - 1); and clipping
// to a ball never moves two gradients further apart (two that lie outside by r or more end up closer by the factor r).  So
// whatever the gradient was before update k reaches the end of the chunk scaled by at most the product of 1 / (|u_i| - 1) over the
// later updates with |u_i| > 2.  Groups for which that is below 2^-CLIP_FORGET, far under the last bit of a double, are not walked: the
// walk starts from zero at the first group that can be seen in the result (lstm_clip_start_kernel), at group 0 if there is none,
// or if any update is not finite.  Gradients that are carried back through many steps grow by orders of magnitude per sequence
// (median |u| 2e5 for 64 steps of 128 units), and a few dozen updates decide the result.  What is not walked is not gathered and
// has no Gram blocks either: that step of 256 samples, on a batch in device memory, went from 1682 us to 496 (289 since, with the recurrences above and lstm_clip_start_kernel's
// condition).  Where nothing can be left out it took 1685 (now 1618): the norms and the search take 8 us, and the rows of zeros come without launches of their own.
constexpr int CG = 128, CG_THREADS = 512, CG_PAD = CG, CG_TILE = 160;        // CG_PAD: rows of zeros before a chunk: group -1
constexpr int CG_GD = CG + 1;
constexpr long CG_MAX_K = 1L << 20;                         // updates per worker chunk
__host__ __device__ __forceinline__ int clip_zs(int ZW) { return (ZW + 3) & ~3; }                 // row stride of Zm
__host__ __device__ __forceinline__ int clip_tile(int ZW) { const int n = (ZW + CG_TILE - 1) / CG_TILE; return (ZW + n - 1) / n; }
inline size_t clip_smem(int ZW) {
  const int wp = clip_tile(ZW) | 1; const size_t slab = ((size_t)2 * CG * wp + CG * 8 + (size_t)wp * 8 + 8) * sizeof(float), walk = (size_t)CG * CG_GD * sizeof(double);
  return slab > walk ? slab : walk;
}
// Rows of Dm [., 4H] and Zm [., zs] as `u` lays them out, a warp each; this rank's updates are the first ones.
// (Zeroing those rows separately took two to four more launches per chunk.)  `un` (may be null): receives |u_k|^2 = |d_k|^2 |z_k|^2.  With a block per row
// the rows that are left out, nearly all of 16 384, cost 12 us.
__global__ void __launch_bounds__(256) lstm_gather_updates_kernel(const float* __restrict__ D, const float* __restrict__ x, const float* __restrict__ h_all, float* __restrict__ Dm, float* __restrict__ Zm,
                                           int T, int in, int H, int zs, const UpdateRows u, const int* __restrict__ start, float* __restrict__ un) {
  const int R4 = 4 * H, ZW = in + H + 1, lane = threadIdx.x & 31;
  const long row = blockIdx.x * 8L + (threadIdx.x >> 5); if (row >= u.rows) return;
  const UpdateRows::At at = u.at(row); const long k = at.k;
  if (start && at.r < (long)(start[at.chunk] - 1) * CG) return;               // before the first walked group and the one it is multiplied with
  if (!at.update) {
    for (int e = lane; e < R4 + zs; e += 32) { if (e < R4) Dm[row * R4 + e] = 0.f; else Zm[row * zs + e - R4] = 0.f; }
    return;
  }
  const int s = (int)(k / T), t = T - 1 - (int)(k % T); float d2 = 0.f, z2 = 0.f;
#pragma unroll 4
  for (int e = lane; e < R4; e += 32) { const float v = D[((long)s * T + t) * R4 + e]; Dm[row * R4 + e] = v; d2 = fmaf(v, v, d2); }
#pragma unroll 4
  for (int c = lane; c < zs; c += 32) {
    float v;
    if (c < in) v = x[(long)s * T * in + (long)(T - 1) * in + c];                 // input of the LAST forward call (lstm.go:592-621)
    else if (c < in + H) v = t > 0 ? h_all[((long)s * T + (t - 1)) * H + (c - in)] : 0.f;
    else v = c < ZW ? 1.f : 0.f;
    Zm[row * zs + c] = v; z2 = fmaf(v, v, z2);
  }
  if (!un) return;
  d2 = warp_sum(d2); z2 = warp_sum(z2);
  if (lane == 0) un[k] = d2 * z2;
}
// rows of `w` floats from contiguous order into the chunks' layout (after a gather over the ranks)
__global__ void lstm_place_rows_kernel(const float* __restrict__ src, float* __restrict__ dst, int w, const UpdateRows u) {
  const long k = blockIdx.x, row = u.row_of(k);
  for (int e = threadIdx.x; e < w; e += blockDim.x) dst[row * w + e] = src[k * w + e];
}
__global__ void lstm_gram_mul_kernel(float* __restrict__ G, const float* __restrict__ G2, long total4, int groups, const int* __restrict__ start) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total4; i += (long)gridDim.x * blockDim.x) {
    const int j = (int)(i / (CG * CG / 2)); if (start && j % groups < start[j / groups]) continue;
    float4 a = reinterpret_cast<float4*>(G)[i]; const float4 b = reinterpret_cast<const float4*>(G2)[i];
    a.x *= b.x; a.y *= b.y; a.z *= b.z; a.w *= b.w; reinterpret_cast<float4*>(G)[i] = a;
  }
}
constexpr int CLIP_FORGET = 128, CLIP_FEW = 32, CLIP_TAIL = 16, CLIP_SKIP_MIN = 64;      // (last groups whose launches are never left out; groups from which on the others may be)
constexpr float CLIP_FINITE = 1e36f;                        // squared norms above this count as not finite
// |u_k|^2 of every update, in update order; a warp each.  From the layer's own arrays (d, x, h as in lstm_gather_updates_kernel), so that
// updates that are not walked need not be gathered.
__global__ void __launch_bounds__(256) lstm_update_norms_kernel(const float* __restrict__ D, const float* __restrict__ x, const float* __restrict__ h_all, float* __restrict__ un, int T, int in, int H, long n_updates) {
  const long k = blockIdx.x * 8L + (threadIdx.x >> 5); const int lane = threadIdx.x & 31; if (k >= n_updates) return;
  const long s = k / T; const int t = T - 1 - (int)(k % T); float d2 = 0.f, z2 = 0.f;
  const float* d = D + (s * T + t) * 4 * H; const float* xl = x + s * T * in + (long)(T - 1) * in; const float* h = h_all + (s * T + max(t - 1, 0)) * H;
#pragma unroll 4
  for (int e = lane; e < 4 * H; e += 32) d2 = fmaf(d[e], d[e], d2);
  for (int e = lane; e < in; e += 32) z2 = fmaf(xl[e], xl[e], z2);
  if (t > 0) for (int e = lane; e < H; e += 32) z2 = fmaf(h[e], h[e], z2);
  d2 = warp_sum(d2); z2 = warp_sum(z2) + 1.f;
  if (lane == 0) un[k] = d2 * z2;
}
// ... from gathered rows
__global__ void __launch_bounds__(256) lstm_row_norms_kernel(const float* __restrict__ Dm, const float* __restrict__ Zm, float* __restrict__ un, int R4, int zs, const UpdateRows u) {
  const long k = blockIdx.x * 8L + (threadIdx.x >> 5); const int lane = threadIdx.x & 31; if (k >= u.n) return;
  const long row = u.row_of(k); float d2 = 0.f, z2 = 0.f;
#pragma unroll 4
  for (int e = lane; e < R4; e += 32) d2 = fmaf(Dm[row * R4 + e], Dm[row * R4 + e], d2);
  for (int e = lane; e < zs; e += 32) z2 = fmaf(Zm[row * zs + e], Zm[row * zs + e], z2);
  d2 = warp_sum(d2); z2 = warp_sum(z2);
  if (lane == 0) un[k] = d2 * z2;
}
// start[chunk]: the first group to walk.  `skip` (0: none): condition of the launches for groups before `tail` in a recorded step, which
// are left out as a whole if no chunk starts there.  A launch of the walk that has nothing to do still costs 0.9 us, a condition about 10, and 20
// if its body runs: 128 groups of which the last few are walked 414 -> 289 us (a step of 64 steps, 256 samples), all walked 1604 -> 1618; 32 groups 227
// either way, all walked 520 -> 542: from 64 groups on.
__global__ void __launch_bounds__(1024) lstm_clip_start_kernel(const float* __restrict__ un, long n_updates, long Kc, int* __restrict__ start, cudaGraphConditionalHandle skip, int tail) {
  __shared__ float part[32]; __shared__ int first;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5; const long k0 = blockIdx.x * Kc, n = min(Kc, n_updates - k0); const float* u = un + k0;
  const int groups = (int)((Kc + CG - 1) / CG);
  int fine = 1;
#pragma unroll 8
  for (long k = tid; k < n; k += 1024) fine &= u[k] <= CLIP_FINITE;
  fine = __syncthreads_and(fine);
  // a warp per group, 32 groups at a time from the end: log2 of the factor by which a group's updates shrink what was before it
  float sum = 0.f; int j0 = 0;
  for (int hi = groups; fine && hi > 0; hi -= 32) {
    const int j = hi - 1 - warp; float l = 0.f;
    if (j >= 0) for (int r = lane; r < CG; r += 32) { const long k = (long)j * CG + r; const float q = k < n ? sqrtf(u[k]) : 0.f; if (q > 2.01f) l += log2f(q - 1.f); }      // (0.01: the norms are rounded)
    l = warp_sum(l);
    if (lane == 0) part[warp] = l;
    __syncthreads();
    if (tid == 0) {
      first = -1;
      for (int w = 0; w < 32 && hi - 1 - w >= 0; w++) { sum += part[w]; if (sum >= (float)CLIP_FORGET) { first = hi - 1 - w; break; } }
    }
    __syncthreads();
    if (first >= 0) { j0 = first; break; }
    __syncthreads();
  }
  if (tid == 0) { start[blockIdx.x] = j0; if (skip && j0 < tail) cudaGraphSetConditional(skip, 1); }
}
struct ClipArgs {
  const float *D, *Z, *G;        // rows of a chunk start at chunk * stride (CG_PAD rows of zeros first); G [chunk][group][CG][2 CG]: against groups j-1, j
  double *om, *p, *st;           // [chunk][groups][CG] weights of a group's updates; [chunk][2][CG][slabs] parts of p by parity of the group; [chunk][groups][2]: s_j, |g|^2
  float* g;                      // [chunk][2][4H][ZW]
  const int* start;              // [chunk] first group to walk; null: group 0
  int R4, ZW, groups, slabs; long stride;
};
__global__ void __launch_bounds__(CG_THREADS) lstm_clip_kernel(const ClipArgs a, int j) {
  extern __shared__ __align__(16) float sm[];
  const int chunk = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, R4 = a.R4, ZW = a.ZW, zs = clip_zs(ZW);
  double* om = a.om + (long)chunk * a.groups * CG; double* st = a.st + (long)chunk * a.groups * 2; double* pp = a.p + (long)chunk * 2 * CG * a.slabs;
  // Z and the Gram blocks are written before the loop over the groups: launch 0 waits for them, and the next launch is only let
  // in (pdl_launch) behind a wait, so every later launch can fetch them before it waits for its predecessor.
  // The same goes for the first group to walk.  A launch before it has nothing to do and nothing to wait for: the next one is let
  // in when its blocks are gone.
  if (j == 0) pdl_wait();
  const int j0 = a.start ? a.start[chunk] : 0;
  if (j < j0) return;
  if (blockIdx.x == 0) {
    if (j >= a.groups) { pdl_wait(); return; }
    double* Gd = reinterpret_cast<double*>(sm);                   // [CG][CG_GD]
    __shared__ double vs[CG], fs[CG], cs[2][33];
    const float* Gj = a.G + ((long)chunk * a.groups + j) * CG * 2 * CG;
    const double* pj = pp + (long)(j & 1) * CG * a.slabs;
    double x[CG / 16][4];                                         // the Gram blocks come from before the loop over the groups
#pragma unroll
    for (int k = 0; k < CG / 16; k++) {
      const int r = warp + 16 * k; const float* gr = Gj + (long)r * 2 * CG + lane; double* gd = Gd + r * CG_GD + lane;
#pragma unroll
      for (int q = 0; q < 4; q++) { x[k][q] = gr[32 * q]; gd[32 * q] = gr[CG + 32 * q]; }
    }
    pdl_wait(); pdl_launch();
    const double s1 = j > j0 ? st[2 * (j - 1)] : 0.0;            // s_{j-1}
    {   // v_r: a warp per eight rows, a row's terms over the lanes
      double v[CG / 16];
#pragma unroll
      for (int k = 0; k < CG / 16; k++) v[k] = 0.0;
      if (j > j0) {
        const double* o = om + (long)(j - 1) * CG + lane; double ov[4], ps[CG / 16][4];
#pragma unroll
        for (int q = 0; q < 4; q++) ov[q] = o[32 * q];
#pragma unroll
        for (int k = 0; k < CG / 16; k++) {
#pragma unroll
          for (int q = 0; q < 4; q++) ps[k][q] = lane + 32 * q < a.slabs ? pj[(long)(warp + 16 * k) * a.slabs + lane + 32 * q] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < CG / 16; k++)
          v[k] = fma(s1, (ps[k][0] + ps[k][1]) + (ps[k][2] + ps[k][3]), fma(ov[0], x[k][0], ov[1] * x[k][1]) + fma(ov[2], x[k][2], ov[3] * x[k][3]));
      }
      // sums over the lanes of all eight rows at once: at every exchange a lane keeps half of the rows it still holds
#pragma unroll
      for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) { const double give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k]; v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o); }
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2); v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
      if ((lane & 3) == 0) vs[warp + 16 * (lane >> 2)] = v[0];    // lane bits 4, 3, 2 select row 4, 2, 1
    }
    __syncthreads();
    // Warp 0 walks 32 updates at a time, a row per lane.  With S the product of the clip factors so far and a_r = <g, u_r> / S,
    // adding u_k (whose weight relative to S is c_k = 1 / S) is a_r += c_k G[r][k], off the dependent chain, which is the norm, its
    // reciprocal root (the hardware's approximation and one step of third order) and nothing else.  S is folded into a (and the
    // weights) every eight updates.  The other warps bring the rows after the next 32 up to date meanwhile.
    double n2 = j > j0 ? st[2 * (j - 1) + 1] : 0.0, f = 1.0, Sm = 1.0, c = 1.0, npp = 1.0;
#pragma unroll 1                                                 // (run once per launch: straight-line code would come from a cold instruction cache)
    for (int b = 0; b < 4; b++) {
      if (warp == 0) {
        const int row = 32 * b + lane; const double* gr = Gd + row * CG_GD;
        double av = vs[row];
        if (b > 0) {                                              // what the 32 updates just walked add to this lane's row
          const double* cb = cs[(b - 1) & 1]; double v1 = 0.0, v2 = 0.0;
          av *= cb[32];
#pragma unroll 8
          for (int q = 0; q < 32; q += 2) { v1 = fma(cb[q], gr[32 * (b - 1) + q], v1); v2 = fma(cb[q + 1], gr[32 * (b - 1) + q + 1], v2); }
          av += v1 + v2;
        }
        // at the head of a step f is the last update's factor and Sm the product before it; a and c are relative to that product
        double ck = 0.0, R = 1.0, fk = 1.0, X = 2.0 * Sm * __shfl_sync(0xffffffffu, av, 0), gc = gr[32 * b], dg = Gd[(32 * b) * CG_GD + 32 * b];
        const double* gd = Gd + (32 * b) * CG_GD + 32 * b;        // the diagonal
#pragma unroll 1
        for (int r8 = 0; r8 < 32; r8 += 8) {
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int r = r8 + i, rn = min(r + 1, 31);
            const double np = fma(f, X, n2 + dg);
            double f0; asm volatile("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(f0) : "d"(np));
            c = c * (npp * f); Sm *= f;                           // this update's weight, and the product before its own factor
            av = fma(c, gc, av);
            const double an = __shfl_sync(0xffffffffu, av, (r + 1) & 31);
            const double h = fma(-np * f0, f0, 1.0), fc = fma(f0 * h, fma(h, 0.375, 0.5), f0);
            const bool clip = np > 1.0;                           // clip to norm 1 (lstm.go:738-750)
            gc = gr[32 * b + rn]; dg = gd[rn * (CG_GD + 1)];
            if (lane == r) ck = c;
            f = clip ? fc : 1.0; n2 = clip ? 1.0 : np; npp = clip ? np : 1.0;
            X = 2.0 * Sm * an;
            if (lane == r) fk = f;
          }
          av *= Sm; ck *= Sm; R *= Sm; c = 1.0; Sm = 1.0;
        }
        fs[32 * b + lane] = fk;
        cs[b & 1][lane] = ck; if (lane == 0) cs[b & 1][32] = R;
      }
      __syncthreads();
      if (b < 2 && warp > 0) {
        const int row = 32 * (b + 2) + tid - 32;
        if (row < CG) {
          const double* gr = Gd + row * CG_GD + 32 * b; const double* cb = cs[b & 1]; double v1 = 0.0, v2 = 0.0;
#pragma unroll 8
          for (int q = 0; q < 32; q += 2) { v1 = fma(cb[q], gr[q], v1); v2 = fma(cb[q + 1], gr[q + 1], v2); }
          vs[row] = fma(cb[32], vs[row], v1 + v2);
        }
      }
    }
    if (warp != 0) return;
    // suffix products of the factors, 32 rows at a time
    double p[4];
#pragma unroll
    for (int i = 0; i < 4; i++) p[i] = fs[32 * i + lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int i = 0; i < 4; i++) { const double y = __shfl_down_sync(0xffffffffu, p[i], o); if (lane + o < 32) p[i] *= y; }
    }
    double tail = 1.0;
#pragma unroll
    for (int i = 3; i >= 0; i--) { p[i] *= tail; om[(long)j * CG + lane + 32 * i] = p[i]; tail = __shfl_sync(0xffffffffu, p[i], 0); }
    if (lane == 0) { st[2 * j] = tail; st[2 * j + 1] = n2; }
    return;
  }
  // eight rows of the gradient matrix
  const int slab = blockIdx.x - 1, i0 = slab * 8, nr = min(8, R4 - i0), tile = clip_tile(ZW), wp = tile | 1;
  float* zp = sm; float* zn = zp + CG * wp; float* od = zn + CG * wp; float* gt = od + CG * 8;      // Z of group j-1, of group j+1 [CG][wp]; om d [CG][8]; the new rows [tile][8]
  __shared__ double red[4][CG];
  const float* D = a.D + chunk * a.stride * R4; const float* Z = a.Z + chunk * a.stride * zs;
  const float* go = a.g + ((long)chunk * 2 + ((j - 1) & 1)) * R4 * ZW; float* gw = a.g + ((long)chunk * 2 + (j & 1)) * R4 * ZW;
  const bool old = j > j0, next = j + 1 < a.groups;
  auto stage = [&](float* dst, int group, int c0, int w) {         // rows of a group, columns c0 .. c0 + w - 1, all copies in flight at once
    const float* src = Z + ((long)CG_PAD + (long)group * CG) * zs + c0;
    for (int r = warp; r < CG; r += CG_THREADS / 32) for (int c = lane; c < w; c += 32) cp_async4(dst + r * wp + c, src + (long)r * zs + c);
  };
  if (old) stage(zp, j - 1, 0, min(tile, ZW));
  if (next) stage(zn, j + 1, 0, min(tile, ZW));
  pdl_wait(); pdl_launch();                                        // what follows reads the launch before
  const double s1 = old ? st[2 * (j - 1)] : 0.0;                 // s_{j-1}
  if (old) for (int e = tid; e < CG * 8; e += CG_THREADS) {
    const int r = e >> 3, i = e & 7;
    od[e] = i < nr ? (float)(om[(long)(j - 1) * CG + r] * (double)D[((long)CG_PAD + (long)(j - 1) * CG + r) * R4 + i0 + i]) : 0.f;
  }
  float t[8];
#pragma unroll
  for (int i = 0; i < 8; i++) t[i] = 0.f;
  const int pr = tid & (CG - 1), pq = tid >> 7;                    // second half of the work: row r of group j+1, a quarter of the columns
  for (int c0 = 0; c0 < ZW; c0 += tile) {
    const int w = min(tile, ZW - c0);
    float gv[4] = {0.f, 0.f, 0.f, 0.f};                            // the old rows' values
    if (old && tid < 2 * w) {
      const int rg = tid >= w ? 4 : 0, c = tid - (rg ? w : 0);
#pragma unroll
      for (int i = 0; i < 4; i++) if (rg + i < nr) gv[i] = go[(long)(i0 + rg + i) * ZW + c0 + c];
    }
    if (c0 > 0) __syncthreads();
    if (c0 > 0 && old) stage(zp, j - 1, c0, w);                   // (the first tile is under way)
    if (c0 > 0 && next) stage(zn, j + 1, c0, w);
    cp_async_wait();
    __syncthreads();
    if (tid < 2 * w) {                                             // four rows of a column (2 CG_TILE <= CG_THREADS)
      const int rg = tid >= w ? 4 : 0, c = tid - (rg ? w : 0);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      if (old) {
        const float* zc = zp + c; const float* oc = od + rg;
#pragma unroll 16
        for (int r = 0; r < CG; r++) {
          const float z = zc[r * wp]; const float4 q = *reinterpret_cast<const float4*>(oc + 8 * r);
          acc[0] = fmaf(q.x, z, acc[0]); acc[1] = fmaf(q.y, z, acc[1]); acc[2] = fmaf(q.z, z, acc[2]); acc[3] = fmaf(q.w, z, acc[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) if (rg + i < nr) {
        if (old) acc[i] = (float)fma(s1, (double)gv[i], (double)acc[i]);
        gw[(long)(i0 + rg + i) * ZW + c0 + c] = acc[i];
      }
      *reinterpret_cast<float4*>(gt + 8 * c + rg) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();
    if (next && old) {
      const int per = (w + 3) >> 2, ce = min(w, (pq + 1) * per);
#pragma unroll 4
      for (int c = pq * per; c < ce; c++) {
        const float z = zn[pr * wp + c]; const float4 q0 = *reinterpret_cast<const float4*>(gt + 8 * c), q1 = *reinterpret_cast<const float4*>(gt + 8 * c + 4);
        t[0] = fmaf(q0.x, z, t[0]); t[1] = fmaf(q0.y, z, t[1]); t[2] = fmaf(q0.z, z, t[2]); t[3] = fmaf(q0.w, z, t[3]);
        t[4] = fmaf(q1.x, z, t[4]); t[5] = fmaf(q1.y, z, t[5]); t[6] = fmaf(q1.z, z, t[6]); t[7] = fmaf(q1.w, z, t[7]);
      }
    }
  }
  if (!next) return;
  double acc = 0.0;
  if (old) {
    const float* d = D + ((long)CG_PAD + (long)(j + 1) * CG + pr) * R4 + i0;
#pragma unroll
    for (int i = 0; i < 8; i++) if (i < nr) acc = fma((double)d[i], (double)t[i], acc);
  }
  red[pq][pr] = acc;
  __syncthreads();
  if (tid < CG) pp[((long)((j + 1) & 1) * CG + tid) * a.slabs + slab] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
}
// chunk results [nchunks][2][4H][in+H+1], buffer `par` -> flat layout gWx[4H,in] | gWh[4H,H] | gb[4H], chunks added in worker order
__global__ void lstm_scatter_grad_kernel(const float* __restrict__ Gc, int par, int nchunks, int in, int H, float* __restrict__ out) {
  const int R4 = 4 * H, ZW = in + H + 1; const long total = (long)R4 * ZW;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i / ZW), c = (int)(i % ZW);
    float v = 0.f; for (int q = 0; q < nchunks; q++) v += Gc[(2L * q + par) * total + i];
    if (c < in) out[(long)r * in + c] = v; else if (c < in + H) out[(long)R4 * in + (long)r * H + (c - in)] = v; else out[(long)R4 * in + (long)R4 * H + r] = v;
  }
}

}  // namespace gn
