// model.cu -- the compiled model (execution plan over device-resident tensors) and the C ABI.
//
// One gn_model owns: the flat parameter buffer, the flat gradient buffer and the Adam moments, all in the
// reference's flat layout (Network.initBuffers, internal/net/net.go:91-127); per-layer activation buffers
// sized for the largest batch seen; and shared scratch.  One gn_train_batch call runs the whole
// Network.TrainBatch (net.go:412-436, :721-784) for a batch on the device.
//
// Batch-level restatement of the per-sample reference semantics:
//  * top-level Dense / Conv2D use each sample's own input and pre-activation (layer.go:488-667);
//  * Dense layers inside MultiHeadAttention / TransformerBlock are called once per token and keep only their
//    LAST call's input and pre-activation (layer.go:352, :496-497, :563-567), so per sample
//        gW = (sum_t dz_t) (x) x_{T-1},   FFN ReLU mask of every token = mask of token T-1
//    which at batch level is  gW = Delta^T * X_last  (a contraction over the batch) with Delta[s] = sum_t dz[s,t];
//  * Embedding gradient: only the last sample of each worker chunk (embedding.go:151-154);
//  * LSTM: see conv_lstm.cuh.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <memory>

#include "common.cuh"
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"
#include "rowops.cuh"
#include "conv_lstm.cuh"
#include "recurrent.cuh"
#include "attention.cuh"
#include "attention_tc.cuh"
#include "conv_direct.cuh"
#include "conv_tc.cuh"
#include "nccl_dl.cuh"

namespace gn {

// ------------------------------------------------------------------ contraction dispatch
static bool force_simt_engine() { static const bool f = [] { const char* e = getenv("GONEURON_CUDA_ENGINE"); return e && strcmp(e, "simt") == 0; }(); return f; }
// Chooses the tensor-core engine for large K-major x K-major products and the SIMT engine for the rest.
static bool gemm_on_tc(Ctx* ctx, const GemmDesc& g) { return !force_simt_engine() && gemm_tc_eligible(ctx, g) && !gemm_outer_small_ok(g); }
static int gemm(Ctx* ctx, const GemmDesc& g) {
  int rc;
  if (gemm_on_tc(ctx, g)) {     // brackets its kernel launches itself
    GemmDesc h = g; BfPlanes w; if (!h.b_planes && wplanes_lookup(ctx, g, &w)) h.b_planes = &w;                 // weight matrices come with prepared planes
    rc = gemm_tc(ctx, h);
  }
  else { ProfScope prof(ctx); rc = gemm_simt(ctx, g); }
  double nb = (double)g.batch1 * g.batch2;
  double flops = 2.0 * g.M * (double)g.N * g.K * nb;
  if (g.flags & (GEMM_SKIP_UPPER | GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0)) flops *= 0.5;   // causal: about half the tiles exist
  ctx->gemm_flops += flops; ctx->gemm_launches++;
  return rc;
}
// Y[M,N] = X[M,K] * W[N,K]^T + bias (+R) (act)           -- Dense forward at batch level
static int gemm_nt(Ctx* ctx, int M, int N, int K, const float* X, long ldx, const float* W, const float* bias, float* Y, long ldy,
                   int act = GN_ACT_LINEAR, const float* R = nullptr, long ldr = 0) {
  GemmDesc g; g.M = M; g.N = N; g.K = K; g.A = X; g.sa_m = ldx; g.sa_k = 1; g.B = W; g.sb_k = 1; g.sb_n = K;
  g.C = Y; g.ldc = ldy; g.bias = bias; g.act = act; g.R = R; g.ldr = ldr; return gemm(ctx, g);
}
// dX[M,K] = dZ[M,N] * W[N,K] (+R)                          -- gradIn = W^T dz   (layer.go:631-663)
static int gemm_nn(Ctx* ctx, int M, int N, int K, const float* dZ, long ldz, const float* W, float* dX, long ldx, const float* R = nullptr, long ldr = 0) {
  GemmDesc g; g.M = M; g.N = K; g.K = N; g.A = dZ; g.sa_m = ldz; g.sa_k = 1; g.B = W; g.sb_k = K; g.sb_n = 1;
  g.C = dX; g.ldc = ldx; g.R = R; g.ldr = ldr; return gemm(ctx, g);
}
// gW[N,K] = dZ[R,N]^T * X[R,K]                              -- gradW += dz (x) x   (layer.go:591-625)
static int gemm_tn(Ctx* ctx, int R, int N, int K, const float* dZ, long ldz, const float* X, long ldx, float* gW) {
  GemmDesc g; g.M = N; g.N = K; g.K = R; g.A = dZ; g.sa_m = 1; g.sa_k = ldz; g.B = X; g.sb_k = ldx; g.sb_n = 1;
  g.C = gW; g.ldc = K; return gemm(ctx, g);
}

// Products with several weight matrices W_j [n, d], `ws` floats apart, in one launch where the tensor-core engine runs them and holds
// their planes as a stack, else one by one.  At 3600 rows of 384 the three projections are 87 tiles each: 1.8 rounds of the SMs
// together, three alone.
// Y_j[M, n] = X W_j^T + b_j; Y_j and b_j are cs and ws floats apart
static int gemm_nt_stack(Ctx* ctx, int parts, int M, int n, int d, const float* X, long ldx, const float* W, long ws, const float* bias, float* Y, long cs, const BfPlanes* x_planes = nullptr,
                         int* zmax = nullptr, int zmax_T = 0, bool* zmax_done = nullptr) {
  GemmDesc g; g.M = M; g.N = parts * n; g.K = d; g.A = X; g.sa_m = ldx; g.sa_k = 1; g.B = W; g.sb_k = 1; g.sb_n = d; g.C = Y; g.ldc = n; g.bias = bias;
  g.n_seg = n; g.c_seg = cs; g.bias_seg = ws; g.a_planes = x_planes; BfPlanes w;
  if (parts > 1 && n % 32 == 0 && gemm_on_tc(ctx, g) && wplanes_lookup(ctx, g, &w)) {
    g.b_planes = &w;
    if (zmax && d <= 2048 && ((reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(Y) | (uintptr_t)((ws | cs) * 4)) & 15) == 0) { g.zmax = zmax; g.zmax_T = zmax_T; *zmax_done = true; }
    return gemm(ctx, g);
  }
  g.N = n; g.n_seg = 0;
  for (int j = 0; j < parts; j++) { g.B = W + j * ws; g.C = Y + j * cs; g.bias = bias ? bias + j * ws : nullptr; GN_TRY(gemm(ctx, g)); g.reuse_a_planes = true; }
  return GN_OK;
}
// dX[M, d] = sum_j dZ_j W_j + R; dZ_j [M, n] are zs floats apart
static int gemm_nn_stack(Ctx* ctx, int parts, int M, int n, int d, const float* dZ, long zs, const float* W, long ws, float* dX, const float* R, const BfPlanes* z_planes = nullptr) {
  GemmDesc g; g.M = M; g.N = d; g.K = parts * n; g.A = dZ; g.sa_m = n; g.sa_k = 1; g.B = W; g.sb_k = d; g.sb_n = 1; g.C = dX; g.ldc = d; g.R = R; g.ldr = d;
  g.k_seg = n; g.a_seg = zs; g.a_planes = z_planes; BfPlanes w;
  if (parts > 1 && n % 32 == 0 && gemm_on_tc(ctx, g) && wplanes_lookup(ctx, g, &w)) { g.b_planes = &w; return gemm(ctx, g); }
  g.K = n; g.k_seg = 0; g.a_planes = nullptr;
  for (int j = 0; j < parts; j++) { g.A = dZ + j * zs; g.B = W + j * ws; GN_TRY(gemm(ctx, g)); g.R = dX; }
  return GN_OK;
}
// gW_j[n, d] = dZ_j^T X, one after the other in memory
static int gemm_tn_stack(Ctx* ctx, int parts, int R, int n, int d, const float* dZ, long zs, const float* X, long ldx, float* gW) {
  GemmDesc g; g.M = parts * n; g.N = d; g.K = R; g.A = dZ; g.sa_m = 1; g.sa_k = n; g.B = X; g.sb_k = ldx; g.sb_n = 1; g.C = gW; g.ldc = d; g.m_seg = n; g.a_seg = zs;
  if (parts > 1 && gemm_on_tc(ctx, g)) return gemm(ctx, g);
  g.M = n; g.m_seg = 0;
  for (int j = 0; j < parts; j++) { g.A = dZ + j * zs; g.C = gW + (long)j * n * d; GN_TRY(gemm(ctx, g)); }
  return GN_OK;
}
// gemm_tn with the bias gradient gb[N] = sum of dZ over its rows, inside the product where the CUDA-core engine runs it.
static int colsum(gn_model* m, const float* in, long ld, int R, int C, float* out, bool accumulate, int slot = 0);
static int weight_bias_grads(gn_model* m, Ctx* ctx, int R, int N, int K, const float* dZ, long ldz, const float* X, long ldx, float* gW, float* gb) {
  GemmDesc g; g.M = N; g.N = K; g.K = R; g.A = dZ; g.sa_m = 1; g.sa_k = ldz; g.B = X; g.sb_k = ldx; g.sb_n = 1; g.C = gW; g.ldc = K;
  if (gemm_on_tc(ctx, g)) GN_TRY(colsum(m, dZ, ldz, R, N, gb, false)); else g.a_sum = gb;
  return gemm(ctx, g);
}

// Does this weight gradient run on the side stream?  Only the CUDA-core engine's products can (no scratch), and only from some
// 3 M multiply-adds on is it worth a fork and a join (a 1.3 M one in a step of small kernels cost 4 us more than it gave).
static bool grads_on_side(Ctx* ctx, int stack, int R, int N, int K, long ldx) {
  if ((double)stack * R * N * K < 3.0e6) return false;
  GemmDesc g; g.M = N; g.N = K; g.K = R; g.sa_m = 1; g.sa_k = N; g.sb_k = ldx; g.sb_n = 1;
  return !gemm_on_tc(ctx, g);
}

struct LayerRT;
static bool ffn_planes_possible(Ctx* ctx, const LayerRT& l, int N, const float* w1, const float* w2);

// ------------------------------------------------------------------ model
struct LayerRT {
  gn_layer_desc d{};
  int in_size = 0, out_size = 0;
  int64_t p_off = 0, p_cnt = 0;
  // forward state kept for backward
  DevBuf out, z;                       // activation / pre-activation  [cap, out_size]
  DevBuf q, k, v, att, r1, n1, mid, r2, stat;   // TransformerBlock
  DevBuf att_m, att_l, att_d;          // fused attention: per-row softmax maximum, sum, and dO.O  [batch*heads*T]
  AttnSaved attn_saved;                // tcgen05 attention: operand planes of Q, K, V kept from the training forward pass for the backward pass
  DevBuf gate, up, zlast, rope;        // TransformerBlock variants: SwiGLU projections [tokens, ff]; GELU: last token's pre-activation [batch, ff]; cos | sin table
  int ff_act = GN_ACT_RELU; bool rms = false, use_rope = false;
  DevBuf mid_inv, mid_last;            // FFN hidden activation kept as operand planes (in `mid`): row scales [tokens], fp32 last-token rows [batch, ff]
  bool mid_is_planes = false;          // set by the forward pass, read by the backward pass
  DevBuf pre_i, c_all, h_all, dgate;   // LSTM
  DevBuf idx;                          // int32 payload: MaxPool argmax / embedding token ids
  const float* fin = nullptr;          // input of the last forward call (device pointer, not owned)
  int64_t s_off = 0, s_cnt = 0;        // BatchNorm2D: slice of the model's state buffer (running mean | running variance)
  // Tokens that the layers above read (TransformerBlock, Embedding; see plan_token_rows): 0 = all of a sequence's tokens, 1 = token 0,
  // 2 = token 0 and the last one.  `out` (and everything behind a block's attention) then holds that many rows per sequence.
  int out_rows = 0;
  // A block whose backward pass needs a few rows only (token 0, last token) copies them to `keep` (keep_rows) and shares its
  // activation buffers with the other blocks
  DevBuf keep; bool kept = false;
  bool in_row0 = false, row0_grad = false;   // block input is token 0 only; the gradient of the output is nonzero at token 0 only
  bool grad_replicated = false;        // multi-GPU: every rank already holds the gradient of the whole global batch (no all-reduce)
  float bn_eps = 1e-5f, bn_mom = 0.1f;
};

}  // namespace gn

struct gn_ctx { gn::Ctx c; bool alive = true; };

namespace gn { struct StepGraph; }
struct gn_model {
  ~gn_model();
  void drop_graphs();
  gn_ctx* ctx = nullptr;
  std::mutex mu;
  std::vector<gn::LayerRT> L;
  int loss_kind = 0, W = 1;
  int64_t P = 0; int in_size = 0, out_size = 0;
  gn::DevBuf params, grads, m1, v2, state; int64_t NS = 0;
  int cur_first_sample = 0;             // global index of the first sample of the batch being processed (Dropout's stream position)
  int cur_global_batch = 0;             // size of the global batch being processed (all ranks)
  uint64_t epoch = 0;                   // counts (re)allocations of the model's buffers
  bool wplanes_layerwise = false;       // this step renewed the weight planes layer by layer behind the parameter update
  const float* fwd_planes_src = nullptr; gn::BfPlanes fwd_planes{};     // operand planes of the tensor at fwd_planes_src, written by the LayerNorm that produced it
  float lr = 1e-3f, b1 = 0.9f, b2 = 0.999f, eps = 1e-8f; int timestep = 0;
  int cap = 0; bool cap_training = false;   // batch capacity of the activation buffers, and whether they can hold a training pass
  gn::DevBuf shared[19];                // activation buffers that TransformerBlocks share
  gn::DevBuf lossg, loss_s, loss_sum;
  std::vector<gn::DevBuf> scratch;      // growable shared scratch, by slot
  float last_inv_batch = 1.f;
  bool head_fused = false;              // the last forward pass left the head's softmax to head_loss_kernel
  bool stats_timed = false;             // the last step's event times have been read
  gn::DevBuf io;                        // Adam coefficients | host batch: x, y
  std::vector<std::unique_ptr<gn::StepGraph>> graphs; uint64_t graph_clock = 0;
  gn_step_stats stats{};
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ar0 = nullptr, ar1 = nullptr, comm_done = nullptr, gather_ev = nullptr;
  std::vector<cudaEvent_t> layer_ev;    // gradient of layer i complete (multi-GPU: releases its all-reduce)
  bool alive = true;
  bool has_lstm = false;
  gn::WeightPlaneTable wplanes;         // prepared tensor-core operand planes of the Dense / TransformerBlock weight matrices
};

namespace gn {

// Head of gn_model::io (floats); size of the context's pinned blocks (1 MiB); largest batch that goes through the inbound one
// (beyond that the driver's own pageable copy, which overlaps its two stages, is the quicker way)
constexpr size_t IO_ARGS = 64, STAGE_FLOATS = 1 << 18, STAGE_IN = 1 << 17;

enum Slot { S_BNG = 0, S_EMB, S_GRAM0, S_GRAM1, S_DM, S_ZM, S_W, S_TV, S_G0, S_G1, S_ND0, S_ND1, S_ND2, S_ND3, S_ND4, S_NFF, S_NFF2, S_NFF3, S_RN, S_NFFI, S_LNP0, S_LNI0, S_LNP1, S_LNI1, S_RS32, S_ATT0, S_ATT1, S_DELTA, S_PART, S_PART2, S_DZ, S_SCAN, S_XROWS, S_SIDE, S_PART3, S_PART4, S_COUNT };

static int ensure(gn_model* m, int slot, size_t n, float** out) {
  if ((int)m->scratch.size() < S_COUNT) m->scratch.resize(S_COUNT);
  DevBuf& b = m->scratch[slot];
  if (b.n < n) { GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream)); if (m->ctx->c.side_pending) GN_CUDA(cudaStreamSynchronize(m->ctx->c.side_stream)); m->epoch++; GN_TRY(b.alloc(n)); }
  *out = b.p; return GN_OK;
}

// All-gather of equal per-rank pieces on the communication stream, ordered after everything queued on the main stream so
// far; the main stream then waits for the result.  `send` may be the rank's own piece inside `recv` (in place).
static int all_gather_on_comm(gn_model* m, const float* send, float* recv, size_t count_per_rank, const char* what) {
  Ctx* ctx = &m->ctx->c;
  GN_CUDA(cudaEventRecord(m->gather_ev, ctx->stream));
  GN_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->gather_ev, 0));
  int rc = ctx->nccl->AllGather(send, recv, count_per_rank, NCCL_FLOAT32, ctx->comm, ctx->comm_stream);
  if (rc) return fail(GN_ERR_NCCL, "ncclAllGather(%s): %s", what, ctx->nccl->GetErrorString(rc));
  GN_CUDA(cudaEventRecord(m->gather_ev, ctx->comm_stream));
  GN_CUDA(cudaStreamWaitEvent(ctx->stream, m->gather_ev, 0));
  return GN_OK;
}

static int plan_layers(gn_model* m, const gn_layer_desc* layers, int n) {
  int cur = -1; int64_t off = 0;
  for (int i = 0; i < n; i++) {
    LayerRT l; l.d = layers[i]; const gn_layer_desc& d = l.d;
    switch (d.kind) {
      case GN_LAYER_DENSE:
        if (d.in_size <= 0 || d.out_size <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: Dense sizes must be positive", i);
        if (d.activation < GN_ACT_LINEAR || d.activation > GN_ACT_ELU) return fail(GN_ERR_UNSUPPORTED, "layer %d: activation %d", i, d.activation);
        l.in_size = d.in_size; l.out_size = d.out_size; l.p_cnt = (int64_t)d.in_size * d.out_size + d.out_size; break;
      case GN_LAYER_CONV2D: {
        if (d.in_size <= 0 || d.out_size <= 0 || d.kernel <= 0 || d.stride <= 0 || d.in_h <= 0 || d.in_w <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad Conv2D descriptor", i);
        if (d.activation == GN_ACT_SOFTMAX || d.activation == GN_ACT_LOGSOFTMAX) return fail(GN_ERR_UNSUPPORTED, "layer %d: Conv2D with a softmax activation", i);
        if (d.activation < GN_ACT_LINEAR || d.activation > GN_ACT_ELU) return fail(GN_ERR_UNSUPPORTED, "layer %d: activation %d", i, d.activation);
        int oh = (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, ow = (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1;
        l.in_size = d.in_size * d.in_h * d.in_w; l.out_size = d.out_size * oh * ow;
        l.p_cnt = (int64_t)d.out_size * d.in_size * d.kernel * d.kernel + d.out_size; break; }
      case GN_LAYER_CONV1D: {
        if (d.in_size <= 0 || d.out_size <= 0 || d.kernel <= 0 || d.stride <= 0 || d.padding < 0 || d.in_w <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad Conv1D descriptor", i);
        if (d.activation < GN_ACT_LINEAR || d.activation > GN_ACT_ELU || d.activation == GN_ACT_SOFTMAX || d.activation == GN_ACT_LOGSOFTMAX)
          return fail(GN_ERR_UNSUPPORTED, "layer %d: Conv1D activation %d", i, d.activation);
        const int ol = (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1;
        if (ol <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: Conv1D output length %d", i, ol);
        l.in_size = d.in_size * d.in_w; l.out_size = d.out_size * ol; l.p_cnt = (int64_t)d.out_size * d.in_size * d.kernel + d.out_size; break; }
      case GN_LAYER_MAXPOOL2D:
      case GN_LAYER_AVGPOOL2D: {
        if (d.in_size <= 0 || d.kernel <= 0 || d.stride <= 0 || d.padding < 0 || d.in_h <= 0 || d.in_w <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad pooling descriptor", i);
        int oh = (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, ow = (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1;
        l.in_size = d.in_size * d.in_h * d.in_w; l.out_size = d.in_size * oh * ow; break; }
      case GN_LAYER_FLATTEN:
        if (cur < 0) return fail(GN_ERR_INVALID_ARG, "Flatten cannot be the first layer");
        l.in_size = l.out_size = cur; break;
      case GN_LAYER_LSTM_UNROLLED:
        if (d.in_size <= 0 || d.out_size <= 0 || d.seq_len <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad LSTM descriptor", i);
        if (d.out_size > 1024) return fail(GN_ERR_UNSUPPORTED, "layer %d: LSTM hidden size > 1024", i);
        l.in_size = d.seq_len * d.in_size; l.out_size = d.return_seq ? d.seq_len * d.out_size : d.out_size;
        l.p_cnt = (int64_t)4 * d.out_size * d.in_size + (int64_t)4 * d.out_size * d.out_size + 4 * d.out_size; m->has_lstm = true; break;
      case GN_LAYER_GRU_UNROLLED:
        if (d.in_size <= 0 || d.out_size <= 0 || d.seq_len <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad GRU descriptor", i);
        if (((size_t)2 * d.out_size * d.out_size + 3 * (size_t)d.out_size) * sizeof(float) > 200 * 1024) return fail(GN_ERR_UNSUPPORTED, "layer %d: GRU hidden size %d (both recurrent matrices must fit shared memory)", i, d.out_size);
        l.in_size = d.seq_len * d.in_size; l.out_size = d.return_seq ? d.seq_len * d.out_size : d.out_size;
        l.p_cnt = (int64_t)3 * d.out_size * d.in_size + (int64_t)2 * d.out_size * d.out_size + 3 * d.out_size; break;
      case GN_LAYER_EMBEDDING: {
        int T = d.seq_len; for (int j = i + 1; j < n && T <= 0; j++) T = layers[j].seq_len;
        if (T <= 0 || d.in_size <= 0 || d.out_size <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: Embedding needs vocab, dim and a sequence length", i);
        l.d.seq_len = T; l.in_size = T; l.out_size = T * d.out_size; l.p_cnt = (int64_t)d.in_size * d.out_size; break; }
      case GN_LAYER_POSENC:
        if (d.seq_len <= 0 || d.dim <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad PositionalEncoding descriptor", i);
        l.in_size = l.out_size = d.seq_len * d.dim; l.p_cnt = (int64_t)d.seq_len * d.dim; break;
      case GN_LAYER_TRANSFORMER_BLOCK:
        if (d.seq_len <= 0 || d.dim <= 0 || d.heads <= 0 || d.ff_dim <= 0 || d.dim % d.heads) return fail(GN_ERR_INVALID_ARG, "layer %d: bad TransformerBlock descriptor (dim must be divisible by heads)", i);
        if (d.activation != 0 && d.activation != GN_ACT_RELU && d.activation != GN_ACT_GELU && d.activation != GN_ACT_SILU) return fail(GN_ERR_UNSUPPORTED, "layer %d: TransformerBlock feed-forward activation %d", i, d.activation);
        l.ff_act = d.activation == 0 ? GN_ACT_RELU : d.activation; l.rms = d.kernel != 0; l.use_rope = d.stride != 0;
        if (l.use_rope && (d.dim / d.heads) % 2) return fail(GN_ERR_INVALID_ARG, "layer %d: rotary embeddings need an even head size", i);
        l.in_size = l.out_size = d.seq_len * d.dim;
        l.p_cnt = 4 * ((int64_t)d.dim * d.dim + d.dim) + (l.rms ? 2 : 4) * (int64_t)d.dim
                + (l.ff_act == GN_ACT_SILU ? 2 * (int64_t)d.dim * d.ff_dim : (int64_t)d.dim * d.ff_dim + d.ff_dim) + ((int64_t)d.ff_dim * d.dim + d.dim); break;
      case GN_LAYER_CLS_POOLING:
        if (d.seq_len <= 0 || d.dim <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad CLSPooling descriptor", i);
        l.in_size = d.seq_len * d.dim; l.out_size = d.dim; break;
      case GN_LAYER_DROPOUT: {
        float pr = 0.f; memcpy(&pr, &d.dim, 4);
        if (d.in_size <= 0 || !(pr >= 0.f && pr < 1.f)) return fail(GN_ERR_INVALID_ARG, "layer %d: bad Dropout descriptor", i);
        if (cur >= 0 && cur != d.in_size) return fail(GN_ERR_INVALID_ARG, "layer %d: Dropout size %d does not match its input %lld", i, d.in_size, (long long)cur);
        if (m->W > 1) return fail(GN_ERR_UNSUPPORTED, "layer %d: Dropout with more than one virtual worker (every worker clone restarts the random stream)", i);
        l.in_size = l.out_size = d.in_size; l.s_off = m->NS; l.s_cnt = 2; m->NS += 2; l.bn_mom = pr; break; }
      case GN_LAYER_BATCHNORM2D:
        if (d.in_size <= 0 || d.in_h <= 0 || d.in_w <= 0) return fail(GN_ERR_INVALID_ARG, "layer %d: bad BatchNorm2D descriptor", i);
        l.in_size = l.out_size = d.in_size * d.in_h * d.in_w; l.p_cnt = 2 * (int64_t)d.in_size; l.s_off = m->NS; l.s_cnt = 2 * (int64_t)d.in_size; m->NS += l.s_cnt;
        if (d.reserved) memcpy(&l.bn_eps, &d.reserved, 4); if (d.dim) memcpy(&l.bn_mom, &d.dim, 4); break;
      case GN_LAYER_LAYERNORM:
        if (cur < 0 || d.dim <= 0 || cur % d.dim) return fail(GN_ERR_INVALID_ARG, "layer %d: LayerNorm width must divide the input size", i);
        l.in_size = l.out_size = cur; l.p_cnt = 2 * (int64_t)d.dim; break;
      case GN_LAYER_RMSNORM:
        if (cur < 0 || d.dim <= 0 || cur % d.dim) return fail(GN_ERR_INVALID_ARG, "layer %d: RMSNorm width must divide the input size", i);
        l.in_size = l.out_size = cur; l.p_cnt = d.dim; l.bn_eps = 1e-5f; if (d.reserved) memcpy(&l.bn_eps, &d.reserved, 4); break;
      default: return fail(GN_ERR_UNSUPPORTED, "layer %d: unknown layer kind %d", i, d.kind);
    }
    if (cur >= 0 && l.in_size != cur) return fail(GN_ERR_INVALID_ARG, "layer %d: input size mismatch: expected %d, got %d", i, l.in_size, cur);
    if (i == 0) m->in_size = l.in_size;
    cur = l.out_size; l.p_off = off; off += l.p_cnt;
    m->L.push_back(std::move(l));
  }
  m->out_size = cur; m->P = off; return GN_OK;
}

static void plan_token_rows(gn_model* m, bool training);
// Activation buffers of a TransformerBlock, by number (k, v and up are views: q | k | v and gate | up lie in one buffer each).
constexpr int NBLK = 18;
static DevBuf& block_buf(LayerRT& l, int k) {
  DevBuf* b[NBLK] = {&l.q, &l.k, &l.v, &l.att, &l.r1, &l.n1, &l.mid, &l.r2, &l.out, &l.stat, &l.gate, &l.up, &l.mid_last, &l.zlast, &l.mid_inv, &l.att_m, &l.att_l, &l.att_d};
  return *b[k];
}
static void block_sizes(const LayerRT& l, size_t c, size_t (&n)[NBLK]) {
  const gn_layer_desc& d = l.d; const size_t nd = c * d.seq_len * d.dim, nf = c * d.seq_len * d.ff_dim, nt = c * d.seq_len, bf = c * d.ff_dim;
  const size_t v[NBLK] = {3 * nd, 0, 0, nd, nd, nd, nf, nd, nd, 4 * nt, l.ff_act == GN_ACT_SILU ? 2 * nf : 0, 0, bf, l.ff_act == GN_ACT_GELU ? bf : 0, nt, nt * d.heads, nt * d.heads, nt * d.heads};
  for (int k = 0; k < NBLK; k++) n[k] = v[k];
}
// Which blocks can use one set of activation buffers: all of them in inference; in training those whose backward pass needs the
// few rows in `keep` (gradient at token 0 only, causal), and the top one, which runs last in the forward pass and first in
// the backward pass.  `out` alternates between two buffers (a block reads its input until its end).
static bool block_shares(const gn_model* m, const LayerRT& l, bool training) {
  if (!training) return true;
  int n_cls = 0, after = 0;
  for (auto& x : m->L) { if (x.d.kind == GN_LAYER_CLS_POOLING) n_cls++; else if (n_cls && x.d.kind == GN_LAYER_TRANSFORMER_BLOCK) after++; }
  return n_cls == 1 && after == 0 && l.row0_grad && (l.d.causal || l.out_rows);
}
// (Re)allocates every per-layer activation buffer for `cap` samples.
static int alloc_activations(gn_model* m, int cap, bool training) {
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream));
  DeviceMemory::Idle waited;                  // (between steps the context's other streams have been joined to this one)
  size_t c = (size_t)cap;
  plan_token_rows(m, training);
  m->epoch++;
  m->cap = 0; m->cap_training = false;        // until every buffer is there: after a failure the next call, of whatever size, starts over
  size_t most[NBLK] = {}; int n_shared = 0;
  for (auto& l : m->L) if (l.d.kind == GN_LAYER_TRANSFORMER_BLOCK) {
    for (int k = 0; k < NBLK; k++) block_buf(l, k).release();
    if (block_shares(m, l, training)) { size_t need[NBLK]; block_sizes(l, c, need); for (int k = 0; k < NBLK; k++) most[k] = std::max(most[k], need[k]); n_shared++; }
  }
  for (int k = 0; k < NBLK; k++) GN_TRY(m->shared[k].alloc(most[k]));
  GN_TRY(m->shared[NBLK].alloc(n_shared > 1 ? most[8] : 0));
  n_shared = 0;
  GN_TRY(m->io.alloc(IO_ARGS + (c * m->in_size + 63) / 64 * 64 + 64 + c * m->out_size));
  GN_TRY(m->lossg.alloc(c * m->out_size)); GN_TRY(m->loss_s.alloc(c)); GN_TRY(m->loss_sum.alloc(4));
  for (auto& l : m->L) {
    const gn_layer_desc& d = l.d;
    switch (d.kind) {
      case GN_LAYER_DENSE:
        GN_TRY(l.out.alloc(c * l.out_size));
        if (d.activation != GN_ACT_LINEAR && d.activation != GN_ACT_RELU) GN_TRY(l.z.alloc(c * l.out_size));
        break;
      case GN_LAYER_CONV2D: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.z.alloc(c * l.out_size)); break;
      case GN_LAYER_MAXPOOL2D: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.idx.alloc(c * l.out_size)); break;
      case GN_LAYER_AVGPOOL2D: GN_TRY(l.out.alloc(c * l.out_size)); break;
      case GN_LAYER_CONV1D: GN_TRY(l.out.alloc(c * l.out_size)); break;
      case GN_LAYER_DROPOUT: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.z.alloc(c * l.out_size)); break;      // z = the mask
      case GN_LAYER_FLATTEN: break;
      case GN_LAYER_LSTM_UNROLLED: {
        size_t th = c * d.seq_len * d.out_size;
        GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.pre_i.alloc(th)); GN_TRY(l.c_all.alloc(th)); GN_TRY(l.h_all.alloc(th)); GN_TRY(l.z.alloc(th)); GN_TRY(l.dgate.alloc(4 * th)); break; }      // pre_i: input gates, z: tanh of the cell states
      case GN_LAYER_GRU_UNROLLED: {
        size_t th = c * d.seq_len * d.out_size;     // pre_i: pre-activations [.,T,3H]; c_all: h_{t-1}; z: r (.) h_{t-1}; dgate: deltas [.,T,3H]
        GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.pre_i.alloc(3 * th)); GN_TRY(l.c_all.alloc(th)); GN_TRY(l.h_all.alloc(th)); GN_TRY(l.z.alloc(th)); GN_TRY(l.dgate.alloc(3 * th)); break; }
      case GN_LAYER_EMBEDDING: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.idx.alloc(c * d.seq_len)); break;
      case GN_LAYER_POSENC: GN_TRY(l.out.alloc(c * l.out_size)); break;
      case GN_LAYER_TRANSFORMER_BLOCK: {
        size_t need[NBLK]; block_sizes(l, c, need);
        const bool share = block_shares(m, l, training), kept = share && training && !l.out_rows;
        for (int k = 0; k < NBLK; k++) {
          DevBuf& b = block_buf(l, k);
          const bool own = !share || (training && (k == 12 || k == 13));      // the last token's feed-forward rows are read by the backward pass
          if (own) GN_TRY(b.alloc(need[k])); else b.view(need[k] ? m->shared[k == 8 && n_shared % 2 ? NBLK : k].p : nullptr, need[k]);
        }
        if (share) n_shared++;
        const size_t nd = need[3], nf = need[6]; l.k.view(l.q.p + nd, nd); l.v.view(l.q.p + 2 * nd, nd);
        if (need[10]) l.up.view(l.gate.p + nf, nf);
        if (kept) GN_TRY(l.keep.alloc(c * (5 * (size_t)d.dim + 3 * (size_t)d.ff_dim + 4))); else l.keep.release();
        break; }
      case GN_LAYER_CLS_POOLING: GN_TRY(l.out.alloc(c * l.out_size)); break;
      case GN_LAYER_LAYERNORM: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.stat.alloc(2 * c * (l.in_size / d.dim))); break;
      case GN_LAYER_RMSNORM: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.stat.alloc(c * (l.in_size / d.dim))); break;
      case GN_LAYER_BATCHNORM2D: GN_TRY(l.out.alloc(c * l.out_size)); GN_TRY(l.stat.alloc(3 * c * d.in_size)); break;
    }
  }
  m->cap = cap; m->cap_training = training; return GN_OK;
}
static int ensure_capacity(gn_model* m, int B, bool training) {
  if (B <= m->cap && (!training || m->cap_training)) return GN_OK;
  return alloc_activations(m, std::max(B, m->cap), training || m->cap_training);
}

static inline unsigned ew_grid(Ctx* ctx, long n, int block = 256) { long g = (n + block - 1) / block; long mx = (long)ctx->sm_count * 16; return (unsigned)std::max<long>(1, std::min(g, mx)); }

// out[c] (=|+=) sum over R rows of in[r*ld + c]
static int colsum(gn_model* m, const float* in, long ld, int R, int C, float* out, bool accumulate, int slot) {
  Ctx* ctx = &m->ctx->c;
  // slabs of 16 rows and up for a batch (bound by the latency of a slab's loads), of 64 and up for many rows
  const int chunks = std::max(1, R <= 1024 ? std::min(R / 16, 16) : std::min(R / 64, 128));
  float* part; GN_TRY(ensure(m, slot ? slot : S_PART, (size_t)chunks * C * 2, &part));
  GN_LAUNCH(ctx, colsum_partial_kernel, dim3(cdiv(C, 128), chunks), 128, 0, in, ld, R, C, part);
  GN_LAUNCH(ctx, colsum_final_kernel, cdiv(C, 128), 128, 0, part, chunks, C, out, accumulate ? 1 : 0);
  return check_launch("colsum");
}

// LayerNorm / RMSNorm: the row-in-registers kernels where the row length and the alignment allow it.  stat: [2][rows] mean | deviation, or [rows] rms.
// `po` (optional): the output also as operand planes; *emitted tells the caller whether the kernel that ran could do it.
static bool norm_vec_ok(int n, std::initializer_list<const void*> ptrs) {
  uintptr_t a = 0; for (auto p : ptrs) a |= reinterpret_cast<uintptr_t>(p);
  return n % 4 == 0 && n <= 1024 && (a & 15) == 0;
}
template <bool RMS, int NV> struct NormRun {
  static void fwd(Ctx* ctx, const float* x, const float* ga, const float* be, float* y, float* sa, float* sb, long rows, int n, float eps, const RowPlaneOut& po) {
    if ((n + 127) / 128 == NV) { GN_LAUNCH(ctx, (norm_fwd_vec_kernel<NV, RMS>), cdiv(rows, 8), 256, 0, x, ga, be, y, sa, sb, rows, n, eps, po); }
    else if constexpr (NV > 1) NormRun<RMS, NV - 1>::fwd(ctx, x, ga, be, y, sa, sb, rows, n, eps, po);
  }
  static void bwd(Ctx* ctx, int blocks, const float* g, const float* x, const float* ga, const float* sa, const float* sb, float* dx, float* part, long rows, int n, long ldx, long lds, const RowPlaneOut& po) {
    if ((n + 127) / 128 == NV) { GN_LAUNCH(ctx, (norm_bwd_vec_kernel<NV, RMS>), blocks, 256, 0, g, x, ga, sa, sb, dx, part, rows, n, ldx, lds, po); }
    else if constexpr (NV > 1) NormRun<RMS, NV - 1>::bwd(ctx, blocks, g, x, ga, sa, sb, dx, part, rows, n, ldx, lds, po);
  }
};
template <int NV> struct EmbedRun {
  static void fwd(Ctx* ctx, const float* ids, const float* E, const float* P, float* out, long tokens, int T, int d, int V, int* idx, int row0_only, const RowPlaneOut& po) {
    if ((d + 127) / 128 == NV) { GN_LAUNCH(ctx, embedding_fwd_vec_kernel<NV>, cdiv(tokens, 8), 256, 0, ids, E, P, out, tokens, T, d, V, idx, ctx->d_status, row0_only, po); }
    else if constexpr (NV > 1) EmbedRun<NV - 1>::fwd(ctx, ids, E, P, out, tokens, T, d, V, idx, row0_only, po);
  }
};
static int norm_forward(Ctx* ctx, bool rms, const float* x, const float* gamma, const float* beta, float* y, float* stat, long rows, int n, float eps,
                        const RowPlaneOut* po = nullptr, bool* emitted = nullptr) {
  if (norm_vec_ok(n, {x, y, gamma, beta})) {
    const RowPlaneOut out = po ? *po : RowPlaneOut{};
    if (emitted) *emitted = out.p != nullptr;
    if (rms) NormRun<true, 8>::fwd(ctx, x, gamma, beta, y, stat, stat, rows, n, eps, out);
    else NormRun<false, 8>::fwd(ctx, x, gamma, beta, y, stat, stat + rows, rows, n, eps, out);
  } else {
    if (emitted) *emitted = false;
    if (rms) GN_LAUNCH(ctx, rmsnorm_fwd_kernel, cdiv(rows, 8), 256, 0, x, gamma, y, stat, rows, n, eps);
    else GN_LAUNCH(ctx, layernorm_fwd_kernel, cdiv(rows, 8), 256, 0, x, gamma, beta, y, stat, stat + rows, rows, n, eps);
  }
  return check_launch("norm_forward");
}
// Register-row kernel: dx and the parameter sums from one reading of g and x; the blocks' partial sums are added by a second launch
// unless there is only one: beside the main stream if `side_slot` names a scratch slot that is this call's own until the layer's end.
static int norm_backward_vec(gn_model* m, bool rms, const float* g, const float* x, long ldx, const float* gamma, const float* sa, const float* sb, long lds, float* dx,
                             float* gGamma, float* gBeta, long rows, int n, const RowPlaneOut& out, int side_slot = 0) {
  Ctx* ctx = &m->ctx->c; float* part;
  const int blocks = (int)std::max<long>(1, std::min<long>((rows + 7) / 8, (n <= 512 ? 2L : 1L) * ctx->sm_count));      // as many as are resident
  const bool direct = blocks == 1 && (rms || gBeta == gGamma + n) && (reinterpret_cast<uintptr_t>(gGamma) & 15) == 0;
  if (direct) part = gGamma; else GN_TRY(ensure(m, side_slot ? side_slot : S_PART2, (size_t)blocks * 2 * n, &part));
  if (rms) NormRun<true, 8>::bwd(ctx, blocks, g, x, gamma, sa, sb, dx, part, rows, n, ldx, lds, out);
  else NormRun<false, 8>::bwd(ctx, blocks, g, x, gamma, sa, sb, dx, part, rows, n, ldx, lds, out);
  if (!direct) {
    auto final = [&]() -> int { GN_LAUNCH(ctx, layernorm_pgrad_final_kernel, cdiv(n, 32), 1024, 0, part, blocks, n, gGamma, rms ? nullptr : gBeta); return GN_OK; };
    GN_TRY(side_slot ? side_run(ctx, final) : final());
  }
  return check_launch("norm_backward");
}
// dx (may alias g), gGamma and gBeta (null for RMSNorm) are written.
static int norm_backward(gn_model* m, bool rms, const float* g, const float* x, const float* gamma, const float* stat, float* dx, float* gGamma, float* gBeta, long rows, int n,
                         const RowPlaneOut* po = nullptr, bool* emitted = nullptr, int side_slot = 0) {
  Ctx* ctx = &m->ctx->c; float* part;
  if (norm_vec_ok(n, {g, x, dx, gamma})) {
    const RowPlaneOut out = po ? *po : RowPlaneOut{};
    if (emitted) *emitted = out.p != nullptr;
    return norm_backward_vec(m, rms, g, x, n, gamma, stat, rms ? stat : stat + rows, 1, dx, gGamma, gBeta, rows, n, out, side_slot);
  }
  if (emitted) *emitted = false;
  const int chunks = (int)std::max<long>(1, std::min<long>(rows / 64, 128));
  GN_TRY(ensure(m, S_PART2, (size_t)chunks * 2 * n, &part));
  if (rms) {
    GN_LAUNCH(ctx, rmsnorm_pgrad_partial_kernel, dim3(cdiv(n, 128), chunks), 128, 0, g, x, stat, rows, n, part);
    GN_LAUNCH(ctx, rmsnorm_pgrad_final_kernel, cdiv(n, 128), 128, 0, part, chunks, n, gGamma);
    GN_LAUNCH(ctx, rmsnorm_bwd_kernel, cdiv(rows, 8), 256, 0, g, x, gamma, stat, dx, rows, n);
  } else {
    GN_LAUNCH(ctx, layernorm_pgrad_partial_kernel, dim3(cdiv(n, 128), chunks), 128, 0, g, x, stat, stat + rows, rows, n, part);
    GN_LAUNCH(ctx, layernorm_pgrad_final_kernel, cdiv(n, 32), 1024, 0, part, chunks, n, gGamma, gBeta);
    GN_LAUNCH(ctx, layernorm_bwd_kernel, cdiv(rows, 8), 256, 0, g, x, gamma, stat, stat + rows, dx, rows, n);
  }
  return check_launch("norm_backward");
}
// cos | sin of the rotary embedding per (position, pair index), with the reference's conversions (transformer.go:217-221):
// theta and position * theta are rounded to float32, cos and sin taken in float64 and rounded to float32.
static int rope_table(Ctx* ctx, LayerRT& l) {
  const int T = l.d.seq_len, hd = l.d.dim / l.d.heads, half = hd / 2;
  if (l.rope.n >= (size_t)T * half * 2) return GN_OK;
  std::vector<float> tab((size_t)T * half * 2);
  for (int t = 0; t < T; t++) for (int i = 0; i < half; i++) {
    const float theta = (float)std::pow(10000.0, -(double)(2 * i) / (double)hd);
    const float mt = (float)t * theta;
    tab[((size_t)t * half + i) * 2] = (float)std::cos((double)mt); tab[((size_t)t * half + i) * 2 + 1] = (float)std::sin((double)mt);
  }
  GN_TRY(l.rope.alloc(tab.size()));
  GN_CUDA(copy_h2d(ctx, l.rope.p, tab.data(), tab.size() * 4)); return GN_OK;
}

// Rotation of one or two arrays of `rows` rows, T positions per sequence, in place
static void rope(Ctx* ctx, const LayerRT& l, float* x, float* y, int rows, int T, float sign, int tstep) {
  const int D = l.d.dim, hd = D / l.d.heads;
  const bool vec = hd % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  if (vec) GN_LAUNCH(ctx, rope_kernel<4>, dim3(ew_grid(ctx, (long)rows * (D / 8)), y ? 2 : 1), 256, 0, x, y, (const float*)l.rope.p, (long)rows, T, D, hd, sign, tstep);
  else GN_LAUNCH(ctx, rope_kernel<1>, dim3(ew_grid(ctx, (long)rows * (D / 2)), y ? 2 : 1), 256, 0, x, y, (const float*)l.rope.p, (long)rows, T, D, hd, sign, tstep);
}
// A LayerNorm of a block can hand its output to the next contraction as operand planes (RowPlaneOut) when that
// contraction runs on the tensor-core engine; `slotp` / `sloti` receive the planes and the inverse row scales.
static bool norm_planes_wanted(Ctx* ctx, int rows, int n, int consumer_n) {
  static const bool off = getenv("GONEURON_CUDA_NO_NORM_PLANES") != nullptr;
  if (off || force_simt_engine() || n % 4 || n > 1024) return false;
  GemmDesc g; g.M = rows; g.N = consumer_n; g.K = n; g.sa_m = n; g.sa_k = 1; g.sb_k = 1; g.sb_n = n;
  return gemm_tc_eligible(ctx, g) && !gemm_outer_small_ok(g);
}
static int norm_planes_alloc(gn_model* m, int slotp, int sloti, int rows, int n, RowPlaneOut* po, BfPlanes* planes, float* rownorm) {
  float *pp, *pi; const int ldp = tc_ldp(n); GN_TRY(ensure(m, slotp, (size_t)rows * ldp, &pp)); GN_TRY(ensure(m, sloti, (size_t)rows, &pi));
  *planes = BfPlanes{reinterpret_cast<__half*>(pp), pi, rows, n, ldp, 1};
  *po = RowPlaneOut{planes->base, pi, rownorm};
  return GN_OK;
}

// The fused kernels (attention.cuh) are the default; GONEURON_CUDA_ATTENTION=unfused selects the path that
// materialises the score matrices and runs the five products as batched contractions on the tcgen05 engine.
static bool use_fused_attention(const gn_layer_desc& d) {
  static const bool unfused = [] { const char* e = getenv("GONEURON_CUDA_ATTENTION"); return e && strcmp(e, "unfused") == 0; }();
  return !unfused && attn_fused_supported(d.dim / d.heads, d.dim);
}

// ---------------------------------------------------------------- Conv2D
// Register-tiled CUDA-core kernels (conv_direct.cuh) or implicit GEMM on the tensor cores (conv_tc.cuh); what neither takes (a stride
// above one on the CUDA cores, other windows) runs on the plain direct kernels of conv_lstm.cuh.
enum ConvEngine { CONV_AUTO, CONV_CUDA, CONV_TC };
static ConvEngine conv_engine(Ctx* ctx, const ConvShape& c, ConvEngine want) {
  if (want == CONV_AUTO) want = conv_direct_preferred(c) ? CONV_CUDA : CONV_TC;
  return want == CONV_TC && conv_tc_supported(ctx, c) ? CONV_TC : CONV_CUDA;
}
// z / out: [B, outC, oH, oW].  Bias and the activation are applied by the kernel that makes the sums (on the tensor cores LINEAR and
// RELU; the others from the kept pre-activation z, which only they need).
static int conv_forward(Ctx* ctx, const ConvShape& c, int act, float alpha, const float* x, const float* p, float* z, float* out, ConvEngine want) {
  const long n = (long)c.B * c.outC * c.oH * c.oW; const float* bias = p + (long)c.outC * c.inC * c.k * c.k;
  const bool simple = act == GN_ACT_LINEAR || act == GN_ACT_RELU;
  if (conv_engine(ctx, c, want) == CONV_TC) {
    GN_TRY(conv_tc_forward(ctx, c, x, p, bias, simple ? out : z, simple ? act : GN_ACT_LINEAR));
    if (!simple) GN_LAUNCH(ctx, act_forward_kernel, ew_grid(ctx, n), 256, 0, z, out, n, act, alpha);
  } else if (conv_direct_supported(c)) return conv_direct_forward(ctx, c, x, p, bias, simple ? nullptr : z, out, act, alpha);
  else GN_LAUNCH(ctx, conv2d_fwd_kernel, ew_grid(ctx, n), 256, 0, x, p, bias, z, out, c, act, alpha);
  return check_launch("conv_forward");
}
// g: gradient with respect to the activation; gW / gb and dx (may be null) are written.
static int conv_backward(gn_model* m, const ConvShape& c, int act, float alpha, const float* g, const float* x, const float* p, const float* z, const float* out,
                         float* gW, float* gb, float* dx, ConvEngine want) {
  Ctx* ctx = &m->ctx->c;
  const long n = (long)c.B * c.outC * c.oH * c.oW; const int nW = c.outC * c.inC * c.k * c.k;
  const ConvEngine eng = conv_engine(ctx, c, want); const bool direct = eng == CONV_CUDA && conv_direct_supported(c);
  // ReLU'(z) = [z > 0] = [a > 0], so ReLU works from the activation (the caller passes LINEAR if g already carries it)
  const float* dz = g;
  if (act != GN_ACT_LINEAR) {
    float* dzb; GN_TRY(ensure(m, S_DZ, (size_t)n, &dzb));
    GN_LAUNCH(ctx, act_backward_kernel, ew_grid(ctx, n), 256, 0, g, act == GN_ACT_RELU ? out : z, dzb, n, act, alpha); dz = dzb;
  }
  if (direct) {
    float* part; GN_TRY(ensure(m, S_PART, conv_wgrad_part_floats(ctx, c), &part));
    GN_TRY(conv_direct_wgrad(ctx, c, dz, x, part, gW));
    return dx ? conv_direct_dgrad(ctx, c, dz, p, dx) : GN_OK;
  }
  if (eng == CONV_TC) {
    float* part; GN_TRY(ensure(m, S_PART, (size_t)c.B * (nW + c.outC), &part));
    GN_TRY(conv_tc_wgrad(ctx, c, dz, x, part, gW, gb));
  } else if (c.k == 3 || c.k == 5 || c.k == 1) {
    const int pairs = c.outC * c.inC, slices = std::max(1, std::min(c.B, (4 * ctx->sm_count + pairs - 1) / pairs)), ng = nW + c.outC;
    float* part; GN_TRY(ensure(m, S_PART, (size_t)slices * ng, &part));
    if (c.k == 3) GN_LAUNCH(ctx, conv2d_wgrad_tile_kernel<3>, dim3(pairs, slices), 256, 0, dz, x, part, c, slices);
    else if (c.k == 5) GN_LAUNCH(ctx, conv2d_wgrad_tile_kernel<5>, dim3(pairs, slices), 256, 0, dz, x, part, c, slices);
    else GN_LAUNCH(ctx, conv2d_wgrad_tile_kernel<1>, dim3(pairs, slices), 256, 0, dz, x, part, c, slices);
    GN_LAUNCH(ctx, conv_wgrad_final_kernel, cdiv(ng, 32), 256, 0, (const float*)part, slices, ng, gW);          // weights, then biases: gb follows gW
  } else GN_LAUNCH(ctx, conv2d_wgrad_kernel, nW + c.outC, 256, 0, dz, x, gW, gb, c);
  if (dx) {
    const long ni = (long)c.B * c.inC * c.H * c.W;
    if (eng == CONV_TC && c.s == 1) { float* wtmp; GN_TRY(ensure(m, S_DELTA, (size_t)nW, &wtmp)); GN_TRY(conv_tc_dgrad(ctx, c, dz, p, wtmp, dx)); }
    else if (c.s == 1 && c.k == 3) GN_LAUNCH(ctx, conv2d_dgrad_s1_kernel<3>, ew_grid(ctx, ni), 256, 0, dz, p, dx, c);
    else if (c.s == 1 && c.k == 5) GN_LAUNCH(ctx, conv2d_dgrad_s1_kernel<5>, ew_grid(ctx, ni), 256, 0, dz, p, dx, c);
    else GN_LAUNCH(ctx, conv2d_dgrad_kernel, ew_grid(ctx, ni), 256, 0, dz, p, dx, c);
  }
  return check_launch("conv_backward");
}

// ---------------------------------------------------------------- forward
static int attention_forward(gn_model* m, LayerRT& l, int B, float* P) {
  Ctx* ctx = &m->ctx->c; const gn_layer_desc& d = l.d;
  const int T = d.seq_len, D = d.dim, Hh = d.heads, hd = D / Hh; const long TD = (long)T * D, TT = (long)T * T;
  GemmDesc g; g.M = T; g.N = T; g.K = hd; g.A = l.q.p; g.sa_m = D; g.sa_k = 1; g.B = l.k.p; g.sb_k = 1; g.sb_n = D;
  g.C = P; g.ldc = T; g.batch1 = B; g.batch2 = Hh; g.a_b1 = TD; g.a_b2 = hd; g.b_b1 = TD; g.b_b2 = hd; g.c_b1 = Hh * TT; g.c_b2 = TT;
  g.flags = d.causal ? GEMM_SKIP_UPPER : 0;
  GN_TRY(gemm(ctx, g));
  long rows = (long)B * Hh * T;
  float inv_scale = 1.f / sqrtf((float)hd);
  GN_LAUNCH(ctx, attn_softmax_kernel, cdiv(rows, 8), 256, 0, P, T, inv_scale, d.causal, rows);
  GemmDesc o; o.M = T; o.N = hd; o.K = T; o.A = P; o.sa_m = T; o.sa_k = 1; o.B = l.v.p; o.sb_k = D; o.sb_n = 1;
  o.C = l.att.p; o.ldc = D; o.batch1 = B; o.batch2 = Hh; o.a_b1 = Hh * TT; o.a_b2 = TT; o.b_b1 = TD; o.b_b2 = hd; o.c_b1 = TD; o.c_b2 = hd;
  o.flags = d.causal ? GEMM_KEND_AT_M0 : 0;
  return gemm(ctx, o);
}

// Views into a TransformerBlock's slice of a flat buffer: MHA (wQ, wK, wV, wOut, each W | b) | norm1 | norm2 | ff1 | ff2
// (transformer.go:1038-1056).  RMSNorm has a gain only (be1 = be2 = null); a SwiGLU first layer is W (gate) | V (up) without
// biases (w1 = W, v1 = V, b1 = null).
struct BlockParams { const float *wq, *bq, *wk, *bk, *wv, *bv, *wo, *bo, *g1, *be1, *g2, *be2, *w1, *b1, *v1, *w2, *b2; };
static BlockParams block_params(const float* p, int D, int F, bool rms = false, int ff_act = GN_ACT_RELU) {
  BlockParams b; long dd = (long)D * D;
  b.wq = p; b.bq = p + dd; p += dd + D; b.wk = p; b.bk = p + dd; p += dd + D; b.wv = p; b.bv = p + dd; p += dd + D; b.wo = p; b.bo = p + dd; p += dd + D;
  if (rms) { b.g1 = p; b.be1 = nullptr; p += D; b.g2 = p; b.be2 = nullptr; p += D; }
  else { b.g1 = p; b.be1 = p + D; p += 2 * D; b.g2 = p; b.be2 = p + D; p += 2 * D; }
  if (ff_act == GN_ACT_SILU) { b.w1 = p; b.v1 = p + (long)D * F; b.b1 = nullptr; p += 2 * (long)D * F; }
  else { b.w1 = p; b.b1 = p + (long)D * F; b.v1 = nullptr; p += (long)D * F + F; }
  b.w2 = p; b.b2 = p + (long)F * D; return b;
}

// Which tokens of a TransformerBlock's output are read at all.  CLSPooling passes on token 0 and nothing else
// (transformer.go:1684), and the gradient it returns is zero at every other token (:1715-1724).  So, of the block below it:
//   * inference needs token 0 only; training also the last token, whose activations are the input side of the inner Dense
//     layers' weight gradients (layer.go:496-497) -- the queries, the output projection, the norms and the feed-forward
//     part run on those one or two rows per sequence, keys and values on all tokens;
//   * with a causal mask token 0 sees key 0 alone: its attention output is its own value row.  In inference the blocks
//     further down are then only needed at token 0 as well, and in training the gradient stays at token 0 through all of
//     them (the softmax over one score is the constant 1: no gradient reaches the queries and keys).
// The values of the rows that are computed, and every gradient, are those of the computation over all tokens: what is left
// out there are rows that nothing reads and products with rows of zeros.
static void plan_token_rows(gn_model* m, bool training) {
  for (auto& l : m->L) { l.out_rows = 0; l.in_row0 = l.row0_grad = false; }
  for (int li = (int)m->L.size() - 1; li > 0; li--) {
    if (m->L[li].d.kind != GN_LAYER_CLS_POOLING) continue;
    const int T = m->L[li].d.seq_len, D = m->L[li].d.dim; bool top = true;
    for (int k = li - 1; k >= 0 && m->L[k].d.kind == GN_LAYER_TRANSFORMER_BLOCK && m->L[k].d.dim == D && m->L[k].d.seq_len == T; k--) {
      LayerRT& b = m->L[k];
      if (!attn_rows_fit(T, D / b.d.heads)) break;
      b.row0_grad = training;
      if (top || !training) b.out_rows = training && T > 1 ? 2 : 1;
      top = false;
      if (!b.d.causal) break;
      b.in_row0 = !training && T > 1;
    }
  }
}
// Rows per sequence that the layer after `li` wants of an embedding's output: 1 (token 0) or 0 (all).
static int next_rows(const gn_model* m, size_t li, int T, int D) {
  if (li + 1 >= m->L.size()) return 0;
  const LayerRT& n = m->L[li + 1];
  return n.d.kind == GN_LAYER_TRANSFORMER_BLOCK && n.in_row0 && n.d.seq_len == T && n.d.dim == D ? 1 : 0;
}

// Rows that the SwiGLU kernels with plane output take
static bool swiglu_planes_ok(const LayerRT& l) {
  const int F = l.d.ff_dim;
  return !force_simt_engine() && F % 32 == 0 && F <= 4096 && ((reinterpret_cast<uintptr_t>(l.gate.p) | reinterpret_cast<uintptr_t>(l.up.p)) & 15) == 0;
}
template <int NV> struct SwigluRun {
  static void fwd(Ctx* ctx, const float* gate, const float* up, const BfPlanes& p, float* last, int T, int rows, int F) {
    if ((F + 511) / 512 == NV) { GN_LAUNCH(ctx, swiglu_fwd_planes_kernel<NV>, rows, SW_THREADS, 0, gate, up, p.base, p.inv_scale, last, T, F); }
    else if constexpr (NV > 1) SwigluRun<NV - 1>::fwd(ctx, gate, up, p, last, T, rows, F);
  }
  static void bwd(Ctx* ctx, const float* g, const float* gate, const float* up, float* dG, float* dU, const BfPlanes& p, int T, int rows, int F) {
    if ((F + 511) / 512 == NV) { GN_LAUNCH(ctx, swiglu_bwd_planes_kernel<NV>, rows, SW_THREADS, 0, g, gate, up, dG, dU, p.base, p.inv_scale, T, F); }
    else if constexpr (NV > 1) SwigluRun<NV - 1>::bwd(ctx, g, gate, up, dG, dU, p, T, rows, F);
  }
};

static KeepRows keep_layout(const LayerRT& l, int B) {
  const long BD = (long)B * l.d.dim, BF = (long)B * l.d.ff_dim; float* p = l.keep.p;
  return KeepRows{p, p + BD, p + 2 * BD, p + 3 * BD, p + 4 * BD, p + 5 * BD, p + 5 * BD + BF, p + 5 * BD + 2 * BF, p + 5 * BD + 3 * BF};
}
// One TransformerBlock forward.  `TE` rows per sequence go through everything behind the keys and values: all T, or the one
// or two that the layers above read (plan_token_rows).  The backward pass finds the same number in l.out_rows.
static int block_forward(gn_model* m, size_t li, int B, const float* cur, bool training, const float** out) {
  Ctx* ctx = &m->ctx->c; LayerRT& l = m->L[li]; const gn_layer_desc& d = l.d; const float* p = m->params.p + l.p_off;
  const int T = d.seq_len, D = d.dim, F = d.ff_dim, hd = D / d.heads, N = B * T; const BlockParams bp = block_params(p, D, F, l.rms, l.ff_act);
  const int TE = l.out_rows ? l.out_rows : T, NE = B * TE; const bool rows_only = l.out_rows != 0;
  // the block's input rows of the TE tokens: in place, strided (token 0 of every sequence) or gathered (tokens 0 and T - 1)
  const float* xe = cur; long ldx = D;
  const bool in_compact = li > 0 && m->L[li - 1].out_rows == 1;
  if (rows_only && !in_compact && T > 1) {
    if (TE == 1) ldx = (long)T * D;
    else { GN_TRY(ensure(m, S_XROWS, (size_t)NE * D, const_cast<float**>(&xe))); GN_LAUNCH(ctx, gather_ends_kernel, NE, 128, 0, cur, const_cast<float*>(xe), T, D); }
  }
  if (l.in_row0) {
    // causal, token 0 only: it attends to itself alone, so its attention output is its value row
    GN_TRY(gemm_nt(ctx, B, D, D, xe, ldx, bp.wv, bp.bv, l.att.p, D));
  } else {
    // the operand planes of the projections' input come from the norm that produced it (the previous block's) if it made any
    const BfPlanes* xp = m->fwd_planes_src == cur && m->fwd_planes.rows == N && m->fwd_planes.K == D ? &m->fwd_planes : nullptr;
    const long dd = (long)D * D + D;
    const bool tc_att = !rows_only && use_fused_attention(d) && attn_tc_supported(ctx, hd, T, B, d.heads, D); bool zmax_done = false; int* zmax = nullptr;
    AttnSaved* saved = training && !l.row0_grad ? &l.attn_saved : nullptr;      // planes of Q, K and V are kept for a backward pass that walks all queries
    if (tc_att && !l.use_rope) GN_TRY(attn_tc_max_words(ctx, saved, B * d.heads, T, &zmax));
    if (!rows_only) GN_TRY(gemm_nt_stack(ctx, 3, N, D, D, cur, D, bp.wq, dd, bp.bq, l.q.p, l.k.p - l.q.p, xp, zmax, T, &zmax_done));
    else {
      GN_TRY(gemm_nt_stack(ctx, 2, N, D, D, cur, D, bp.wk, dd, bp.bk, l.k.p, l.k.p - l.q.p, xp));
      GN_TRY(gemm_nt(ctx, NE, D, D, xe, ldx, bp.wq, bp.bq, l.q.p, D));
    }
    if (l.use_rope) {   // rotary embeddings on q and k, in place: attention and its backward pass see the rotated tensors (transformer.go:457-461)
      GN_TRY(rope_table(ctx, l));
      rope(ctx, l, l.q.p, rows_only ? nullptr : l.k.p, NE, TE, 1.f, rows_only ? T - 1 : 1);
      if (rows_only) rope(ctx, l, l.k.p, nullptr, N, T, 1.f, 1);
    }
    if (rows_only) GN_TRY(attn_rows_fwd(ctx, l.q.p, l.k.p, l.v.p, l.att.p, B, T, TE, D, d.heads, d.causal));
    else if (use_fused_attention(d)) {
      if (tc_att) GN_TRY(attn_tc_fwd(ctx, l.q.p, l.k.p, l.v.p, l.att.p, l.att_m.p, l.att_l.p, B, T, D, d.heads, d.causal, saved, zmax_done));
      else GN_TRY(attn_fwd(ctx, hd, l.q.p, l.k.p, l.v.p, l.att.p, l.att_m.p, l.att_l.p, B, T, D, d.heads, d.causal));
    } else {
      float* P; GN_TRY(ensure(m, S_ATT0, (size_t)B * d.heads * T * T, &P));
      GN_TRY(attention_forward(m, l, B, P));
    }
  }
  m->fwd_planes_src = nullptr;
  GN_TRY(gemm_nt(ctx, NE, D, D, l.att.p, D, bp.wo, bp.bo, l.r1.p, D, GN_ACT_LINEAR, xe, ldx));          // res1 = x + att
  float* st = l.stat.p;
  // norm 1 hands its output to ff1 as operand planes (and the row norms ff1's plane-writing epilogue needs)
  RowPlaneOut po1{}; BfPlanes n1p{}; bool n1_planes = false; float* rn1 = nullptr;
  if (norm_planes_wanted(ctx, NE, D, F)) { GN_TRY(ensure(m, S_RN, (size_t)NE, &rn1)); GN_TRY(norm_planes_alloc(m, S_LNP0, S_LNI0, NE, D, &po1, &n1p, rn1)); }
  GN_TRY(norm_forward(ctx, l.rms, l.r1.p, bp.g1, bp.be1, l.n1.p, st, (long)NE, D, 1e-5f, po1.p ? &po1 : nullptr, &n1_planes));
  {   // feed-forward: ff1 -> ff2, res2 = norm1 + ff
    GemmDesc g1; g1.M = NE; g1.N = F; g1.K = D; g1.A = l.n1.p; g1.sa_m = D; g1.sa_k = 1; g1.B = bp.w1; g1.sb_k = 1; g1.sb_n = D; g1.C = l.mid.p; g1.ldc = F; g1.bias = bp.b1;
    if (n1_planes) g1.a_planes = &n1p;
    const long nf = (long)NE * F;
    BfPlanes midp{reinterpret_cast<__half*>(l.mid.p), l.mid_inv.p, NE, F, F, 1};
    l.mid_is_planes = ffn_planes_possible(ctx, l, NE, bp.w1, bp.w2);
    if (l.mid_is_planes) {
      // the hidden activation is only ever the A operand of ff2 (and, for its last-token rows, a gate and a weight-gradient
      // input): the epilogue writes it as operand planes into the same buffer, no fp32 copy and no split pass
      const WeightPlaneEntry* we = nullptr; BfPlanes w; wplanes_lookup(ctx, g1, &w, &we);
      float* rn; GN_TRY(ensure(m, S_RN, (size_t)NE, &rn));
      TcPlaneOut po{midp, we->maxabs, l.mid_last.p, TE}; po.z_last = training && l.ff_act == GN_ACT_GELU ? l.zlast.p : nullptr;
      g1.act = l.ff_act; g1.C = nullptr; g1.plane_out = &po; g1.a_rownorm = rn; GN_TRY(gemm(ctx, g1));
    } else if (l.ff_act == GN_ACT_RELU) { g1.act = GN_ACT_RELU; GN_TRY(gemm(ctx, g1)); }
    else if (l.ff_act == GN_ACT_GELU) {
      // the pre-activation of every sequence's last token is what the backward pass differentiates at (layer.go:563-567)
      GN_TRY(gemm(ctx, g1));
      if (training) GN_LAUNCH(ctx, last_token_rows_kernel, ew_grid(ctx, (long)B * F), 256, 0, (const float*)l.mid.p, l.zlast.p, TE, F, (long)B * F);
      GN_LAUNCH(ctx, act_forward_kernel, ew_grid(ctx, nf), 256, 0, (const float*)l.mid.p, l.mid.p, nf, (int)GN_ACT_GELU, 0.f);
    } else {              // SwiGLU: gate and up projections (no biases)
      GN_TRY(gemm_nt_stack(ctx, 2, NE, F, D, l.n1.p, D, bp.w1, (long)F * D, nullptr, l.gate.p, l.up.p - l.gate.p, n1_planes ? &n1p : nullptr));
      GemmDesc c; c.M = NE; c.N = D; c.K = F; c.B = bp.w2; c.sb_k = 1; c.sb_n = F; c.sa_k = 1; c.sa_m = F;
      l.mid_is_planes = swiglu_planes_ok(l) && gemm_on_tc(ctx, c);
      if (l.mid_is_planes) SwigluRun<8>::fwd(ctx, l.gate.p, l.up.p, midp, l.mid_last.p, TE, NE, F);
      else GN_LAUNCH(ctx, swiglu_fwd_kernel, ew_grid(ctx, nf), 256, 0, (const float*)l.gate.p, (const float*)l.up.p, l.mid.p, nf);
    }
    GemmDesc g2; g2.M = NE; g2.N = D; g2.K = F; g2.A = l.mid.p; g2.sa_m = F; g2.sa_k = 1; g2.B = bp.w2; g2.sb_k = 1; g2.sb_n = F; g2.C = l.r2.p; g2.ldc = D; g2.bias = bp.b2; g2.R = l.n1.p; g2.ldr = D;
    if (l.mid_is_planes) g2.a_planes = &midp;
    GN_TRY(gemm(ctx, g2));
  }
  {   // norm 2 hands its output to the next block's projections as operand planes
    RowPlaneOut po2{}; BfPlanes outp{}; bool emitted = false;
    const bool next_is_block = !rows_only && li + 1 < m->L.size() && m->L[li + 1].d.kind == GN_LAYER_TRANSFORMER_BLOCK && m->L[li + 1].d.dim == D && m->L[li + 1].d.seq_len == T;
    if (next_is_block && norm_planes_wanted(ctx, NE, D, D)) GN_TRY(norm_planes_alloc(m, S_LNP1, S_LNI1, NE, D, &po2, &outp, nullptr));
    GN_TRY(norm_forward(ctx, l.rms, l.r2.p, bp.g2, bp.be2, l.out.p, st + 2 * NE, (long)NE, D, 1e-5f, po2.p ? &po2 : nullptr, &emitted));
    if (emitted) { m->fwd_planes = outp; m->fwd_planes_src = l.out.p; }
  }
  l.kept = training && l.keep.n != 0;
  if (l.kept) {
    const KeepRows k = keep_layout(l, B);
    GN_LAUNCH(ctx, keep_rows_kernel, B, 256, 0, (const float*)l.r2.p, (const float*)l.r1.p, (const float*)l.n1.p, (const float*)l.att.p, cur, l.mid_is_planes ? (const float*)nullptr : (const float*)l.mid.p,
              (const float*)l.gate.p, (const float*)l.up.p, (const float*)st, k, T, D, F, B);
  }
  *out = l.out.p; return GN_OK;
}

// A softmax or log-softmax head at the end of the model whose rows fit head_loss_kernel's registers.
static bool head_can_fuse(const gn_model* m) {
  const gn_layer_desc& d = m->L.back().d;
  return d.kind == GN_LAYER_DENSE && (d.activation == GN_ACT_SOFTMAX || d.activation == GN_ACT_LOGSOFTMAX) && d.out_size <= HEAD_MAX_CS * HEAD_THREADS * HEAD_MAX_E;
}
static int forward(gn_model* m, const float* x, int B, const float** y_out, bool training) {
  Ctx* ctx = &m->ctx->c;
  ctx->weight_planes = &m->wplanes;                  // (renewed by the first product of the pass that looks one up)
  m->head_fused = training && head_can_fuse(m);
  m->fwd_planes_src = nullptr;
  plan_token_rows(m, training);
  const float* cur = x;
  for (size_t li = 0; li < m->L.size(); li++) {
    LayerRT& l = m->L[li]; const gn_layer_desc& d = l.d; const float* p = m->params.p + l.p_off;
    l.fin = cur;
    switch (d.kind) {
      case GN_LAYER_DENSE: {
        const float* W = p; const float* bias = p + (long)d.in_size * d.out_size;
        if (d.activation == GN_ACT_LINEAR || d.activation == GN_ACT_RELU) {
          GN_TRY(gemm_nt(ctx, B, d.out_size, d.in_size, cur, d.in_size, W, bias, l.out.p, d.out_size, d.activation));
        } else {
          GN_TRY(gemm_nt(ctx, B, d.out_size, d.in_size, cur, d.in_size, W, bias, l.z.p, d.out_size));
          if (m->head_fused && li + 1 == m->L.size()) {}     // head_loss_kernel takes z
          else if (d.activation == GN_ACT_SOFTMAX || d.activation == GN_ACT_LOGSOFTMAX)
            GN_LAUNCH(ctx, softmax_rows_kernel, B, d.out_size >= 2048 ? 1024 : 256, 0, l.z.p, l.out.p, d.out_size, d.activation == GN_ACT_LOGSOFTMAX ? 1 : 0);
          else { long n = (long)B * d.out_size; GN_LAUNCH(ctx, act_forward_kernel, ew_grid(ctx, n), 256, 0, l.z.p, l.out.p, n, d.activation, act_alpha_of(d.activation, d.reserved)); }
        }
        cur = l.out.p; break; }
      case GN_LAYER_CONV2D: {
        ConvShape c{B, d.in_size, d.out_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        GN_TRY(conv_forward(ctx, c, d.activation, act_alpha_of(d.activation, d.reserved), cur, p, l.z.p, l.out.p, force_simt_engine() ? CONV_CUDA : CONV_AUTO));
        cur = l.out.p; break; }
      case GN_LAYER_MAXPOOL2D: {
        PoolShape c{B, d.in_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        GN_LAUNCH(ctx, maxpool_fwd_kernel, dim3(B * c.C, std::min(cdiv((long)c.oH * c.oW, 256), 65535u)), 256, 0, cur, l.out.p, (int*)l.idx.p, c);
        cur = l.out.p; break; }
      case GN_LAYER_CONV1D: {
        Conv1Shape c{B, d.in_size, d.out_size, d.kernel, d.stride, d.padding, d.in_w, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        long n = (long)B * l.out_size;
        GN_LAUNCH(ctx, conv1d_fwd_kernel, ew_grid(ctx, n), 256, 0, cur, p, p + (long)d.out_size * d.in_size * d.kernel, l.out.p, c, d.activation, act_alpha_of(d.activation, d.reserved));
        cur = l.out.p; break; }
      case GN_LAYER_DROPOUT:
        if (training) {
          const long tot = (long)B * l.in_size;
          GN_LAUNCH(ctx, dropout_fwd_kernel, ew_grid(ctx, cdiv(tot, DROP_RUN)), 256, 0, cur, l.out.p, l.z.p, (const float*)(m->state.p + l.s_off), tot, l.in_size, l.bn_mom,
                    (long)m->cur_first_sample * l.in_size);
          cur = l.out.p;
        }
        break;
      case GN_LAYER_AVGPOOL2D: {
        PoolShape c{B, d.in_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        long n = (long)B * l.out_size;
        GN_LAUNCH(ctx, avgpool_fwd_kernel, ew_grid(ctx, n), 256, 0, cur, l.out.p, c);
        cur = l.out.p; break; }
      case GN_LAYER_FLATTEN: break;
      case GN_LAYER_LSTM_UNROLLED: {
        const int H = d.out_size, in = d.in_size, T = d.seq_len;
        const size_t smem = ((size_t)H * H + (size_t)in * H + 2 * H + in) * sizeof(float);
        if (smem > 200 * 1024) return fail(GN_ERR_UNSUPPORTED, "LSTM of hidden size %d needs %zu bytes of shared memory", H, smem);
        // The input projection has no recurrence in it: Wx[0:H] x_t for all B*T rows is one contraction (only the first H of the
        // 4H gate rows receive it, lstm.go:319-326, :1065-1101); the kernel adds the bias and the recurrent product step by step.
        GN_TRY(gemm_nt(ctx, B * T, H, in, cur, in, p, nullptr, l.pre_i.p, H));
        GN_TRY(lstm_fwd(ctx, p + (long)4 * H * in, p + (long)4 * H * in + (long)4 * H * H, l.pre_i.p, l.c_all.p, l.z.p, l.h_all.p, l.out.p, RecShape{T, in, H, d.return_seq, B}));
        cur = l.out.p; break; }
      case GN_LAYER_GRU_UNROLLED: {
        const int H = d.out_size, in = d.in_size, T = d.seq_len, threads = ((H + 31) / 32) * 32;
        const float* Wx = p; const float* Wh = p + (long)3 * H * in; const float* bias = Wh + (long)2 * H * H;
        // input projection of all three gates and all B*T rows as one contraction (bias in its epilogue), then the recurrence
        GN_TRY(gemm_nt(ctx, B * T, 3 * H, in, cur, in, Wx, bias, l.pre_i.p, 3 * H));
        if (gru_reg_ok(H)) { GN_TRY(gru_fwd_reg(ctx, Wh, l.pre_i.p, l.h_all.p, l.out.p, RecShape{T, in, H, d.return_seq, B})); cur = l.out.p; break; }
        const size_t smem = ((size_t)2 * H * H + 3 * (size_t)H) * sizeof(float);
        GN_CUDA(cudaFuncSetAttribute(gru_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        GN_LAUNCH(ctx, gru_fwd_kernel, B, threads, smem, Wh, l.pre_i.p, l.h_all.p, l.out.p, T, H, d.return_seq);
        cur = l.out.p; break; }
      case GN_LAYER_EMBEDDING: {
        // fused with a directly following PositionalEncoding
        long tokens = (long)B * d.seq_len; const float* P = nullptr;
        bool fuse = li + 1 < m->L.size() && m->L[li + 1].d.kind == GN_LAYER_POSENC && m->L[li + 1].d.dim == d.out_size;
        if (fuse) P = m->params.p + m->L[li + 1].p_off;
        float* dst = fuse ? m->L[li + 1].out.p : l.out.p;
        l.out_rows = next_rows(m, fuse ? li + 1 : li, d.seq_len, d.out_size);
        if (norm_vec_ok(d.out_size, {p, P, dst})) {
          // a block that follows gets its projections' operand planes from here
          RowPlaneOut po{}; const size_t nx = fuse ? li + 2 : li + 1;
          if (!l.out_rows && nx < m->L.size() && m->L[nx].d.kind == GN_LAYER_TRANSFORMER_BLOCK && m->L[nx].d.dim == d.out_size && m->L[nx].d.seq_len == d.seq_len && norm_planes_wanted(ctx, (int)tokens, d.out_size, d.out_size)) {
            GN_TRY(norm_planes_alloc(m, S_LNP1, S_LNI1, (int)tokens, d.out_size, &po, &m->fwd_planes, nullptr)); m->fwd_planes_src = dst;
          }
          EmbedRun<8>::fwd(ctx, cur, p, P, dst, tokens, d.seq_len, d.out_size, d.in_size, (int*)l.idx.p, l.out_rows, po);
        } else
          GN_LAUNCH(ctx, embedding_fwd_kernel, (unsigned)tokens, 128, 0, cur, p, P, dst, tokens, d.seq_len, d.out_size, d.in_size, (int*)l.idx.p, ctx->d_status, l.out_rows);
        cur = dst; if (fuse) { m->L[li + 1].out_rows = l.out_rows; li++; } break; }
      case GN_LAYER_POSENC: {
        long n = (long)B * l.out_size; l.out_rows = 0;
        GN_LAUNCH(ctx, posenc_fwd_kernel, ew_grid(ctx, n), 256, 0, cur, p, l.out.p, n, (long)l.out_size);
        cur = l.out.p; break; }
      case GN_LAYER_TRANSFORMER_BLOCK: GN_TRY(block_forward(m, li, B, cur, training, &cur)); break;
      case GN_LAYER_CLS_POOLING: {
        const int rows = li > 0 && m->L[li - 1].d.kind == GN_LAYER_TRANSFORMER_BLOCK && m->L[li - 1].out_rows ? m->L[li - 1].out_rows : d.seq_len;
        GN_LAUNCH(ctx, cls_fwd_kernel, B, 128, 0, cur, l.out.p, rows, d.dim); cur = l.out.p; break; }
      case GN_LAYER_BATCHNORM2D: {
        const int C = d.in_size, S = d.in_h * d.in_w; const long BC = (long)B * C; float* run = m->state.p + l.s_off;
        if (training) {
          GN_LAUNCH(ctx, bn_fwd_kernel, (unsigned)BC, 256, 0, cur, p, p + C, l.out.p, l.stat.p, C, S, BC, l.bn_eps);
          if (ctx->world > 1) {
            // the running statistics move once per sample in batch order (batchnorm2d.go:352, :376): every rank gathers the
            // per-sample statistics of the whole global batch and walks them in that order, so the replicas stay identical
            const int GB = m->cur_global_batch;
            if (GB != B * ctx->world) return fail(GN_ERR_INVALID_ARG, "BatchNorm2D on %d ranks needs equal shards (global batch %d, this rank %d)", ctx->world, GB, B);
            float* g; GN_TRY(ensure(m, S_BNG, (size_t)2 * GB * C, &g));
            GN_TRY(all_gather_on_comm(m, l.stat.p, g, (size_t)BC, "BatchNorm2D means"));
            GN_TRY(all_gather_on_comm(m, l.stat.p + 2 * BC, g + (size_t)GB * C, (size_t)BC, "BatchNorm2D variances"));
            GN_LAUNCH(ctx, bn_running_kernel, cdiv(C, 32), 256, 0, (const float*)g, (const float*)(g + (size_t)GB * C), run, GB, C, l.bn_mom);
          } else GN_LAUNCH(ctx, bn_running_kernel, cdiv(C, 32), 256, 0, (const float*)l.stat.p, (const float*)(l.stat.p + 2 * BC), run, B, C, l.bn_mom);
        } else {
          long n = BC * S; GN_LAUNCH(ctx, bn_eval_kernel, ew_grid(ctx, n), 256, 0, cur, p, p + C, run, l.out.p, C, S, n, l.bn_eps);
        }
        cur = l.out.p; break; }
      case GN_LAYER_LAYERNORM: {
        long rows = (long)B * (l.in_size / d.dim);
        GN_TRY(norm_forward(ctx, false, cur, p, p + d.dim, l.out.p, l.stat.p, rows, d.dim, 1e-5f));
        cur = l.out.p; break; }
      case GN_LAYER_RMSNORM: {
        long rows = (long)B * (l.in_size / d.dim);
        GN_TRY(norm_forward(ctx, true, cur, p, nullptr, l.out.p, l.stat.p, rows, d.dim, l.bn_eps));
        cur = l.out.p; break; }
    }
    GN_TRY(check_launch("forward"));
  }
  *y_out = cur; return GN_OK;
}

// ---------------------------------------------------------------- backward
// Gradient of one inner Dense of a TransformerBlock at batch level:
//   gb = sum over all tokens of dz ; gW = Delta^T * X_last with Delta[s] = sum_t dz[s,t], X_last[s] = x[s,T-1]
// `x_last` != null: the last-token inputs as a dense [B, in] array instead of a strided view of x; `dz_planes` != null: dz
// exists only as operand planes.
// `stack` > 1: several layers with the same input, whose dz (and, `ws` apart, whose weight gradients) follow one another.
static int token_sums(Ctx* ctx, const float* dz, int n, int T, int out, float* delta) {      // n: sequences (of all layers of a stack)
  const bool vec = out % 4 == 0 && ((reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(delta)) & 15) == 0;
  for (int s0 = 0; s0 < n; s0 += 65535) {                   // (a grid's second dimension)
    const dim3 grid(cdiv(out, 128), std::min(n - s0, 65535)); const float* z = dz + (long)s0 * T * out; float* d = delta + (long)s0 * out;
    if (vec) GN_LAUNCH(ctx, token_sum_vec_kernel, grid, dim3(32, 8), 0, z, T, out, d);
    else GN_LAUNCH(ctx, token_sum_kernel, grid, dim3(128, 4), 0, z, T, out, d);
  }
  return check_launch("token_sums");
}
static int weight_bias_grads_stack(gn_model* m, int stack, int B, int out, int in, const float* delta, const float* x_last, long ldx, float* gW, float* gb, long ws) {
  Ctx* ctx = &m->ctx->c;
  GemmDesc g; g.M = out; g.N = in; g.K = B; g.A = delta; g.sa_m = 1; g.sa_k = out; g.B = x_last; g.sb_k = ldx; g.sb_n = 1; g.C = gW; g.ldc = in;
  g.batch1 = stack; g.a_b1 = (long)B * out; g.c_b1 = ws; g.a_sum = gb;
  if (gemm_outer_small_ok(g)) return gemm(ctx, g);
  for (int j = 0; j < stack; j++) GN_TRY(weight_bias_grads(m, ctx, B, out, in, delta + (long)j * B * out, out, x_last, ldx, gW + j * ws, gb + j * ws));
  return GN_OK;
}
static int inner_dense_param_grads(gn_model* m, const float* dz, int B, int T, int out, const float* x, int in, float* gW, float* gb,
                                   const float* x_last = nullptr, const BfPlanes* dz_planes = nullptr, const float* dz_rowsum32 = nullptr, int stack = 1, long ws = 0) {
  Ctx* ctx = &m->ctx->c; const bool side = grads_on_side(ctx, stack, B, out, in, in); float* delta;
  GN_TRY(ensure(m, side ? S_SIDE : S_DELTA, (size_t)stack * B * out, &delta));
  auto issue = [&]() -> int {
    if (dz_rowsum32) GN_LAUNCH(ctx, token_sum_part32_kernel, dim3(cdiv(out, 512), B), 128, 0, dz_rowsum32, T / 32, out, delta);
    else if (dz_planes) GN_LAUNCH(ctx, token_sum_planes_kernel, dim3(cdiv(out, 128), B), dim3(32, 8), 0, (const __half*)dz_planes->base, (const float*)dz_planes->inv_scale, (long)dz_planes->ldp, T, out, delta);
    else GN_TRY(token_sums(ctx, dz, stack * B, T, out, delta));
    return x_last ? weight_bias_grads_stack(m, stack, B, out, in, delta, x_last, (long)in, gW, gb, ws)
                  : weight_bias_grads_stack(m, stack, B, out, in, delta, x + (long)(T - 1) * in, (long)T * in, gW, gb, ws);
  };
  return side ? side_run(ctx, issue) : issue();
}
// The gradients of a layer from dense rows of dz, beside the main stream where that is possible.
static int side_weight_bias_grads(gn_model* m, int stack, int B, int out, int in, const float* dz, const float* x, long ldx, float* gW, float* gb, long ws = 0) {
  Ctx* ctx = &m->ctx->c; auto issue = [&]() -> int { return weight_bias_grads_stack(m, stack, B, out, in, dz, x, ldx, gW, gb, ws); };
  return grads_on_side(ctx, stack, B, out, in, ldx) ? side_run(ctx, issue) : issue();
}
// The parameter gradients of up to four layers from dense rows of dz, in one launch where they are sums of few outer products; others go one by one when they are
// added.  `chain`: what follows on the main stream are more links of small products (a causal block's token rows), and the launch runs beside them.  Else products over
// all tokens follow, whose blocks want whole SMs: large gradients go beside the main stream at once, one by one, and the launch for the small ones is a link of it.
// (Training steps, us, one launch beside the main stream -> this: 33 x 432 tokens, 512 wide, one block 499 -> 478, 36 x 71, 768 wide, seven 5584 -> 5553.)
struct GradGroup {
  gn_model* m; bool chain; GemmDesc d[4]; int n = 0;
  int add(int B, int out, int in, const float* dz, const float* x, long ldx, float* gW, float* gb) {
    GemmDesc g; g.M = out; g.N = in; g.K = B; g.A = dz; g.sa_m = 1; g.sa_k = out; g.B = x; g.sb_k = ldx; g.sb_n = 1; g.C = gW; g.ldc = in; g.a_sum = gb;
    if (m->ctx->c.profile || !gemm_outer_small_ok(g) || n == 4 || (!chain && grads_on_side(&m->ctx->c, 1, B, out, in, ldx))) return side_weight_bias_grads(m, 1, B, out, in, dz, x, ldx, gW, gb);
    d[n++] = g; return GN_OK;
  }
  int flush() {
    if (!n) return GN_OK;
    Ctx* ctx = &m->ctx->c; double macs = 0; for (int j = 0; j < n; j++) macs += (double)d[j].M * d[j].N * d[j].K;
    ctx->gemm_flops += 2.0 * macs; ctx->gemm_launches++;
    auto issue = [&]() -> int { return gemm_outer_group(ctx, d, n); };
    const int rc = chain && macs >= 3.0e6 ? side_run(ctx, issue) : issue(); n = 0; return rc;
  }
};
// Can the FFN's hidden activation (and its gradient) of this block live as operand planes only?  The two contractions on
// either side must both run on the tensor-core engine with prepared weight planes, and the plane-writing epilogue's shape
// rules must hold.
static bool ffn_planes_possible(Ctx* ctx, const LayerRT& l, int N, const float* w1, const float* w2) {
  static const bool off = getenv("GONEURON_CUDA_NO_PLANE_OUTPUT") != nullptr;
  const gn_layer_desc& d = l.d; const int D = d.dim, F = d.ff_dim;
  if (off || force_simt_engine() || (l.ff_act != GN_ACT_RELU && l.ff_act != GN_ACT_GELU) || F % 32 || D % 32 || D > 2048 || F % 4) return false;
  if ((reinterpret_cast<uintptr_t>(w1 + (long)D * F) & 15) != 0) return false;                                 // ff1's bias is read with 16-byte loads
  BfPlanes w; GemmDesc a; a.M = N; a.N = F; a.K = D; a.B = w1; a.sb_k = 1; a.sb_n = D; a.sa_k = 1; a.sa_m = D;            // n1 W1^T        -> planes
  GemmDesc b; b.M = N; b.N = F; b.K = D; b.B = w2; b.sb_k = F; b.sb_n = 1; b.sa_k = 1; b.sa_m = D;            // dR2 W2         -> planes
  GemmDesc c; c.M = N; c.N = D; c.K = F; c.B = w2; c.sb_k = 1; c.sb_n = F; c.sa_k = 1; c.sa_m = F;            // planes W2^T    (consumer, forward)
  GemmDesc e; e.M = N; e.N = D; e.K = F; e.B = w1; e.sb_k = D; e.sb_n = 1; e.sa_k = 1; e.sa_m = F;            // planes W1      (consumer, backward)
  return gemm_tc_eligible(ctx, a) && gemm_tc_eligible(ctx, b) && gemm_tc_eligible(ctx, c) && gemm_tc_eligible(ctx, e) && wplanes_lookup(ctx, a, &w) && wplanes_lookup(ctx, b, &w);
}

static int block_backward(gn_model* m, LayerRT& l, int B, const float* xin, const float* gout, float* dx) {
  Ctx* ctx = &m->ctx->c; const gn_layer_desc& d = l.d;
  const int T = d.seq_len, D = d.dim, F = d.ff_dim, Hh = d.heads, hd = D / Hh; const int N = B * T; const long ND = (long)N * D;
  BlockParams bp = block_params(m->params.p + l.p_off, D, F, l.rms, l.ff_act); BlockParams gp = block_params(m->grads.p + l.p_off, D, F, l.rms, l.ff_act);
  float *dR2, *dM, *comb, *dR1, *dA, *P = nullptr, *dP = nullptr; float* st = l.stat.p;
  const bool fused = use_fused_attention(d);
  GN_TRY(ensure(m, S_ND0, ND, &dR2)); GN_TRY(ensure(m, S_NFF, (size_t)N * F, &dM)); GN_TRY(ensure(m, S_ND1, ND, &comb));
  GN_TRY(ensure(m, S_ND2, ND, &dR1)); GN_TRY(ensure(m, S_ND3, ND, &dA));
  const bool side = grads_on_side(ctx, 1, B, F, D, D);      // (the block forks its stream anyway)
  if (!fused) { GN_TRY(ensure(m, S_ATT0, (size_t)B * Hh * T * T, &P)); GN_TRY(ensure(m, S_ATT1, (size_t)B * Hh * T * T, &dP)); }
  // norm 2
  // its result goes to the contraction with W2 as operand planes, with the row norms that contraction's plane-writing epilogue needs
  RowPlaneOut pob{}; BfPlanes dR2p{}; bool dR2_planes = false; float* rnb = nullptr;
  if (norm_planes_wanted(ctx, N, D, F)) { GN_TRY(ensure(m, S_RN, (size_t)N, &rnb)); GN_TRY(norm_planes_alloc(m, S_LNP0, S_LNI0, N, D, &pob, &dR2p, rnb)); }
  GN_TRY(norm_backward(m, l.rms, gout, l.r2.p, bp.g2, st + 2 * N, dR2, (float*)gp.g2, (float*)gp.be2, (long)N, D, pob.p ? &pob : nullptr, &dR2_planes, side ? S_PART2 : 0));
  // ff2 then ff1, token by token in the reference (transformer.go:1238-1250)
  GN_TRY(inner_dense_param_grads(m, dR2, B, T, D, l.mid.p, F, (float*)gp.w2, (float*)gp.b2, l.mid_is_planes ? l.mid_last.p : nullptr));
  {
    // dM[s,t,:] = W2^T dR2[s,t,:]; with a ReLU first layer gated by the ReLU pattern of the LAST token of sequence s (fused into the epilogue)
    GemmDesc g; g.M = N; g.N = F; g.K = D; g.A = dR2; g.sa_m = D; g.sa_k = 1; g.B = bp.w2; g.sb_k = F; g.sb_n = 1; g.C = dM; g.ldc = F;
    if (dR2_planes) g.a_planes = &dR2p;
    const bool ffn_planes = l.mid_is_planes && l.ff_act != GN_ACT_SILU;
    if (ffn_planes) {
      g.mask = l.mid_last.p; g.mask_ld = F; g.mask_group = T;
      if (l.ff_act == GN_ACT_GELU) {      // GELU'(z) of the last token multiplies every token's gradient (layer.go:563-567): factors instead of a gate
        float* der; GN_TRY(ensure(m, S_NFF2, (size_t)B * F, &der));
        GN_LAUNCH(ctx, act_deriv_kernel, ew_grid(ctx, (long)B * F), 256, 0, (const float*)l.zlast.p, der, (long)B * F, (int)GN_ACT_GELU); g.mask = der;
      }
    }
    else if (l.ff_act == GN_ACT_RELU) { g.mask = l.mid.p + (long)(T - 1) * F; g.mask_ld = (long)T * F; g.mask_group = T; }
    const long nf = (long)N * F;
    if (ffn_planes) {
      // the gradient of the hidden activation likewise only feeds a token sum and the next contraction: planes only
      const WeightPlaneEntry* we = nullptr; BfPlanes w; wplanes_lookup(ctx, g, &w, &we);
      float *rn, *dinv; GN_TRY(ensure(m, S_RN, (size_t)N, &rn)); GN_TRY(ensure(m, S_NFFI, (size_t)N, &dinv));
      BfPlanes dMp{reinterpret_cast<__half*>(dM), dinv, N, F, F, 1};
      TcPlaneOut po{dMp, we->maxabs, nullptr, 1}; po.scale = l.ff_act == GN_ACT_GELU;
      float* rs32 = nullptr;                               // 32-row sums of dM from the epilogue: the token sums of the ff1 weight gradient
      if (T % 32 == 0 && F % 4 == 0) { GN_TRY(ensure(m, S_RS32, (size_t)(N / 32) * F, &rs32)); po.rowsum32 = rs32; }
      g.C = nullptr; g.plane_out = &po; g.a_rownorm = rn; GN_TRY(gemm(ctx, g));
      GemmDesc h; h.M = N; h.N = D; h.K = F; h.A = dM; h.sa_m = F; h.sa_k = 1; h.B = bp.w1; h.sb_k = D; h.sb_n = 1; h.C = comb; h.ldc = D; h.R = dR2; h.ldr = D; h.a_planes = &dMp;
      GN_TRY(inner_dense_param_grads(m, nullptr, B, T, F, l.n1.p, D, (float*)gp.w1, (float*)gp.b1, nullptr, &dMp, rs32));
      GN_TRY(gemm(ctx, h));
    } else if (l.ff_act != GN_ACT_SILU) {
      GN_TRY(gemm(ctx, g));
      if (l.ff_act == GN_ACT_GELU) GN_LAUNCH(ctx, scale_by_last_deriv_kernel, ew_grid(ctx, nf), 256, 0, dM, (const float*)l.zlast.p, T, F, nf, (int)GN_ACT_GELU);
      GemmDesc h; h.M = N; h.N = D; h.K = F; h.A = dM; h.sa_m = F; h.sa_k = 1; h.B = bp.w1; h.sb_k = D; h.sb_n = 1; h.C = comb; h.ldc = D; h.R = dR2; h.ldr = D;   // combined = gradRes2 + W1^T dz1
      GN_TRY(inner_dense_param_grads(m, dM, B, T, F, l.n1.p, D, (float*)gp.w1, (float*)gp.b1));
      GN_TRY(gemm(ctx, h));
    } else {
      GN_TRY(gemm(ctx, g));
      // SwiGLU keeps every call's state and pops it in reverse (swiglu.go:186-201): token t's gradient meets token T-1-t's
      // input and projections.  The deltas are written at the partner's row, so the weight gradients are plain contractions
      // over all tokens with the layer's inputs; the input gradient comes out in partner order and is reversed when it is
      // added to the residual path.
      float *dGP, *dUP, *Y;
      GN_TRY(ensure(m, S_NFF2, (size_t)2 * nf, &dGP)); dUP = dGP + nf; GN_TRY(ensure(m, S_ND3, ND, &Y));
      BfPlanes dp{}; bool planes = false;
      if (swiglu_planes_ok(l)) {
        GemmDesc q; q.M = N; q.N = D; q.K = 2 * F; q.B = bp.w1; q.sb_k = D; q.sb_n = 1; q.sa_k = 1; q.sa_m = F; BfPlanes w;
        planes = gemm_on_tc(ctx, q) && wplanes_lookup(ctx, q, &w);
      }
      if (planes) {
        float *pp, *pi; GN_TRY(ensure(m, S_NFF3, (size_t)2 * nf, &pp)); GN_TRY(ensure(m, S_NFFI, (size_t)N, &pi));
        dp = BfPlanes{reinterpret_cast<__half*>(pp), pi, N, 2 * F, 2 * F, 1};
        SwigluRun<8>::bwd(ctx, dM, l.gate.p, l.up.p, dGP, dUP, dp, T, N, F);
      } else GN_LAUNCH(ctx, swiglu_bwd_paired_kernel, ew_grid(ctx, nf), 256, 0, (const float*)dM, (const float*)l.gate.p, (const float*)l.up.p, dGP, dUP, T, F, nf);
      GN_TRY(gemm_tn_stack(ctx, 2, N, F, D, dGP, nf, l.n1.p, D, (float*)gp.w1));
      GN_TRY(gemm_nn_stack(ctx, 2, N, F, D, dGP, nf, bp.w1, (long)F * D, Y, nullptr, planes ? &dp : nullptr));
      GN_LAUNCH(ctx, add_token_reversed_kernel, ew_grid(ctx, ND), 256, 0, (const float*)dR2, (const float*)Y, comb, T, D, ND);
    }
  }
  // norm 1
  RowPlaneOut poa{}; BfPlanes dR1p{}; bool dR1_planes = false;
  if (norm_planes_wanted(ctx, N, D, D)) GN_TRY(norm_planes_alloc(m, S_LNP0, S_LNI0, N, D, &poa, &dR1p, nullptr));      // the planes of dR2 are dead by now
  GN_TRY(norm_backward(m, l.rms, comb, l.r1.p, bp.g1, st, dR1, (float*)gp.g1, (float*)gp.be1, (long)N, D, poa.p ? &poa : nullptr, &dR1_planes, side ? S_PART3 : 0));
  // output projection
  GN_TRY(inner_dense_param_grads(m, dR1, B, T, D, l.att.p, D, (float*)gp.wo, (float*)gp.bo));
  {
    GemmDesc g; g.M = N; g.N = D; g.K = D; g.A = dR1; g.sa_m = D; g.sa_k = 1; g.B = bp.wo; g.sb_k = D; g.sb_n = 1; g.C = dA; g.ldc = D;      // dA = dR1 Wo
    if (dR1_planes) g.a_planes = &dR1p;
    GN_TRY(gemm(ctx, g));
  }
  // attention: recompute P (transformer.go:610-622), then dP, dS, dQ, dK, dV
  float *dQ; GN_TRY(ensure(m, S_ND4, 3 * ND, &dQ)); float *dK = dQ + ND, *dV = dK + ND;
  if (fused) {
    static const bool tc_bwd = [] { const char* e = getenv("GONEURON_CUDA_ATTENTION_BWD"); return !(e && !strcmp(e, "mma")); }();
    if (tc_bwd && attn_tc_supported(ctx, hd, T, B, Hh, D)) GN_TRY(attn_tc_bwd(ctx, l.q.p, l.k.p, l.v.p, l.att.p, dA, l.att_m.p, l.att_l.p, l.att_d.p, dQ, dK, dV, B, T, D, Hh, d.causal, &l.attn_saved));
    else GN_TRY(attn_bwd(ctx, hd, l.q.p, l.k.p, l.v.p, l.att.p, dA, l.att_m.p, l.att_l.p, dQ, dK, dV, B, T, D, Hh, d.causal));
  } else {
    const long TD = (long)T * D, TT = (long)T * T; const float inv_scale = 1.f / sqrtf((float)hd); const long rows = (long)B * Hh * T;
    GemmDesc g; g.M = T; g.N = T; g.K = hd; g.A = l.q.p; g.sa_m = D; g.sa_k = 1; g.B = l.k.p; g.sb_k = 1; g.sb_n = D;
    g.C = P; g.ldc = T; g.batch1 = B; g.batch2 = Hh; g.a_b1 = TD; g.a_b2 = hd; g.b_b1 = TD; g.b_b2 = hd; g.c_b1 = Hh * TT; g.c_b2 = TT;
    g.flags = d.causal ? GEMM_SKIP_UPPER : 0; GN_TRY(gemm(ctx, g));
    GN_LAUNCH(ctx, attn_softmax_kernel, cdiv(rows, 8), 256, 0, P, T, inv_scale, d.causal, rows);
    g.A = dA; g.B = l.v.p; g.C = dP; GN_TRY(gemm(ctx, g));                               // dP = dA V^T
    GN_LAUNCH(ctx, attn_ds_kernel, cdiv(rows, 8), 256, 0, P, dP, T, inv_scale, d.causal, rows);   // dP <- dS (scaled)
    GemmDesc q; q.M = T; q.N = hd; q.K = T; q.batch1 = B; q.batch2 = Hh; q.a_b1 = Hh * TT; q.a_b2 = TT; q.b_b1 = TD; q.b_b2 = hd; q.c_b1 = TD; q.c_b2 = hd; q.ldc = D;
    q.sb_k = D; q.sb_n = 1;
    q.A = dP; q.sa_m = T; q.sa_k = 1; q.B = l.k.p; q.C = dQ; q.flags = d.causal ? GEMM_KEND_AT_M0 : 0; GN_TRY(gemm(ctx, q));     // dQ = dS K
    q.A = dP; q.sa_m = 1; q.sa_k = T; q.B = l.q.p; q.C = dK; q.flags = d.causal ? GEMM_KBEG_AT_M0 : 0; GN_TRY(gemm(ctx, q));     // dK = dS^T Q
    q.A = P; q.B = dA; q.C = dV; GN_TRY(gemm(ctx, q));                                                                          // dV = P^T dA
  }
  if (l.use_rope) {   // the conjugate rotation on the gradients of q and k (transformer.go:659-663)
    rope(ctx, l, dQ, dK, N, T, -1.f, 1);
  }
  // q, k, v projections; gradIn = dq + dk + dv, block input gradient = gradRes1 + gradIn
  GN_TRY(inner_dense_param_grads(m, dQ, B, T, D, xin, D, (float*)gp.wq, (float*)gp.bq, nullptr, nullptr, nullptr, 3, (long)D * D + D));
  GN_TRY(gemm_nn_stack(ctx, 3, N, D, D, dQ, ND, bp.wq, (long)D * D + D, dx, dR1));
  return check_launch("block_backward");
}

// Backward pass of a block whose output gradient is zero except at token 0 (plan_token_rows): gout is [B, D], and so is everything
// up to the attention.  The inner layers' other factor is the last token's activation, as always.  dx: [B, D] for a causal
// block (*dx_row0 = true), else [B * T, D].
static int block_backward_row0(gn_model* m, LayerRT& l, int B, const float* xin, const float* gout, float* dx, bool* dx_row0) {
  Ctx* ctx = &m->ctx->c; const gn_layer_desc& d = l.d;
  const int T = d.seq_len, D = d.dim, F = d.ff_dim, TE = l.out_rows ? l.out_rows : T; const long ND = (long)B * T * D, BD = (long)B * D, BF = (long)B * F;
  const BlockParams bp = block_params(m->params.p + l.p_off, D, F, l.rms, l.ff_act); const BlockParams gp = block_params(m->grads.p + l.p_off, D, F, l.rms, l.ff_act);
  // token 0's row of the norms' inputs (and statistics), the last token's rows of the rest; rows of consecutive sequences are ldD (ldF, ldX) apart
  const KeepRows kr = keep_layout(l, B); const int TR = l.kept ? 1 : TE;
  const long ldD = (long)TR * D, ldF = (long)TR * F, NE = (long)B * TR, ldX = l.kept ? D : (long)T * D; const float* st = l.kept ? kr.st : l.stat.p;
  auto last = [&](const DevBuf& b, const float* k, long w) -> const float* { return l.kept ? k : b.p + (long)(TE - 1) * w; };
  const float* r2_0 = l.kept ? kr.r2 : l.r2.p; const float* r1_0 = l.kept ? kr.r1 : l.r1.p;
  const float* n1_last = last(l.n1, kr.n1, D); const float* att_last = last(l.att, kr.att, D); const float* x_last = l.kept ? kr.x : xin + (long)(T - 1) * D;
  const float* gate_last = last(l.gate, kr.gate, F); const float* up_last = last(l.up, kr.up, F);
  const float* mid_last = l.mid_is_planes ? l.mid_last.p : last(l.mid, kr.mid, F); const long ld_mid = l.mid_is_planes ? F : ldF;
  float *dR2, *dR1, *comb, *dA, *dM;
  GN_TRY(ensure(m, S_ND0, BD, &dR2)); GN_TRY(ensure(m, S_ND1, BD, &comb)); GN_TRY(ensure(m, S_ND2, BD, &dR1)); GN_TRY(ensure(m, S_ND3, 2 * BD, &dA)); GN_TRY(ensure(m, S_NFF, BF, &dM));
  const bool side = grads_on_side(ctx, 1, B, F, D, D);      // (the block forks its stream anyway)
  auto norm = [&](const float* g, const float* x, const float* gamma, const float* stat, float* out, float* gG, float* gB, int slot) -> int {
    if (norm_vec_ok(D, {g, x, gamma, out})) return norm_backward_vec(m, l.rms, g, x, ldD, gamma, stat, l.rms ? stat : stat + NE, TR, out, gG, gB, B, D, RowPlaneOut{}, side ? slot : 0);
    GN_LAUNCH(ctx, norm_bwd_rows_kernel, cdiv(B, 4), 128, 0, g, x, ldD, gamma, stat, l.rms ? nullptr : stat + NE, (long)TR, out, B, D);
    GN_LAUNCH(ctx, norm_pgrad_rows_kernel, cdiv(D, 32), 256, 0, g, x, ldD, stat, l.rms ? nullptr : stat + NE, (long)TR, B, D, gG, gB);
    return check_launch("norm_rows");
  };
  GN_TRY(norm(gout, r2_0, bp.g2, st + 2 * NE, dR2, (float*)gp.g2, (float*)gp.be2, S_PART2));
  GradGroup grads{m, d.causal != 0};
  GN_TRY(grads.add(B, D, F, dR2, mid_last, ld_mid, (float*)gp.w2, (float*)gp.b2));
  GemmDesc g; g.M = B; g.N = F; g.K = D; g.A = dR2; g.sa_m = D; g.sa_k = 1; g.B = bp.w2; g.sb_k = F; g.sb_n = 1; g.C = dM; g.ldc = F;
  if (l.ff_act == GN_ACT_RELU) { g.mask = mid_last; g.mask_ld = ld_mid; }
  GN_TRY(gemm(ctx, g));
  if (l.ff_act == GN_ACT_SILU) {
    float *dG, *dU; GN_TRY(ensure(m, S_NFF2, BF, &dG)); GN_TRY(ensure(m, S_NFF3, BF, &dU));
    GN_LAUNCH(ctx, swiglu_bwd_rows_kernel, ew_grid(ctx, BF), 256, 0, (const float*)dM, gate_last, up_last, ldF, dG, dU, F, BF);
    GN_TRY(gemm_tn(ctx, B, F, D, dG, F, n1_last, ldD, (float*)gp.w1));
    GN_TRY(gemm_tn(ctx, B, F, D, dU, F, n1_last, ldD, (float*)gp.v1));
    GN_TRY(gemm_nn(ctx, B, F, D, dG, F, bp.w1, comb, D, dR2, D));
    GN_TRY(gemm_nn(ctx, B, F, D, dU, F, bp.v1, comb, D, comb, D));
  } else {
    if (l.ff_act == GN_ACT_GELU) GN_LAUNCH(ctx, scale_by_last_deriv_kernel, ew_grid(ctx, BF), 256, 0, dM, (const float*)l.zlast.p, 1, F, BF, (int)GN_ACT_GELU);
    GN_TRY(grads.add(B, F, D, dM, n1_last, ldD, (float*)gp.w1, (float*)gp.b1));
    GN_TRY(gemm_nn(ctx, B, F, D, dM, F, bp.w1, comb, D, dR2, D));
  }
  GN_TRY(norm(comb, r1_0, bp.g1, st, dR1, (float*)gp.g1, (float*)gp.be1, S_PART3));
  GN_TRY(grads.add(B, D, D, dR1, att_last, ldD, (float*)gp.wo, (float*)gp.bo));
  GN_TRY(gemm_nn(ctx, B, D, D, dR1, D, bp.wo, dA, D));
  if (d.causal) {
    // the one probability of token 0 is 1: dV = dA at token 0, dQ = dK = 0
    GN_TRY(side_run(ctx, [&]() -> int { GN_CUDA(stream_zero(ctx, (void*)gp.wq, (size_t)(gp.wv - gp.wq) * sizeof(float))); return GN_OK; }));
    GN_TRY(grads.add(B, D, D, dA, x_last, ldX, (float*)gp.wv, (float*)gp.bv));
    GN_TRY(grads.flush());
    GN_TRY(gemm_nn(ctx, B, D, D, dA, D, bp.wv, dx, D, dR1, D));
    *dx_row0 = true; return check_launch("block_backward_row0");
  }
  GN_TRY(grads.flush());
  float *dQ, *dK, *dV, *ks, *vs;
  GN_TRY(ensure(m, S_XROWS, 3 * BD, &dQ)); ks = dQ + BD; vs = ks + BD; GN_TRY(ensure(m, S_ND4, 2 * ND, &dK)); dV = dK + ND;
  GN_TRY(attn_rows_bwd(ctx, l.q.p, (long)TE * D, l.k.p, l.v.p, dA, dQ, dK, dV, ks, vs, B, T, D, d.heads));
  if (l.use_rope) {   // the conjugate rotation (transformer.go:659-663); token 0's angle is zero
    rope(ctx, l, dK, nullptr, B * T, T, -1.f, 1);
    GN_LAUNCH(ctx, token_sum_kernel, dim3(cdiv(D, 128), B), dim3(128, 4), 0, (const float*)dK, T, D, ks);
  }
  GN_TRY(side_weight_bias_grads(m, 3, B, D, D, dQ, x_last, ldX, (float*)gp.wq, (float*)gp.bq, (long)D * D + D));      // dQ | sum of dK | sum of dV
  float* dxq; GN_TRY(ensure(m, S_ND3, 2 * BD, &dxq)); dxq += BD;                           // (behind dA; dR1 may still be read on the side stream)
  GN_TRY(gemm_nn(ctx, B, D, D, dQ, D, bp.wq, dxq, D, dR1, D));
  GN_TRY(gemm_nn_stack(ctx, 2, B * T, D, D, dK, ND, bp.wk, (long)D * D + D, dx, nullptr));
  GN_LAUNCH(ctx, add_row0_kernel, B, 128, 0, (const float*)dxq, dx, T, D);
  *dx_row0 = false; return check_launch("block_backward_row0");
}

static int lstm_backward(gn_model* m, LayerRT& l, size_t li, int B, const float* xin, const float* gout, int global_batch, int first_sample, float* dx) {
  Ctx* ctx = &m->ctx->c; const gn_layer_desc& d = l.d; const int H = d.out_size, in = d.in_size, T = d.seq_len;
  const float* p = m->params.p + l.p_off; const float* Wx = p; const float* Wh = p + (long)4 * H * in; const float* bias = Wh + (long)4 * H * H;
  GN_TRY(lstm_bwd(ctx, gout, Wh, bias, l.pre_i.p, l.c_all.p, l.z.p, l.dgate.p, RecShape{T, in, H, d.return_seq, B}));
  if (li > 0) GN_TRY(gemm_nn(ctx, B * T, 4 * H, in, l.dgate.p, 4 * H, Wx, dx, in));   // dx_t = Wx^T d_t
  // The clipping recurrence (lstm.go:694, :725-751) walks the rank-1 updates d_k z_k^T of a whole worker chunk in sample
  // order, and a chunk may span ranks.  With more than one rank every rank therefore gathers the update factors of the
  // whole global batch (rows in global sample order, all-gather over NVLink) and runs the identical scan over all chunks:
  // each replica ends up with the complete LSTM gradient, and this layer's slice is not all-reduced.
  const int world = ctx->world; const int GB = world > 1 ? global_batch : B; const int row0 = world > 1 ? first_sample : 0;
  if (world > 1 && GB != B * world) return fail(GN_ERR_INVALID_ARG, "LSTM on %d ranks needs equal shards (global batch %d, this rank %d)", world, GB, B);
  l.grad_replicated = world > 1;
  int chunk = (global_batch + m->W - 1) / m->W, nchunks = (GB + chunk - 1) / chunk;
  {
    // The walk over scalars (recurrent.cuh) is the default; GONEURON_CUDA_LSTM_SCAN=cluster asks for the kernel below, which
    // applies the updates one by one to the matrix and otherwise runs only for chunks that are too long.
    static const bool on_matrix = [] { const char* e = getenv("GONEURON_CUDA_LSTM_SCAN"); return e && strcmp(e, "cluster") == 0; }();
    const int R4g = 4 * H, ZWg = in + H + 1, zs = clip_zs(ZWg), slabs = cdiv(R4g, 8);
    const long Kc = (long)chunk * T, n_updates = (long)GB * T, n_local = (long)B * T, groups = (Kc + CG - 1) / CG, ng = (long)nchunks * groups;
    const UpdateRows u = update_rows_of_chunks(n_updates, Kc, nchunks, CG, CG_PAD); const long stride = u.stride, rows = u.rows;
    const bool fits = Kc <= CG_MAX_K && ng <= 65535;
    if (world > 1 && (on_matrix || !fits)) return fail(GN_ERR_UNSUPPORTED, "LSTM on more than one GPU needs the scalar form of the clipping recurrence (worker chunk of %ld updates)", Kc);
    if (!on_matrix && fits) {
      float *G0, *G1, *Dm, *Zm, *dbl, *gmat;
      const size_t n_om = (size_t)ng * CG, n_p = (size_t)nchunks * 2 * CG * slabs;
      GN_TRY(ensure(m, S_GRAM0, (size_t)ng * CG * 2 * CG, &G0)); GN_TRY(ensure(m, S_GRAM1, (size_t)ng * CG * 2 * CG, &G1));
      GN_TRY(ensure(m, S_DM, (size_t)rows * R4g, &Dm)); GN_TRY(ensure(m, S_ZM, (size_t)rows * zs, &Zm));
      GN_TRY(ensure(m, S_TV, 2 * (n_om + n_p + (size_t)ng * 2) + nchunks + n_updates, &dbl)); GN_TRY(ensure(m, S_SCAN, (size_t)nchunks * 2 * R4g * ZWg, &gmat));
      double* db = reinterpret_cast<double*>(dbl); int* start = reinterpret_cast<int*>(db + n_om + n_p + (size_t)ng * 2); float* un = reinterpret_cast<float*>(start + nchunks);
      // One group is always walked.  With more, the search for the first one costs 2 to 5 us (steps of 512 and 4096 updates of which nothing can be left
      // out take 149 instead of 147 and 590 instead of 588), and every group that is left out saves 4 to 13.
      // Few updates are all gathered and their norms come with that; of more the norms come first, so that most need not be
      // gathered (at 32 groups both ways take 300 us, and 595 where nothing can be left out and the norms come first).
      const bool late = groups > 1, few = ng <= CLIP_FEW;
      if (world > 1) {
        // rows of zeros: the group before every chunk's first, and what its last group lacks
        if (nchunks > 8) { GN_CUDA(stream_zero(ctx, Dm, (size_t)rows * R4g * 4)); GN_CUDA(stream_zero(ctx, Zm, (size_t)rows * zs * 4)); }
        else for (int c = 0; c < nchunks; c++) {
          const long n = std::min(Kc, n_updates - c * Kc), r0 = c * stride, r1 = r0 + CG_PAD + n, left = stride - CG_PAD - n;
          GN_CUDA(stream_zero(ctx, Dm + r0 * R4g, (size_t)CG_PAD * R4g * 4)); GN_CUDA(stream_zero(ctx, Zm + r0 * zs, (size_t)CG_PAD * zs * 4));
          if (left > 0) { GN_CUDA(stream_zero(ctx, Dm + r1 * R4g, (size_t)left * R4g * 4)); GN_CUDA(stream_zero(ctx, Zm + r1 * zs, (size_t)left * zs * 4)); }
        }
        float* all; GN_TRY(ensure(m, S_W, (size_t)n_updates * (R4g + zs), &all));
        float* Da = all; float* Za = all + (size_t)n_updates * R4g; float* Dl = Da + (size_t)row0 * T * R4g; float* Zl = Za + (size_t)row0 * T * zs;      // this rank's rows
        GN_LAUNCH(ctx, lstm_gather_updates_kernel, cdiv(n_local, 8), 256, 0, (const float*)l.dgate.p, xin, (const float*)l.h_all.p, Dl, Zl, T, in, H, zs, update_rows_of_rank(n_local), (const int*)nullptr, (float*)nullptr);
        GN_TRY(all_gather_on_comm(m, Dl, Da, (size_t)n_local * R4g, "LSTM update factors D"));
        GN_TRY(all_gather_on_comm(m, Zl, Za, (size_t)n_local * zs, "LSTM update factors Z"));
        GN_LAUNCH(ctx, lstm_place_rows_kernel, (unsigned)n_updates, 128, 0, (const float*)Da, Dm, R4g, u);
        GN_LAUNCH(ctx, lstm_place_rows_kernel, (unsigned)n_updates, 128, 0, (const float*)Za, Zm, zs, u);
        if (late) GN_LAUNCH(ctx, lstm_row_norms_kernel, cdiv(n_updates, 8), 256, 0, (const float*)Dm, (const float*)Zm, un, R4g, zs, u);
      }
      auto gather = [&](const int* from, float* norms) {
        GN_LAUNCH(ctx, lstm_gather_updates_kernel, cdiv(rows, 8), 256, 0, (const float*)l.dgate.p, xin, (const float*)l.h_all.p, Dm, Zm, T, in, H, zs, u, from, norms);
      };
      if (world == 1 && (!late || few)) gather(nullptr, late ? un : nullptr);
      else if (world == 1) GN_LAUNCH(ctx, lstm_update_norms_kernel, cdiv(n_updates, 8), 256, 0, (const float*)l.dgate.p, xin, (const float*)l.h_all.p, un, T, in, H, n_updates);
      // in a recorded step the launches for all but the last groups are one conditional node
      cudaGraphConditionalHandle skip = 0; const int tail = groups >= CLIP_SKIP_MIN && ctx->rec && ctx->rec->condition(&skip) ? (int)groups - CLIP_TAIL : 0;
      if (late) GN_LAUNCH(ctx, lstm_clip_start_kernel, nchunks, 1024, 0, (const float*)un, n_updates, Kc, start, skip, tail); else start = nullptr;
      if (world == 1 && late && !few) gather(start, nullptr);
      // Gram blocks of every group against the group before it and itself
      GemmDesc g; g.M = CG; g.N = 2 * CG; g.batch1 = nchunks; g.batch2 = (int)groups; g.ldc = 2 * CG; g.z_first = start; g.c_b1 = groups * CG * 2 * CG; g.c_b2 = CG * 2 * CG; g.sa_k = g.sb_k = 1;
      g.K = R4g; g.A = Dm + (long)CG_PAD * R4g; g.sa_m = R4g; g.B = Dm; g.sb_n = R4g; g.a_b1 = g.b_b1 = stride * R4g; g.a_b2 = g.b_b2 = (long)CG * R4g; g.C = G0; GN_TRY(gemm(ctx, g));
      g.K = ZWg; g.A = Zm + (long)CG_PAD * zs; g.sa_m = zs; g.B = Zm; g.sb_n = zs; g.a_b1 = g.b_b1 = stride * zs; g.a_b2 = g.b_b2 = (long)CG * zs; g.C = G1; GN_TRY(gemm(ctx, g));
      const long q4 = ng * CG * 2 * CG / 4;
      GN_LAUNCH(ctx, lstm_gram_mul_kernel, ew_grid(ctx, q4), 256, 0, G0, (const float*)G1, q4, (int)groups, (const int*)start);
      const ClipArgs a{Dm, Zm, G0, db, db + n_om, db + n_om + n_p, gmat, start, R4g, ZWg, (int)groups, slabs, stride};
      const size_t smem = clip_smem(ZWg);
      GN_CUDA(cudaFuncSetAttribute(lstm_clip_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      auto walk = [&](int from, int to) -> int { for (int j = from; j < to; j++) GN_EARLY_LAUNCH(ctx, lstm_clip_kernel, dim3(1 + slabs, nchunks), CG_THREADS, smem, a, j); return GN_OK; };
      if (tail) { int rc = GN_OK; GN_CUDA(ctx->rec->only_if(ctx->stream, skip, [&] { rc = walk(0, tail); })); GN_TRY(rc); }
      GN_TRY(walk(tail, (int)groups + 1));
      GN_LAUNCH(ctx, lstm_scatter_grad_kernel, cdiv((long)R4g * ZWg, 256), 256, 0, (const float*)gmat, (int)(groups & 1), nchunks, in, H, m->grads.p + l.p_off);
      return check_launch("lstm_backward");
    }
  }
  const int R4 = 4 * H, ZW = in + H + 1, rpc = (R4 + SCAN_CLUSTER - 1) / SCAN_CLUSTER;
  size_t smem = ((size_t)rpc * ZW + rpc + ZW + 33) * sizeof(float);
  if (smem > 220 * 1024) return fail(GN_ERR_UNSUPPORTED, "LSTM gradient of %d x %d per cluster CTA exceeds shared memory", rpc, ZW);
  float* scan; GN_TRY(ensure(m, S_SCAN, (size_t)nchunks * R4 * ZW, &scan));
  GN_CUDA(cudaFuncSetAttribute(lstm_grad_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{}; cfg.gridDim = dim3(nchunks * SCAN_CLUSTER); cfg.blockDim = dim3(SCAN_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1]; at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = SCAN_CLUSTER; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  GN_CUDA(cudaLaunchKernelEx(&cfg, lstm_grad_scan_kernel, (const float*)l.dgate.p, xin, (const float*)l.h_all.p, scan, T, in, H, B, chunk, 0));
  ctx->launches++;
  // worker gradients are summed in worker order (net.go:694-700)
  GN_LAUNCH(ctx, colsum_final_kernel, cdiv((long)R4 * ZW, 128), 128, 0, scan, nchunks, R4 * ZW, m->grads.p + l.p_off, 0);
  return check_launch("lstm_backward");
}

static AdamArgs adam_args(float lr, float b1, float b2, float eps, int t, float grad_scale);
static int adam_launch(Ctx* ctx, float* p, const float* g, float* m1, float* v, int64_t n, const AdamArgs& a, const AdamArgs* dargs, const int* status, cudaStream_t stream,
                       const float* loss_sum, float* ret, const WeightPlaneTable* t = nullptr);

static int backward(gn_model* m, int B, const float* gloss, int global_batch, int first_sample) {
  Ctx* ctx = &m->ctx->c;
  const float* g = gloss;
  float* pp[2] = {nullptr, nullptr}; int flip = 0;
  size_t maxio = 0; for (auto& l : m->L) maxio = std::max<size_t>(maxio, std::max(l.in_size, l.out_size));
  GN_TRY(ensure(m, S_G0, (size_t)B * maxio, &pp[0])); GN_TRY(ensure(m, S_G1, (size_t)B * maxio, &pp[1]));
  // This layer's slice of the flat gradient buffer is final: sum it over the ranks while earlier layers still compute
  // (unless every rank already holds the whole sum), and apply this slice's Adam update right behind it on the
  // communication stream -- the layer's parameters are not read again in this step -- so that neither the exchange
  // nor the optimiser pass is left over when the backward pass ends.  GONEURON_CUDA_COMM=end issues the same sequence
  // for all layers after the backward pass instead (no overlap; for measurements).
  static const bool comm_at_end = [] { const char* e = getenv("GONEURON_CUDA_COMM"); return e && !strcmp(e, "end"); }();
  std::vector<int> deferred;
  bool gated = false;                                       // g already carries the derivative of the ReLU below it
  auto relu_conv_below = [&](int li) { return li > 0 && m->L[li - 1].d.kind == GN_LAYER_CONV2D && m->L[li - 1].d.activation == GN_ACT_RELU; };
  bool row0 = false; int row0_T = 0, row0_D = 0;            // g holds the gradient of token 0 of every sequence, [B, row0_D]; the other tokens' is zero
  auto layer_comm = [&](int li) -> int {
    LayerRT& l = m->L[li]; float* gr = m->grads.p + l.p_off;
    GN_CUDA(cudaEventRecord(m->layer_ev[li], ctx->stream));
    GN_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->layer_ev[li], 0));
    if (!l.grad_replicated) {
      int rc = ctx->nccl->AllReduce(gr, gr, (size_t)l.p_cnt, NCCL_FLOAT32, NCCL_SUM, ctx->comm, ctx->comm_stream);
      if (rc) return fail(GN_ERR_NCCL, "ncclAllReduce(grads of layer %d): %s", li, ctx->nccl->GetErrorString(rc));
    }
    GN_TRY(adam_launch(ctx, m->params.p + l.p_off, gr, m->m1.p + l.p_off, m->v2.p + l.p_off, l.p_cnt,
                       adam_args(m->lr, m->b1, m->b2, m->eps, m->timestep + 2, (float)(1.0 / (double)global_batch)), nullptr, ctx->d_status, ctx->comm_stream, nullptr, nullptr));
    // ... and the layer's prepared operand planes right behind the update, still hidden behind the earlier layers' backward pass
    if (!m->wplanes.e.empty() && m->wplanes.used) {
      int j0, j1; m->wplanes.layer_range(li, &j0, &j1);
      GN_TRY(wplanes_refresh_range(ctx, m->wplanes, j0, j1, ctx->comm_stream));
      m->wplanes_layerwise = true;
    }
    return GN_OK;
  };
  for (int li = (int)m->L.size() - 1; li >= 0; li--) {
    LayerRT& l = m->L[li]; const gn_layer_desc& d = l.d;
    const float* xin = l.fin;
    // (a layer below may read the same floats as sequences of another length and width: token 0 is then a different part of them)
    const bool takes_row0 = d.kind == GN_LAYER_TRANSFORMER_BLOCK ? l.row0_grad : d.kind == GN_LAYER_POSENC ? d.seq_len == row0_T && d.dim == row0_D
                                                                                : d.kind == GN_LAYER_EMBEDDING && d.seq_len == row0_T && d.out_size == row0_D;
    if (row0 && !takes_row0) {
      const long n = (long)B * row0_T * row0_D;             // a layer that wants the gradient of every token: zeros except token 0
      GN_LAUNCH(ctx, cls_bwd_kernel, ew_grid(ctx, n), 256, 0, g, pp[flip], row0_T, row0_D, n); g = pp[flip]; flip ^= 1; row0 = false;
    }
    const float* p = m->params.p + l.p_off; float* gr = m->grads.p + l.p_off;
    float* dx = pp[flip]; bool need_dx = li > 0;
    switch (d.kind) {
      case GN_LAYER_DENSE: {
        const float* W = p; long wn = (long)d.in_size * d.out_size; const float* dz = g;
        if (d.activation != GN_ACT_LINEAR && !(m->head_fused && li + 1 == (int)m->L.size()) && !gated) {
          float* dzb; GN_TRY(ensure(m, S_DZ, (size_t)B * d.out_size, &dzb)); long n = (long)B * d.out_size;
          if (d.activation == GN_ACT_SOFTMAX || d.activation == GN_ACT_LOGSOFTMAX)
            GN_LAUNCH(ctx, head_jacobian_kernel, B, 256, 0, g, l.out.p, dzb, d.out_size, d.activation == GN_ACT_LOGSOFTMAX ? 1 : 0);
          else GN_LAUNCH(ctx, act_backward_kernel, ew_grid(ctx, n), 256, 0, g, d.activation == GN_ACT_RELU ? l.out.p : l.z.p, dzb, n, d.activation, act_alpha_of(d.activation, d.reserved));
          dz = dzb;
        }
        GemmDesc gw; gw.M = d.out_size; gw.N = d.in_size; gw.K = B; gw.A = dz; gw.sa_m = 1; gw.sa_k = d.out_size; gw.B = xin; gw.sb_k = d.in_size; gw.sb_n = 1; gw.C = gr; gw.ldc = d.in_size;
        if (gemm_on_tc(ctx, gw)) {      // the bias gradient beside the weight gradient's operand planes and product (batch 1000, 1100 outputs: 10 us)
          GN_TRY(side_run(ctx, [&]() -> int { return colsum(m, dz, d.out_size, B, d.out_size, gr + wn, false, S_PART4); }));
          GN_TRY(gemm(ctx, gw));
        } else if (need_dx) GN_TRY(side_weight_bias_grads(m, 1, B, d.out_size, d.in_size, dz, xin, d.in_size, gr, gr + wn));
        else GN_TRY(weight_bias_grads(m, ctx, B, d.out_size, d.in_size, dz, d.out_size, xin, d.in_size, gr, gr + wn));
        gated = false;
        if (need_dx) {
          // a Dense(ReLU) below: its derivative, [activation > 0], gates this product's epilogue
          const LayerRT& b = m->L[li - 1]; gated = b.d.kind == GN_LAYER_DENSE && b.d.activation == GN_ACT_RELU;
          GemmDesc gd; gd.M = B; gd.N = d.in_size; gd.K = d.out_size; gd.A = dz; gd.sa_m = d.out_size; gd.sa_k = 1; gd.B = W; gd.sb_k = d.in_size; gd.sb_n = 1; gd.C = dx; gd.ldc = d.in_size;
          if (gated) { gd.mask = b.out.p; gd.mask_ld = d.in_size; }
          GN_TRY(gemm(ctx, gd)); g = dx; flip ^= 1;
        }
        break; }
      case GN_LAYER_CONV2D: {
        ConvShape c{B, d.in_size, d.out_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        const int nW = d.out_size * d.in_size * d.kernel * d.kernel;
        GN_TRY(conv_backward(m, c, gated ? (int)GN_ACT_LINEAR : d.activation, act_alpha_of(d.activation, d.reserved), g, xin, p, l.z.p, l.out.p, gr, gr + nW, need_dx ? dx : nullptr, force_simt_engine() ? CONV_CUDA : CONV_AUTO));
        gated = false;
        if (need_dx) { g = dx; flip ^= 1; }
        break; }
      case GN_LAYER_MAXPOOL2D: {
        PoolShape c{B, d.in_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        if (c.k <= c.s) {
          gated = relu_conv_below(li);
          if (c.k == 2 && c.s == 2 && c.p == 0 && c.H == 2 * c.oH && c.W == 2 * c.oW)
            GN_LAUNCH(ctx, maxpool_bwd_2x2_kernel, dim3(B * c.C, std::min(cdiv((long)c.oH * c.oW, 256), 65535u)), 256, 0, g, (const int*)l.idx.p, (const float*)l.out.p, dx, c, gated ? 1 : 0);
          else GN_LAUNCH(ctx, maxpool_bwd_gather_kernel, dim3(B * c.C, std::min(cdiv((long)c.H * c.W, 256), 65535u)), 256, 0, g, (const int*)l.idx.p, (const float*)l.out.p, dx, c, gated ? 1 : 0);
          g = dx; flip ^= 1; break;
        }
        GN_CUDA(stream_zero(ctx, dx, (size_t)B * l.in_size * sizeof(float)));
        long n = (long)B * l.out_size;
        GN_LAUNCH(ctx, maxpool_bwd_kernel, ew_grid(ctx, n), 256, 0, g, (const int*)l.idx.p, dx, c);
        g = dx; flip ^= 1; break; }
      case GN_LAYER_CONV1D: {
        Conv1Shape c{B, d.in_size, d.out_size, d.kernel, d.stride, d.padding, d.in_w, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        const int nW = d.out_size * d.in_size * d.kernel;
        GN_LAUNCH(ctx, conv1d_wgrad_kernel, nW + d.out_size, 256, 0, g, xin, gr, gr + nW, c);
        if (need_dx) { long ni = (long)B * l.in_size; GN_LAUNCH(ctx, conv1d_dgrad_kernel, ew_grid(ctx, ni), 256, 0, g, p, dx, c); g = dx; flip ^= 1; }
        break; }
      case GN_LAYER_DROPOUT:
        if (need_dx) { long n = (long)B * l.in_size; GN_LAUNCH(ctx, dropout_bwd_kernel, ew_grid(ctx, n), 256, 0, g, (const float*)l.z.p, dx, n, l.bn_mom); g = dx; flip ^= 1; }
        break;
      case GN_LAYER_AVGPOOL2D: {
        PoolShape c{B, d.in_size, d.kernel, d.stride, d.padding, d.in_h, d.in_w,
                    (d.in_h + 2 * d.padding - d.kernel) / d.stride + 1, (d.in_w + 2 * d.padding - d.kernel) / d.stride + 1};
        if (need_dx) { long n = (long)B * l.in_size; GN_LAUNCH(ctx, avgpool_bwd_kernel, ew_grid(ctx, n), 256, 0, g, dx, c); g = dx; flip ^= 1; }
        break; }
      case GN_LAYER_FLATTEN: break;
      case GN_LAYER_LSTM_UNROLLED:
        GN_TRY(lstm_backward(m, l, li, B, xin, g, global_batch, first_sample, dx)); if (need_dx) { g = dx; flip ^= 1; } break;
      case GN_LAYER_GRU_UNROLLED: {
        const int H = d.out_size, in = d.in_size, T = d.seq_len, threads = ((H + 31) / 32) * 32;
        const float* Wx = p; const float* Wh = p + (long)3 * H * in;
        float* gWx = gr; float* gWh = gr + (long)3 * H * in; float* gb = gWh + (long)2 * H * H;
        if (gru_reg_ok(H)) GN_TRY(gru_bwd_reg(ctx, g, Wh, l.pre_i.p, l.h_all.p, l.dgate.p, l.c_all.p, l.z.p, RecShape{T, in, H, d.return_seq, B}));
        else GN_LAUNCH(ctx, gru_bwd_kernel, B, threads, (size_t)2 * H * sizeof(float), g, Wh, (const float*)l.pre_i.p, (const float*)l.h_all.p, l.dgate.p, l.c_all.p, l.z.p, T, H, d.return_seq);
        // input weights and biases: every step's delta meets the input of the LAST forward call (gru.go:429-447), so per sample
        // gWx = (sum_t d_t) (x) x_{T-1}: the same batch-level contraction as the inner Dense layers of a TransformerBlock
        GN_TRY(inner_dense_param_grads(m, l.dgate.p, B, T, 3 * H, xin, in, gWx, gb));
        // recurrent weights: update rows from h_{t-1}, reset rows from the candidate's delta and r (.) h_{t-1} (gru.go:450-476)
        GN_TRY(gemm_tn(ctx, B * T, H, H, l.dgate.p, 3 * H, l.c_all.p, H, gWh));
        GN_TRY(gemm_tn(ctx, B * T, H, H, l.dgate.p + 2 * H, 3 * H, l.z.p, H, gWh + (long)H * H));
        if (need_dx) { GN_TRY(gemm_nn(ctx, B * T, 3 * H, in, l.dgate.p, 3 * H, Wx, dx, in)); g = dx; flip ^= 1; }
        break; }
      case GN_LAYER_EMBEDDING: {
        // Only the last sample of every worker chunk reaches the table (embedding.go:151-154): global samples
        // c*chunk + chunk - 1 and the very last one.
        const int chunk = (global_batch + m->W - 1) / m->W, T = row0 ? 1 : d.seq_len, Tid = d.seq_len, dim = d.out_size;     // T: tokens of a sample with a gradient
        const int nq = (global_batch + chunk - 1) / chunk;                       // qualifying samples of the global batch
        auto q_sample = [&](int q) { return std::min(global_batch - 1, q * chunk + chunk - 1); };
        GN_CUDA(stream_zero(ctx, gr, (size_t)l.p_cnt * sizeof(float)));     // most rows of the table have no gradient
        const size_t smem = (size_t)T * sizeof(int);
        if (smem > 48 * 1024) GN_CUDA(cudaFuncSetAttribute(embedding_bwd_sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const bool sparse = ctx->world > 1 && (double)nq * T * (dim + 1) < 0.5 * (double)l.p_cnt;
        if (sparse) {
          // few samples, large table: exchange those samples' rows (nq * T * (dim + 1) floats) instead of all-reducing the table;
          // every rank then builds the complete table gradient itself
          float* buf; GN_TRY(ensure(m, S_EMB, (size_t)nq * T * (dim + 1) + (size_t)nq * T, &buf));
          float* rows = buf; float* idsf = buf + (size_t)nq * T * dim; int* idsi = reinterpret_cast<int*>(idsf + (size_t)nq * T);
          GN_CUDA(stream_zero(ctx, buf, (size_t)nq * T * (dim + 1) * sizeof(float)));
          for (int q = 0; q < nq; q++) {
            const int sl = q_sample(q) - first_sample; if (sl < 0 || sl >= B) continue;
            GN_LAUNCH(ctx, embedding_pack_kernel, T, 128, 0, g + (size_t)sl * T * dim, (const int*)l.idx.p + (size_t)sl * Tid, rows + (size_t)q * T * dim, idsf + (size_t)q * T, T, dim);
          }
          GN_CUDA(cudaEventRecord(m->gather_ev, ctx->stream));
          GN_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->gather_ev, 0));
          int rc = ctx->nccl->AllReduce(buf, buf, (size_t)nq * T * (dim + 1), NCCL_FLOAT32, NCCL_SUM, ctx->comm, ctx->comm_stream);
          if (rc) return fail(GN_ERR_NCCL, "ncclAllReduce(embedding rows): %s", ctx->nccl->GetErrorString(rc));
          GN_CUDA(cudaEventRecord(m->gather_ev, ctx->comm_stream));
          GN_CUDA(cudaStreamWaitEvent(ctx->stream, m->gather_ev, 0));
          GN_LAUNCH(ctx, ids_to_int_kernel, cdiv((long)nq * T, 256), 256, 0, (const float*)idsf, idsi, nq * T);
          for (int q = 0; q < nq; q++)
            GN_LAUNCH(ctx, embedding_bwd_sample_kernel, T, 128, smem, (const float*)(rows + (size_t)q * T * dim), (const int*)(idsi + (size_t)q * T), gr, T, dim);
          l.grad_replicated = true;
        } else {
          for (int q = 0; q < nq; q++) {
            const int sl = q_sample(q) - first_sample; if (sl < 0 || sl >= B) continue;
            GN_LAUNCH(ctx, embedding_bwd_sample_kernel, T, 128, smem, g + (size_t)sl * T * dim, (const int*)l.idx.p + (size_t)sl * Tid, gr, T, dim);
          }
          l.grad_replicated = false;
        }
        break; }
      case GN_LAYER_POSENC:
        if (row0) GN_CUDA(stream_zero(ctx, gr, (size_t)l.p_cnt * sizeof(float)));
        { const int n = row0 ? d.dim : l.out_size; GN_TRY(colsum(m, g, n, B, n, gr, false)); } break;     // gP = sum over samples; dx = g
      case GN_LAYER_TRANSFORMER_BLOCK:
        if (row0) GN_TRY(block_backward_row0(m, l, B, xin, g, dx, &row0)); else GN_TRY(block_backward(m, l, B, xin, g, dx));
        g = dx; flip ^= 1; break;
      case GN_LAYER_CLS_POOLING: {
        long n = (long)B * l.in_size;
        if (li > 0 && m->L[li - 1].row0_grad) { row0 = true; row0_T = d.seq_len; row0_D = d.dim; break; }
        GN_LAUNCH(ctx, cls_bwd_kernel, ew_grid(ctx, n), 256, 0, g, dx, d.seq_len, d.dim, n); g = dx; flip ^= 1; break; }
      case GN_LAYER_BATCHNORM2D: {
        const int C = d.in_size, S = d.in_h * d.in_w; const long BC = (long)B * C;
        float* pg; GN_TRY(ensure(m, S_DELTA, (size_t)B * 2 * C, &pg));
        gated = relu_conv_below(li);
        GN_LAUNCH(ctx, bn_bwd_kernel, (unsigned)BC, 256, 0, g, xin, p, l.stat.p, dx, pg, C, S, BC, gated ? 1 : 0);
        GN_TRY(colsum(m, pg, 2 * C, B, 2 * C, gr, false));
        g = dx; flip ^= 1; break; }
      case GN_LAYER_LAYERNORM: {
        long rows = (long)B * (l.in_size / d.dim);
        GN_TRY(norm_backward(m, false, g, xin, p, l.stat.p, dx, gr, gr + d.dim, rows, d.dim));
        g = dx; flip ^= 1; break; }
      case GN_LAYER_RMSNORM: {
        long rows = (long)B * (l.in_size / d.dim);
        GN_TRY(norm_backward(m, true, g, xin, p, l.stat.p, dx, gr, nullptr, rows, d.dim)); g = dx; flip ^= 1;
        break; }
    }
    GN_TRY(side_join(ctx));
    GN_TRY(check_launch("backward"));
    if (ctx->world > 1 && l.p_cnt > 0) {
      if (comm_at_end) deferred.push_back(li); else GN_TRY(layer_comm(li));
    }
  }
  for (int li : deferred) GN_TRY(layer_comm(li));
  return GN_OK;
}

// ---------------------------------------------------------------- Adam
static void adam_coeffs(float lr, float b1, float b2, int t, float* effLR) {
  // opt.go:237-242: bias terms through float64 pow, rounded to float32; sqrt through float64
  float bias1 = (float)(1.0 - std::pow((double)b1, (double)t));
  float bias2 = (float)(1.0 - std::pow((double)b2, (double)t));
  *effLR = lr * (float)std::sqrt((double)bias2) / bias1;
}
static AdamArgs adam_args(float lr, float b1, float b2, float eps, int t, float grad_scale) {
  float effLR; adam_coeffs(lr, b1, b2, t, &effLR);
  return AdamArgs{effLR, b1, b2, 1.f - b1, 1.f - b2, eps, grad_scale};
}
static int adam_launch(Ctx* ctx, float* p, const float* g, float* m1, float* v, int64_t n, const AdamArgs& a, const AdamArgs* dargs, const int* status,
                       cudaStream_t stream, const float* loss_sum, float* ret, const WeightPlaneTable* t) {
  const unsigned grid = (unsigned)std::max<long>(1, std::min<long>(cdiv((n + 3) / 4, 256), 8L * ctx->sm_count)); stream = stream ? stream : ctx->stream;      // one resident round
  if (t) {
    GN_CUDA(stream_zero(ctx, stream, t->mx.p, t->e.size() * sizeof(int)));
    GN_LAUNCH_ON(ctx, stream, adam_kernel<true>, grid, 256, 0, p, g, m1, v, (long)n, a, dargs, status, loss_sum, ret, reinterpret_cast<const PlaneRange*>(t->ranges.p), (int)t->e.size(), reinterpret_cast<int*>(t->mx.p));
  } else GN_LAUNCH_ON(ctx, stream, adam_kernel<false>, grid, 256, 0, p, g, m1, v, (long)n, a, dargs, status, loss_sum, ret, nullptr, 0, nullptr);
  return check_launch("adam");
}
// Meaning of a non-zero status word.
static int status_error(int st) {
  if (st == GN_STATUS_BAD_TOKEN) return fail(GN_ERR_INVALID_ARG, "a token id outside [0, vocabulary) was given to an Embedding layer (embedding.go:124-129); parameters and optimiser state are unchanged");
  return fail(GN_ERR_TIMEOUT, "a device-side bounded wait gave up (status word %d); parameters and optimiser state are unchanged", st);
}
static int clear_status(Ctx* c, int st) { cudaMemsetAsync(c->d_status, 0, sizeof(int), c->stream); cudaStreamSynchronize(c->stream); return status_error(st); }
// Reads the status word; non-zero clears it and becomes an error (GN_ERR_TIMEOUT: a bounded device-side wait gave up).
static int check_status_word(Ctx* c) {
  int st = 0; GN_CUDA(copy_d2h(c, &st, c->d_status, sizeof(int)));
  return st != 0 ? clear_status(c, st) : GN_OK;
}

// The step in two halves: everything that needs x only, then what needs y.  A host y is copied while the first half runs.
static int issue_forward(gn_model* m, const float* x_dev, int B, int global_batch, int first_sample, const float** yp) {
  Ctx* ctx = &m->ctx->c;
  m->cur_first_sample = first_sample; m->cur_global_batch = global_batch;
  GN_TRY(forward(m, x_dev, B, yp, true));
  for (auto& l : m->L) if (l.d.kind == GN_LAYER_DROPOUT)          // every rank moves the stream on by the whole global batch
    GN_LAUNCH(ctx, dropout_advance_kernel, 1, 1, 0, m->state.p + l.s_off, (unsigned long long)global_batch * (unsigned long long)l.in_size);
  return GN_OK;
}
static int issue_backward(gn_model* m, const float* yp, const float* y_dev, int B, int global_batch, int first_sample, const AdamArgs& a) {
  Ctx* ctx = &m->ctx->c; unsigned* ticket = reinterpret_cast<unsigned*>(ctx->d_status + 1);
  if (m->head_fused) {
    // z -> loss and dz in one kernel; the smallest cluster whose registers hold a row
    const LayerRT& h = m->L.back(); const int n = m->out_size, lg = h.d.activation == GN_ACT_LOGSOFTMAX;
    int cs = 1; while (cs < HEAD_MAX_CS && n > cs * HEAD_THREADS * 4) cs *= 2;
    const int per = cdiv(n, cs * HEAD_THREADS); const dim3 grid(B * cs);
    auto* K = per <= 1 ? head_loss_kernel<1> : per <= 4 ? head_loss_kernel<4> : head_loss_kernel<HEAD_MAX_E>;
    GN_CLUSTER_LAUNCH(ctx, K, grid, HEAD_THREADS, 0, cs, (const float*)h.z.p, y_dev, m->lossg.p, m->loss_s.p, n, B, cs, lg, m->loss_kind, ticket, m->loss_sum.p);
  } else GN_LAUNCH(ctx, loss_rows_kernel, B, m->out_size <= 64 ? 32 : 256, 0, yp, y_dev, m->lossg.p, m->loss_s.p, m->out_size, m->loss_kind, ticket, m->loss_sum.p);
  GN_TRY(backward(m, B, m->lossg.p, global_batch, first_sample));
  if (ctx->world > 1) {
    // loss sum over the ranks, then the main stream waits for the communication stream (per-layer gradient
    // all-reduces were issued during the backward pass); ar0..ar1 brackets the exposed wait
    GN_CUDA(cudaEventRecord(m->layer_ev.back(), ctx->stream));
    GN_CUDA(cudaStreamWaitEvent(ctx->comm_stream, m->layer_ev.back(), 0));
    int rc = ctx->nccl->AllReduce(m->loss_sum.p, m->loss_sum.p, 1, NCCL_FLOAT32, NCCL_SUM, ctx->comm, ctx->comm_stream);
    if (rc) return fail(GN_ERR_NCCL, "ncclAllReduce(loss): %s", ctx->nccl->GetErrorString(rc));
    GN_CUDA(cudaEventRecord(m->comm_done, ctx->comm_stream));
    GN_CUDA(cudaEventRecord(m->ar0, ctx->stream));
    GN_CUDA(cudaStreamWaitEvent(ctx->stream, m->comm_done, 0));
    GN_CUDA(cudaEventRecord(m->ar1, ctx->stream));
    // (the update was applied slice by slice behind each layer's all-reduce, see backward())
    GN_LAUNCH(ctx, finish_kernel, 1, 32, 0, (const float*)m->loss_sum.p, ctx->d_ret, 1, (const int*)ctx->d_status, ctx->d_ret);
    return check_launch("finish");
  }
  // Network.Step (net.go:260-284): NewStep() then StepInPlace with t = timestep + 1.  The pass reads the status word
  // first: after a bounded wait gave up it changes nothing.
  return adam_launch(ctx, m->params.p, m->grads.p, m->m1.p, m->v2.p, m->P, a, reinterpret_cast<const AdamArgs*>(m->io.p), ctx->d_status, nullptr, m->loss_sum.p, ctx->d_ret,
                     m->wplanes.used && !m->wplanes.e.empty() ? &m->wplanes : nullptr);
}

// Recorded launches of a step (or of an inference pass).  A call whose sizes and buffers have been seen before is replayed as one or
// two CUDA graphs: a step is 10 to 300 launches of a few microseconds each, which the host would otherwise issue one by one.  The
// first call with a set of sizes runs launch by launch (it may allocate), the second is recorded (GraphRec).  A graph refers to
// buffers by address, so it is dropped when the model or the context has replaced one (epoch).  What differs from call to
// call lies in memory: inputs, the Adam coefficients (head of the model's `io` buffer), the results.
struct StepGraph {
  int B, global_batch, first_sample; const float *x, *y; bool staged, training; unsigned spin; uint64_t epoch_m, epoch_c;
  bool same(const StepGraph& o) const {
    return B == o.B && global_batch == o.global_batch && first_sample == o.first_sample && x == o.x && y == o.y && staged == o.staged && training == o.training && spin == o.spin &&
           epoch_m == o.epoch_m && epoch_c == o.epoch_c;
  }
  cudaGraphExec_t exec[2] = {nullptr, nullptr}; bool recorded = false; uint64_t uses = 0, next_try = 1, last_use = 0;
  int64_t launches = 0, gemm_launches = 0; double gemm_flops = 0, gemm_bytes = 0, split_bytes = 0; const float* out = nullptr;
  void drop() { for (auto& e : exec) if (e) { cudaGraphExecDestroy(e); e = nullptr; } recorded = false; }
  bool due() { return !recorded && ++uses >= next_try; }      // (a graph that could not be made is tried again after 4, 16, 64 ... uses)
  void done(bool ok) { recorded = ok; if (!ok) { drop(); next_try *= 4; } }
};
constexpr size_t MAX_GRAPHS = 8;                             // per model: batch sizes and device-resident batches in turn
static StepGraph* find_graph(gn_model* m, StepGraph key) {
  Ctx* ctx = &m->ctx->c;
  static const bool off = getenv("GONEURON_CUDA_NO_GRAPHS") != nullptr;
  if (off || ctx->world > 1 || ctx->profile || ctx->tc_tile_queue) return nullptr;
  key.epoch_m = m->epoch; key.epoch_c = ctx->epoch; key.spin = ctx->spin_limit; key.last_use = ++m->graph_clock;
  for (auto& g : m->graphs) if (g->same(key)) { g->last_use = key.last_use; return g.get(); }
  return nullptr;
}
// Remembers a set of sizes that has just run launch by launch (the epochs are those after the run).
static void note_graph(gn_model* m, StepGraph key) {
  Ctx* ctx = &m->ctx->c;
  key.epoch_m = m->epoch; key.epoch_c = ctx->epoch; key.spin = ctx->spin_limit; key.last_use = ++m->graph_clock;
  for (auto it = m->graphs.begin(); it != m->graphs.end();) {      // stale ones can never match again
    if ((*it)->epoch_m != key.epoch_m || (*it)->epoch_c != key.epoch_c) { (*it)->drop(); it = m->graphs.erase(it); } else ++it;
  }
  for (auto& g : m->graphs) if (g->same(key)) return;
  if (m->graphs.size() >= MAX_GRAPHS) {
    auto old = std::min_element(m->graphs.begin(), m->graphs.end(), [](auto& a, auto& b) { return a->last_use < b->last_use; });
    (*old)->drop(); m->graphs.erase(old);
  }
  m->graphs.emplace_back(new StepGraph(key));
}
// What `issue` would launch as a graph; *out stays null when that cannot be made (the caller then runs it directly).
template <class F> static void record(gn_model* m, F&& issue, cudaGraphExec_t* out) {
  Ctx* ctx = &m->ctx->c; const uint64_t em = m->epoch, ec = ctx->epoch; *out = nullptr;
  struct Guard { Ctx* c; ~Guard() { c->side_pending = false; cudaGetLastError(); } } guard{ctx};
  *out = record_graph(ctx->rec, ctx->graph_conditions, [&] { return issue() == GN_OK && em == m->epoch && ec == ctx->epoch; });      // (a buffer that was replaced may be in earlier nodes)
}
static void reset_counters(Ctx* ctx) { ctx->gemm_flops = 0; ctx->gemm_launches = 0; ctx->gemm_ms = 0; ctx->ev_used = 0; ctx->gemm_bytes = 0; ctx->split_bytes = 0; }

// x and y: device memory, or (host = true) host memory.
static int train_step_issue(gn_model* m, const float* x, const float* y, bool host, int B, int global_batch, int first_sample) {
  Ctx* ctx = &m->ctx->c; const size_t nx = (size_t)B * m->in_size, ny = (size_t)B * m->out_size, y_at = IO_ARGS + (nx + 63) / 64 * 64;
  const float inv = (float)(1.0 / (double)global_batch);                                        // net.go:703
  m->last_inv_batch = inv;
  const AdamArgs a = adam_args(m->lr, m->b1, m->b2, m->eps, m->timestep + 2, inv);
  GN_TRY(wplanes_need_max(ctx, m->wplanes));                   // (a recorded step relies on them)
  // small host batches (or a small x: token ids) go through one pinned block together with the coefficients: one copy instead of three
  const bool staged = host && y_at + ny <= STAGE_IN, staged_x = staged || (host && nx * 4 < (128u << 10));
  memcpy(ctx->h_stage, &a, sizeof a);
  const float* xd = host ? m->io.p + IO_ARGS : x; const float* yd = host ? m->io.p + y_at : y;
  if (staged_x) memcpy(ctx->h_stage + IO_ARGS, x, nx * 4);
  if (staged) memcpy(ctx->h_stage + y_at, y, ny * 4);
  StepGraph key{B, global_batch, first_sample, xd, yd, staged, true};
  StepGraph* g = find_graph(m, key);
  const float* yp = nullptr;
  auto copy_in = [&]() -> int { GN_CUDA(stream_copy(ctx, m->io.p, ctx->h_stage, (staged ? y_at + ny : staged_x ? IO_ARGS + nx : IO_ARGS) * 4, cudaMemcpyHostToDevice)); return GN_OK; };
  auto first = [&]() -> int { return issue_forward(m, xd, B, global_batch, first_sample, &yp); };
  auto second = [&]() -> int { return issue_backward(m, yp, yd, B, global_batch, first_sample, a); };
  const bool split = host && !staged;                          // y is copied between the halves
  if (g && g->due()) {
    const int64_t l0 = ctx->launches; reset_counters(ctx);
    m->wplanes.dirty = true;                                   // as in every step: the parameters have moved since the planes were written
    if (split) {
      record(m, [&]() -> int { GN_TRY(copy_in()); return first(); }, &g->exec[0]);
      if (g->exec[0]) record(m, second, &g->exec[1]);
    } else record(m, [&]() -> int { GN_TRY(copy_in()); GN_TRY(first()); return second(); }, &g->exec[0]);
    g->launches = ctx->launches - l0; ctx->launches = l0; g->gemm_launches = ctx->gemm_launches; g->gemm_flops = ctx->gemm_flops; g->gemm_bytes = ctx->gemm_bytes; g->split_bytes = ctx->split_bytes;
    g->done(g->exec[0] && (!split || g->exec[1]));
    if (!g->recorded) { m->wplanes.dirty = true; forget_planes(ctx); }
  }
  reset_counters(ctx);
  if (split && !staged_x) GN_CUDA(cudaMemcpyAsync(m->io.p + IO_ARGS, x, nx * 4, cudaMemcpyHostToDevice, ctx->stream));
  GN_CUDA(cudaEventRecord(m->ev0, ctx->stream));
  const bool replay = g && g->recorded;
  if (replay) { GN_CUDA(cudaGraphLaunch(g->exec[0], ctx->stream)); }
  else { GN_TRY(copy_in()); GN_TRY(first()); }
  if (split) {                                               // on a stream of its own: it must not wait for the first half
    GN_CUDA(cudaMemcpyAsync(m->io.p + y_at, y, ny * 4, cudaMemcpyHostToDevice, ctx->copy_stream));
    GN_CUDA(cudaEventRecord(ctx->copy_ev, ctx->copy_stream)); GN_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->copy_ev, 0));
  }
  if (replay) { if (split) GN_CUDA(cudaGraphLaunch(g->exec[1], ctx->stream)); }
  else GN_TRY(second());
  GN_CUDA(cudaEventRecord(m->ev1, ctx->stream));
  if (replay) {
    ctx->launches += g->launches; ctx->gemm_launches = g->gemm_launches; ctx->gemm_flops = g->gemm_flops; ctx->gemm_bytes = g->gemm_bytes; ctx->split_bytes = g->split_bytes;
    forget_planes(ctx);
  }
  GN_CUDA(cudaStreamSynchronize(ctx->stream));                // the loss sum and the status word are in host memory now
  if (!g) note_graph(m, key);
  return GN_OK;
}

// A call that fails after work has been queued must not leave that work running behind the caller's back (the pinned blocks are the next
// call's): waits for all of the context's streams.
static int drained(gn_model* m, int rc) {
  Ctx* ctx = &m->ctx->c; const std::string msg = last_error();
  for (auto s : {ctx->comm_stream, ctx->copy_stream, ctx->side_stream, ctx->stream}) if (s) cudaStreamSynchronize(s);
  cudaGetLastError(); ctx->side_pending = false;
  m->wplanes.dirty = true; m->wplanes.max_ok = false; forget_planes(ctx); last_error() = msg; return rc;
}

static int train_step(gn_model* m, const float* x, const float* y, bool host, int B, int global_batch, int first_sample, float* mean_loss) {
  Ctx* ctx = &m->ctx->c;
  if (global_batch <= 0) { global_batch = B; first_sample = 0; }
  GN_TRY(ensure_capacity(m, B, true));
  int64_t launches0 = ctx->launches;
  m->wplanes_layerwise = false;
  int rc = train_step_issue(m, x, y, host, B, global_batch, first_sample);
  if (rc != GN_OK) return drained(m, rc);
  int st; memcpy(&st, &ctx->h_ret[1], sizeof(int));
  if (st != 0) { m->wplanes.dirty = true; m->wplanes.max_ok = false; return clear_status(ctx, st); }         // the Adam pass saw the same word and left parameters, moments and the step counter alone
  m->timestep += 1;
  m->wplanes.max_ok = m->wplanes.used;               // left behind by the update
  m->wplanes.dirty = !m->wplanes_layerwise;          // the parameters moved: their operand planes are stale, unless they were renewed layer by layer behind the update
  m->wplanes_layerwise = false;
  if (mean_loss) *mean_loss = ctx->h_ret[0] / (float)global_batch;
  m->stats.kernel_launches = ctx->launches - launches0;
  m->stats.gemm_flops = ctx->gemm_flops; m->stats.gemm_launches = ctx->gemm_launches; m->stats.gemm_ms = 0.f;
  m->stats.gemm_bytes = ctx->gemm_bytes; m->stats.split_bytes = ctx->split_bytes; m->stats_timed = false;
  if (ctx->profile) { float tot = 0.f; for (size_t i = 0; i < ctx->ev_used; i++) { float ms = 0.f; cudaEventElapsedTime(&ms, ctx->ev_pool[i].first, ctx->ev_pool[i].second); tot += ms; } m->stats.gemm_ms = tot; }
  return GN_OK;
}

// Batched inference, host to host.
static int forward_issue(gn_model* m, const float* x, int B, float* out) {
  Ctx* ctx = &m->ctx->c; const size_t nx = (size_t)B * m->in_size, ny = (size_t)B * m->out_size;
  const bool staged = nx <= STAGE_IN, small = ny <= STAGE_FLOATS;      // through the pinned blocks, in and out
  const float* xd = m->io.p + IO_ARGS; const float* yp = nullptr;
  if (staged) memcpy(ctx->h_stage, x, nx * 4);
  if (m->wplanes.used) GN_TRY(wplanes_refresh(ctx, m->wplanes));           // no-op unless the parameters changed since the last pass
  auto body = [&]() -> int {
    if (staged) GN_CUDA(stream_copy(ctx, m->io.p + IO_ARGS, ctx->h_stage, nx * 4, cudaMemcpyHostToDevice));
    GN_TRY(forward(m, xd, B, &yp, false));
    // a few KB are written to host memory by a kernel, more by the copy engine
    const bool by_kernel = ny <= 4096;
    if (small && !by_kernel) GN_CUDA(stream_copy(ctx, ctx->h_out, yp, ny * 4, cudaMemcpyDeviceToHost));
    GN_LAUNCH(ctx, finish_kernel, by_kernel ? cdiv(ny, 256) : 1, by_kernel ? 256 : 32, 0, yp, ctx->d_out, by_kernel ? (int)ny : 0, (const int*)ctx->d_status, ctx->d_ret);
    return check_launch("finish");
  };
  StepGraph key{B, 0, 0, xd, nullptr, staged, false};
  StepGraph* g = find_graph(m, key);
  if (g && g->due()) {
    const int64_t l0 = ctx->launches;
    record(m, body, &g->exec[0]);
    ctx->launches = l0; g->done(g->exec[0] != nullptr); g->out = yp;
    if (!g->recorded) { m->wplanes.dirty = true; forget_planes(ctx); }
  }
  if (!staged) GN_CUDA(cudaMemcpyAsync(m->io.p + IO_ARGS, x, nx * 4, cudaMemcpyHostToDevice, ctx->stream));
  if (g && g->recorded) { GN_CUDA(cudaGraphLaunch(g->exec[0], ctx->stream)); yp = g->out; forget_planes(ctx); }
  else GN_TRY(body());
  if (!small) GN_CUDA(cudaMemcpyAsync(out, yp, ny * 4, cudaMemcpyDeviceToHost, ctx->stream));
  GN_CUDA(cudaStreamSynchronize(ctx->stream));
  if (!g) note_graph(m, key);
  if (small) memcpy(out, ctx->h_out, ny * 4);
  return GN_OK;
}
static int forward_batch(gn_model* m, const float* x, int B, float* out) {
  GN_TRY(ensure_capacity(m, B, false));
  const int rc = forward_issue(m, x, B, out);
  if (rc != GN_OK) return drained(m, rc);
  Ctx* ctx = &m->ctx->c; int st; memcpy(&st, &ctx->h_ret[1], sizeof(int));
  return st != 0 ? clear_status(ctx, st) : GN_OK;
}

static int make_ctx(int device, int rank, int world, const unsigned char* id, gn_ctx** out) {
  if (!out) return fail(GN_ERR_INVALID_ARG, "out is null");
  int n = 0; cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) return fail(GN_ERR_NO_DEVICE, "no CUDA device: %s", cudaGetErrorString(e));
  if (device < 0 || device >= n) return fail(GN_ERR_INVALID_ARG, "device %d out of range [0,%d)", device, n);
  GN_CUDA(cudaSetDevice(device));
  cudaDeviceProp prop; GN_CUDA(cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10) return fail(GN_ERR_NO_DEVICE, "device %d is sm_%d%d; this library is built for sm_100a only", device, prop.major, prop.minor);
  // a context that fails half way releases what it already holds
  struct Guard { gn_ctx* c; ~Guard() { if (!c) return;
      if (c->c.comm && c->c.nccl) c->c.nccl->CommDestroy(c->c.comm);
      if (c->c.comm_stream) cudaStreamDestroy(c->c.comm_stream);
      if (c->c.d_status) cudaFree(c->c.d_status);
      if (c->c.h_block) cudaFreeHost(c->c.h_block);
      if (c->c.tc_queue_pool) cudaFree(c->c.tc_queue_pool);
      if (c->c.copy_ev) cudaEventDestroy(c->c.copy_ev);
      if (c->c.copy_stream) cudaStreamDestroy(c->c.copy_stream);
      if (c->c.fork_ev) cudaEventDestroy(c->c.fork_ev);
      if (c->c.join_ev) cudaEventDestroy(c->c.join_ev);
      if (c->c.side_stream) cudaStreamDestroy(c->c.side_stream);
      if (c->c.stream) cudaStreamDestroy(c->c.stream);
      delete c; } } guard{new gn_ctx()};
  gn_ctx* c = guard.c;
  c->c.device = device; c->c.rank = rank; c->c.world = world; c->c.sm_count = prop.multiProcessorCount;
  if (const char* e = getenv("GONEURON_CUDA_SM_RESERVE")) c->c.sm_reserve = std::max(0, std::min(atoi(e), prop.multiProcessorCount / 2));
  GN_CUDA(cudaStreamCreateWithFlags(&c->c.stream, cudaStreamNonBlocking));
  GN_CUDA(cudaStreamCreateWithFlags(&c->c.copy_stream, cudaStreamNonBlocking)); GN_CUDA(cudaEventCreateWithFlags(&c->c.copy_ev, cudaEventDisableTiming));
  GN_CUDA(cudaStreamCreateWithFlags(&c->c.side_stream, cudaStreamNonBlocking));
  GN_CUDA(cudaEventCreateWithFlags(&c->c.fork_ev, cudaEventDisableTiming)); GN_CUDA(cudaEventCreateWithFlags(&c->c.join_ev, cudaEventDisableTiming));
  GN_CUDA(cudaMalloc(&c->c.d_status, 4 * sizeof(int)));      // status word | ticket of the loss kernels | a scratch word
  GN_CUDA(cudaMemsetAsync(c->c.d_status, 0, 4 * sizeof(int), c->c.stream)); GN_CUDA(cudaStreamSynchronize(c->c.stream));
  GN_CUDA(cudaHostAlloc((void**)&c->c.h_block, (2 * STAGE_FLOATS + 64) * sizeof(float), cudaHostAllocMapped));
  c->c.h_ret = c->c.h_block; c->c.h_stage = c->c.h_block + 64; c->c.h_out = c->c.h_stage + STAGE_FLOATS;
  GN_CUDA(cudaHostGetDevicePointer((void**)&c->c.d_ret, c->c.h_ret, 0)); c->c.d_out = c->c.d_ret + (c->c.h_out - c->c.h_ret);
  tc_init(&c->c);
  if (world > 1) {
    NcclApi* api = nccl_api(); if (!api) return fail(GN_ERR_NCCL, "libnccl.so.2 could not be loaded");
    NcclUniqueId uid; memcpy(uid.internal, id, GN_UNIQUE_ID_BYTES);
    c->c.nccl = api;
    int rc = api->CommInitRank(&c->c.comm, world, uid, rank);
    if (rc) { c->c.comm = nullptr; return fail(GN_ERR_NCCL, "ncclCommInitRank: %s", api->GetErrorString(rc)); }
    GN_CUDA(cudaStreamCreateWithFlags(&c->c.comm_stream, cudaStreamNonBlocking));
  }
  guard.c = nullptr;
  DeviceMemory::get().count(device, 0, 1);
  DeviceMemory::get().streams(device, {c->c.stream, c->c.side_stream, c->c.copy_stream, c->c.comm_stream}, true);
  *out = c; return GN_OK;
}

}  // namespace gn

using namespace gn;

void gn_model::drop_graphs() { for (auto& g : graphs) g->drop(); graphs.clear(); }
gn_model::~gn_model() { drop_graphs(); }

#define CHECK_MODEL(m) do { if (!(m) || !(m)->alive) return fail(GN_ERR_INVALID_ARG, "model handle is null or destroyed"); } while (0)
#define USE_DEVICE(m) GN_CUDA(cudaSetDevice((m)->ctx->c.device))

extern "C" {

const char* gn_last_error(void) { return last_error().c_str(); }

int gn_init(int device, gn_ctx** out) { return make_ctx(device, 0, 1, nullptr, out); }

int gn_get_unique_id(unsigned char id[GN_UNIQUE_ID_BYTES]) {
  if (!id) return fail(GN_ERR_INVALID_ARG, "id is null");
  NcclApi* api = nccl_api(); if (!api) return fail(GN_ERR_NCCL, "libnccl.so.2 could not be loaded");
  NcclUniqueId uid; int rc = api->GetUniqueId(&uid); if (rc) return fail(GN_ERR_NCCL, "ncclGetUniqueId: %s", api->GetErrorString(rc));
  memcpy(id, uid.internal, GN_UNIQUE_ID_BYTES); return GN_OK;
}

int gn_init_rank(int device, int rank, int world_size, const unsigned char id[GN_UNIQUE_ID_BYTES], gn_ctx** out) {
  if (world_size < 1 || rank < 0 || rank >= world_size) return fail(GN_ERR_INVALID_ARG, "rank %d / world %d invalid", rank, world_size);
  if (world_size > 1 && !id) return fail(GN_ERR_INVALID_ARG, "id is null");
  return make_ctx(device, rank, world_size, id, out);
}

int gn_shutdown(gn_ctx* ctx) {
  if (!ctx || !ctx->alive) return GN_OK;
  cudaSetDevice(ctx->c.device);
  if (ctx->c.stream) cudaStreamSynchronize(ctx->c.stream);
  if (ctx->c.comm_stream) { cudaStreamSynchronize(ctx->c.comm_stream); }
  if (ctx->c.comm && ctx->c.nccl) ctx->c.nccl->CommDestroy(ctx->c.comm);
  for (auto& e : ctx->c.ev_pool) { cudaEventDestroy(e.first); cudaEventDestroy(e.second); }
  ctx->c.ev_pool.clear();
  ctx->c.release_owned();                               // operand-plane scratch of the contraction and attention engines
  DeviceMemory::get().streams(ctx->c.device, {ctx->c.stream, ctx->c.side_stream, ctx->c.copy_stream, ctx->c.comm_stream}, false);
  if (ctx->c.d_status) cudaFree(ctx->c.d_status);
  if (ctx->c.h_block) { cudaFreeHost(ctx->c.h_block); ctx->c.h_block = nullptr; }
  if (ctx->c.tc_queue_pool) { cudaFree(ctx->c.tc_queue_pool); ctx->c.tc_queue_pool = nullptr; }
  if (ctx->c.t0) { cudaEventDestroy(ctx->c.t0); cudaEventDestroy(ctx->c.t1); ctx->c.t0 = ctx->c.t1 = nullptr; }
  if (ctx->c.copy_ev) { cudaEventDestroy(ctx->c.copy_ev); ctx->c.copy_ev = nullptr; }
  if (ctx->c.copy_stream) { cudaStreamDestroy(ctx->c.copy_stream); ctx->c.copy_stream = nullptr; }
  if (ctx->c.fork_ev) { cudaEventDestroy(ctx->c.fork_ev); ctx->c.fork_ev = nullptr; }
  if (ctx->c.join_ev) { cudaEventDestroy(ctx->c.join_ev); ctx->c.join_ev = nullptr; }
  if (ctx->c.side_stream) { cudaStreamDestroy(ctx->c.side_stream); ctx->c.side_stream = nullptr; }
  if (ctx->c.stream) cudaStreamDestroy(ctx->c.stream);
  if (ctx->c.comm_stream) cudaStreamDestroy(ctx->c.comm_stream);
  ctx->c.comm_stream = nullptr;
  ctx->c.comm = nullptr; ctx->c.d_status = nullptr; ctx->c.stream = nullptr; ctx->alive = false;
  DeviceMemory::get().count(ctx->c.device, 0, -1);
  return GN_OK;   // the handle itself stays allocated so that a second call is harmless
}

int gn_ctx_world_size(gn_ctx* ctx, int* world_size, int* rank) {
  if (!ctx || !ctx->alive) return fail(GN_ERR_INVALID_ARG, "context is null or shut down");
  if (world_size) *world_size = ctx->c.world; if (rank) *rank = ctx->c.rank; return GN_OK;
}

int gn_ctx_set_spin_limit(gn_ctx* ctx, unsigned int polls) {
  if (!ctx || !ctx->alive) return fail(GN_ERR_INVALID_ARG, "context is null or shut down");
  ctx->c.spin_limit = polls == 0 ? TC_SPIN_LIMIT : polls; return GN_OK;
}

int gn_synchronize(gn_ctx* ctx) {
  if (!ctx || !ctx->alive) return fail(GN_ERR_INVALID_ARG, "context is null or shut down");
  GN_CUDA(cudaSetDevice(ctx->c.device)); GN_CUDA(cudaStreamSynchronize(ctx->c.stream)); return GN_OK;
}

int gn_timer_start(gn_ctx* ctx) {
  if (!ctx || !ctx->alive) return fail(GN_ERR_INVALID_ARG, "context is null or shut down");
  GN_CUDA(cudaSetDevice(ctx->c.device));
  if (!ctx->c.t0) { GN_CUDA(cudaEventCreate(&ctx->c.t0)); GN_CUDA(cudaEventCreate(&ctx->c.t1)); }
  GN_CUDA(cudaEventRecord(ctx->c.t0, ctx->c.stream)); return GN_OK;
}
int gn_timer_stop(gn_ctx* ctx, float* ms) {
  if (!ctx || !ctx->alive || !ms || !ctx->c.t0) return fail(GN_ERR_INVALID_ARG, "timer not started");
  GN_CUDA(cudaSetDevice(ctx->c.device));
  GN_CUDA(cudaEventRecord(ctx->c.t1, ctx->c.stream)); GN_CUDA(cudaEventSynchronize(ctx->c.t1));
  GN_CUDA(cudaEventElapsedTime(ms, ctx->c.t0, ctx->c.t1)); return GN_OK;
}

int gn_model_create(gn_ctx* ctx, const gn_layer_desc* layers, int n_layers, int loss_kind, int virtual_workers, gn_model** out) {
  if (!ctx || !ctx->alive) return fail(GN_ERR_INVALID_ARG, "context is null or shut down");
  if (!layers || n_layers <= 0 || !out) return fail(GN_ERR_INVALID_ARG, "layers/out is null or n_layers <= 0");
  if (loss_kind != GN_LOSS_MSE && loss_kind != GN_LOSS_CROSS_ENTROPY) return fail(GN_ERR_UNSUPPORTED, "loss kind %d", loss_kind);
  GN_CUDA(cudaSetDevice(ctx->c.device));
  std::unique_ptr<gn_model> m(new gn_model());
  m->ctx = ctx; m->loss_kind = loss_kind; m->W = virtual_workers < 1 ? 1 : virtual_workers;
  GN_TRY(plan_layers(m.get(), layers, n_layers));
  size_t P = (size_t)std::max<int64_t>(m->P, 4);
  GN_TRY(m->params.alloc(P)); GN_TRY(m->grads.alloc(P)); GN_TRY(m->m1.alloc(P)); GN_TRY(m->v2.alloc(P));
  // cudaMemset is asynchronous to the host and runs on the legacy default stream, which the context's non-blocking
  // stream does not wait for: a memset issued that way can land AFTER the first training step has written its
  // gradients (seen as all-zero LSTM gradients after the GPU had been idle).  So: the context's own stream, then wait.
  {
    cudaStream_t st = ctx->c.stream;
    GN_CUDA(cudaMemsetAsync(m->params.p, 0, P * 4, st)); GN_CUDA(cudaMemsetAsync(m->grads.p, 0, P * 4, st));
    GN_CUDA(cudaMemsetAsync(m->m1.p, 0, P * 4, st)); GN_CUDA(cudaMemsetAsync(m->v2.p, 0, P * 4, st));
    GN_CUDA(cudaStreamSynchronize(st));
  }
  if (ctx->c.tc_ok && !force_simt_engine() && !getenv("GONEURON_CUDA_NO_WEIGHT_PLANES")) {
    // weight matrices large enough to run on the tensor-core engine get prepared operand planes (both orientations)
    std::vector<WeightPlaneEntry> mats; int cur_layer = 0;
    auto add = [&](int64_t off, int out, int in, bool has_bias = true, int parts = 1, int64_t stride = 0) {      // (a stack's parts: multiples of 32 rows)
      if ((double)out * in < 64.0 * 64.0) return;
      WeightPlaneEntry e{m->params.p + off, parts * out, in, {}, {}, out, stride}; e.bias = has_bias ? m->params.p + off + (int64_t)out * in : nullptr; e.layer = cur_layer; mats.push_back(e);
    };
    for (auto& l : m->L) {
      const gn_layer_desc& d = l.d; cur_layer = (int)(&l - m->L.data());
      if (d.kind == GN_LAYER_DENSE) add(l.p_off, d.out_size, d.in_size);
      else if (d.kind == GN_LAYER_TRANSFORMER_BLOCK) {
        const int64_t dd = (int64_t)d.dim * d.dim + d.dim; int64_t o = l.p_off;
        if (d.dim % 32 == 0) { add(o, d.dim, d.dim, true, 3, dd); o += 3 * dd; } else for (int k = 0; k < 3; k++) { add(o, d.dim, d.dim); o += dd; }
        add(o, d.dim, d.dim); o += dd;
        o += (l.rms ? 2 : 4) * (int64_t)d.dim;
        if (l.ff_act == GN_ACT_SILU) {
          const int64_t df = (int64_t)d.dim * d.ff_dim;
          if (d.ff_dim % 32 == 0) add(o, d.ff_dim, d.dim, false, 2, df); else { add(o, d.ff_dim, d.dim, false); add(o + df, d.ff_dim, d.dim, false); }
          o += 2 * df;
        }
        else { add(o, d.ff_dim, d.dim); o += (int64_t)d.dim * d.ff_dim + d.ff_dim; }
        add(o, d.dim, d.ff_dim);
      }
    }
    GN_TRY(wplanes_build(&ctx->c, m->wplanes, mats));
  }
  if (m->NS > 0) {
    GN_TRY(m->state.alloc((size_t)m->NS));
    std::vector<float> init((size_t)m->NS, 0.f);     // running mean 0, running variance 1 (batchnorm2d.go:124-128)
    for (auto& l : m->L) if (l.d.kind == GN_LAYER_BATCHNORM2D) for (int64_t k = l.s_cnt / 2; k < l.s_cnt; k++) init[l.s_off + k] = 1.f;
    GN_CUDA(copy_h2d(&ctx->c, m->state.p, init.data(), (size_t)m->NS * 4));
  }
  GN_CUDA(cudaEventCreate(&m->ev0)); GN_CUDA(cudaEventCreate(&m->ev1)); GN_CUDA(cudaEventCreate(&m->ar0)); GN_CUDA(cudaEventCreate(&m->ar1));
  GN_CUDA(cudaEventCreateWithFlags(&m->comm_done, cudaEventDisableTiming)); GN_CUDA(cudaEventCreateWithFlags(&m->gather_ev, cudaEventDisableTiming));
  m->layer_ev.resize(m->L.size() + 1);
  for (auto& e : m->layer_ev) GN_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  m->scratch.resize(S_COUNT);
  DeviceMemory::get().count(ctx->c.device, 1, 0);
  *out = m.release(); return GN_OK;
}

int gn_model_destroy(gn_model* m) {
  if (!m || !m->alive) return GN_OK;
  std::lock_guard<std::mutex> lk(m->mu);
  cudaSetDevice(m->ctx->c.device);
  bool idle = true;
  if (m->ctx->alive) for (auto s : {m->ctx->c.stream, m->ctx->c.side_stream, m->ctx->c.copy_stream, m->ctx->c.comm_stream}) if (s) idle = cudaStreamSynchronize(s) == cudaSuccess && idle;
  if (m->ctx->c.weight_planes == &m->wplanes) m->ctx->c.weight_planes = nullptr;
  std::unique_ptr<DeviceMemory::Idle> waited(idle ? new DeviceMemory::Idle() : nullptr);
  m->wplanes = gn::WeightPlaneTable();
  m->drop_graphs();
  m->L.clear(); m->scratch.clear(); for (auto& b : m->shared) b.release(); m->state.release(); m->params.release(); m->grads.release(); m->m1.release(); m->v2.release();
  m->io.release(); m->lossg.release(); m->loss_s.release(); m->loss_sum.release();
  if (m->ev0) cudaEventDestroy(m->ev0); if (m->ev1) cudaEventDestroy(m->ev1); if (m->ar0) cudaEventDestroy(m->ar0); if (m->ar1) cudaEventDestroy(m->ar1);
  if (m->comm_done) cudaEventDestroy(m->comm_done); if (m->gather_ev) cudaEventDestroy(m->gather_ev); m->gather_ev = nullptr; for (auto e : m->layer_ev) cudaEventDestroy(e); m->layer_ev.clear();
  DeviceMemory::get().count(m->ctx->c.device, -1, 0);
  m->ev0 = m->ev1 = m->ar0 = m->ar1 = m->comm_done = nullptr; m->alive = false; return GN_OK;
}

int gn_model_param_count(gn_model* m, int64_t* n) { CHECK_MODEL(m); if (!n) return fail(GN_ERR_INVALID_ARG, "n is null"); *n = m->P; return GN_OK; }
int gn_model_in_size(gn_model* m, int64_t* n) { CHECK_MODEL(m); if (!n) return fail(GN_ERR_INVALID_ARG, "n is null"); *n = m->in_size; return GN_OK; }
int gn_model_out_size(gn_model* m, int64_t* n) { CHECK_MODEL(m); if (!n) return fail(GN_ERR_INVALID_ARG, "n is null"); *n = m->out_size; return GN_OK; }

int gn_model_set_params(gn_model* m, const float* host, int64_t n) {
  CHECK_MODEL(m); if (!host || n != m->P) return fail(GN_ERR_INVALID_ARG, "set_params: expected %lld floats, got %lld", (long long)m->P, (long long)n);
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(cudaMemcpyAsync(m->params.p, host, (size_t)n * 4, cudaMemcpyHostToDevice, m->ctx->c.stream));
  m->wplanes.dirty = true; m->wplanes.max_ok = false;
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream)); return GN_OK;
}
int gn_model_get_params(gn_model* m, float* host, int64_t n) {
  CHECK_MODEL(m); if (!host || n != m->P) return fail(GN_ERR_INVALID_ARG, "get_params: expected %lld floats, got %lld", (long long)m->P, (long long)n);
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(cudaMemcpyAsync(host, m->params.p, (size_t)n * 4, cudaMemcpyDeviceToHost, m->ctx->c.stream));
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream)); return GN_OK;
}
int gn_model_get_grads(gn_model* m, float* host, int64_t n) {
  CHECK_MODEL(m); if (!host || n != m->P) return fail(GN_ERR_INVALID_ARG, "get_grads: expected %lld floats, got %lld", (long long)m->P, (long long)n);
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(cudaMemcpyAsync(host, m->grads.p, (size_t)n * 4, cudaMemcpyDeviceToHost, m->ctx->c.stream));
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream));
  // the device keeps the batch-summed gradient; the 1/batch factor of net.go:702-706 is applied inside the Adam
  // pass and here, with the same float32 multiplication
  const float inv = m->last_inv_batch;
  for (int64_t i = 0; i < n; i++) host[i] *= inv;
  return GN_OK;
}

int gn_model_state_count(gn_model* m, int64_t* n) { CHECK_MODEL(m); if (!n) return fail(GN_ERR_INVALID_ARG, "n is null"); *n = m->NS; return GN_OK; }
int gn_model_get_state(gn_model* m, float* host, int64_t n) {
  CHECK_MODEL(m); if (n != m->NS || (n > 0 && !host)) return fail(GN_ERR_INVALID_ARG, "get_state: expected %lld floats, got %lld", (long long)m->NS, (long long)n);
  if (n == 0) return GN_OK;
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream)); GN_CUDA(copy_d2h(&m->ctx->c, host, m->state.p, (size_t)n * 4)); return GN_OK;
}
int gn_model_set_state(gn_model* m, const float* host, int64_t n) {
  CHECK_MODEL(m); if (n != m->NS || (n > 0 && !host)) return fail(GN_ERR_INVALID_ARG, "set_state: expected %lld floats, got %lld", (long long)m->NS, (long long)n);
  if (n == 0) return GN_OK;
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(cudaStreamSynchronize(m->ctx->c.stream)); GN_CUDA(copy_h2d(&m->ctx->c, m->state.p, host, (size_t)n * 4)); return GN_OK;
}

int gn_adam_set(gn_model* m, float lr, float beta1, float beta2, float eps, int timestep) {
  CHECK_MODEL(m); std::lock_guard<std::mutex> lk(m->mu);
  // zero betas / eps select the defaults, as Adam.StepInPlace does (opt.go:211-223)
  m->lr = lr; m->b1 = beta1 == 0.f ? 0.9f : beta1; m->b2 = beta2 == 0.f ? 0.999f : beta2; m->eps = eps == 0.f ? 1e-8f : eps;
  if (timestep >= 0) m->timestep = timestep; return GN_OK;
}
int gn_adam_get_state(gn_model* m, float* m1, float* v, int64_t n, int* timestep) {
  CHECK_MODEL(m); if (n != m->P) return fail(GN_ERR_INVALID_ARG, "adam state: expected %lld floats", (long long)m->P);
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  if (m1) GN_CUDA(copy_d2h(&m->ctx->c, m1, m->m1.p, (size_t)n * 4));
  if (v) GN_CUDA(copy_d2h(&m->ctx->c, v, m->v2.p, (size_t)n * 4));
  if (timestep) *timestep = m->timestep; return GN_OK;
}
int gn_adam_set_state(gn_model* m, const float* m1, const float* v, int64_t n, int timestep) {
  CHECK_MODEL(m); if (n != m->P || !m1 || !v) return fail(GN_ERR_INVALID_ARG, "adam state: expected %lld floats", (long long)m->P);
  std::lock_guard<std::mutex> lk(m->mu); USE_DEVICE(m);
  GN_CUDA(copy_h2d(&m->ctx->c, m->m1.p, m1, (size_t)n * 4)); GN_CUDA(copy_h2d(&m->ctx->c, m->v2.p, v, (size_t)n * 4));
  if (timestep >= 0) m->timestep = timestep; return GN_OK;
}

int gn_train_batch_device(gn_model* m, const float* x_dev, const float* y_dev, int batch, int global_batch, int first_sample, float* mean_loss) {
  CHECK_MODEL(m); if (!x_dev || !y_dev || batch <= 0) return fail(GN_ERR_INVALID_ARG, "train_batch: null input or batch <= 0");
  std::lock_guard<std::mutex> lk(m->mu); std::lock_guard<std::mutex> run_lk(m->ctx->c.run_mu); USE_DEVICE(m);
  return train_step(m, x_dev, y_dev, false, batch, global_batch, first_sample, mean_loss);
}

int gn_train_batch(gn_model* m, const float* x, const float* y, int batch, int global_batch, int first_sample, float* mean_loss) {
  CHECK_MODEL(m); if (!x || !y || batch <= 0) return fail(GN_ERR_INVALID_ARG, "train_batch: null input or batch <= 0");
  std::lock_guard<std::mutex> lk(m->mu); std::lock_guard<std::mutex> run_lk(m->ctx->c.run_mu); USE_DEVICE(m);
  return train_step(m, x, y, true, batch, global_batch, first_sample, mean_loss);
}

int gn_forward_batch(gn_model* m, const float* x, int batch, float* out) {
  CHECK_MODEL(m); if (!x || !out || batch <= 0) return fail(GN_ERR_INVALID_ARG, "forward_batch: null pointer or batch <= 0");
  std::lock_guard<std::mutex> lk(m->mu); std::lock_guard<std::mutex> run_lk(m->ctx->c.run_mu); USE_DEVICE(m);
  return forward_batch(m, x, batch, out);
}

int gn_device_alloc(gn_ctx* ctx, int64_t n, float** dev) {
  if (!ctx || !ctx->alive || !dev || n <= 0) return fail(GN_ERR_INVALID_ARG, "device_alloc: bad argument");
  GN_CUDA(cudaSetDevice(ctx->c.device)); cudaError_t e = cudaMalloc(dev, (size_t)n * 4);
  if (e != cudaSuccess) return fail(GN_ERR_OOM, "cudaMalloc(%lld floats): %s", (long long)n, cudaGetErrorString(e)); return GN_OK;
}
int gn_device_free(gn_ctx* ctx, float* dev) { if (!ctx || !ctx->alive) return GN_OK; cudaSetDevice(ctx->c.device); if (dev) cudaFree(dev); return GN_OK; }
int gn_device_upload(gn_ctx* ctx, float* dev, const float* host, int64_t n) {
  if (!ctx || !ctx->alive || !dev || !host) return fail(GN_ERR_INVALID_ARG, "device_upload: bad argument");
  GN_CUDA(cudaSetDevice(ctx->c.device)); GN_CUDA(cudaMemcpyAsync(dev, host, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->c.stream)); GN_CUDA(cudaStreamSynchronize(ctx->c.stream)); return GN_OK;
}
int gn_device_download(gn_ctx* ctx, float* host, const float* dev, int64_t n) {
  if (!ctx || !ctx->alive || !dev || !host) return fail(GN_ERR_INVALID_ARG, "device_download: bad argument");
  GN_CUDA(cudaSetDevice(ctx->c.device)); GN_CUDA(cudaMemcpyAsync(host, dev, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->c.stream)); GN_CUDA(cudaStreamSynchronize(ctx->c.stream)); return GN_OK;
}

int gn_model_last_stats(gn_model* m, gn_step_stats* out) { CHECK_MODEL(m); if (!out) return fail(GN_ERR_INVALID_ARG, "out is null");
  std::lock_guard<std::mutex> lk(m->mu);
  if (!m->stats_timed && m->stats.kernel_launches > 0) {      // event times are read when somebody asks for them
    cudaEventElapsedTime(&m->stats.step_ms, m->ev0, m->ev1);
    m->stats.allreduce_ms = 0.f; if (m->ctx->c.world > 1) cudaEventElapsedTime(&m->stats.allreduce_ms, m->ar0, m->ar1);
    m->stats_timed = true;
  }
  *out = m->stats; return GN_OK; }
int gn_model_set_profiling(gn_model* m, int level) { CHECK_MODEL(m); m->ctx->c.profile = level; return GN_OK; }

int gn_op_gemm_nt(gn_ctx* ctx, int engine, int M, int N, int K, const float* A, const float* B, const float* bias, float* C) {
  if (!ctx || !ctx->alive || !A || !B || !C || M <= 0 || N <= 0 || K <= 0) return fail(GN_ERR_INVALID_ARG, "op_gemm_nt: bad argument");
  Ctx* c = &ctx->c; std::lock_guard<std::mutex> run_lk(c->run_mu); GN_CUDA(cudaSetDevice(c->device));
  DevBuf dA, dB, dC, db; GN_TRY(dA.alloc((size_t)M * K)); GN_TRY(dB.alloc((size_t)N * K)); GN_TRY(dC.alloc((size_t)M * N)); if (bias) GN_TRY(db.alloc(N));
  GN_CUDA(cudaMemcpyAsync(dA.p, A, (size_t)M * K * 4, cudaMemcpyHostToDevice, c->stream)); GN_CUDA(cudaMemcpyAsync(dB.p, B, (size_t)N * K * 4, cudaMemcpyHostToDevice, c->stream));
  if (bias) GN_CUDA(cudaMemcpyAsync(db.p, bias, (size_t)N * 4, cudaMemcpyHostToDevice, c->stream));
  GemmDesc g; g.M = M; g.N = N; g.K = K; g.A = dA.p; g.sa_m = K; g.sa_k = 1; g.B = dB.p; g.sb_k = 1; g.sb_n = K; g.C = dC.p; g.ldc = N; g.bias = bias ? db.p : nullptr;
  if (engine == 1) { if (!gemm_tc_supported(c, g)) return fail(GN_ERR_UNSUPPORTED, "tcgen05 engine cannot run this shape (M=%d N=%d K=%d)", M, N, K); GN_TRY(gemm_tc(c, g)); }
  else GN_TRY(gemm_simt(c, g));
  GN_CUDA(cudaMemcpyAsync(C, dC.p, (size_t)M * N * 4, cudaMemcpyDeviceToHost, c->stream)); GN_CUDA(cudaStreamSynchronize(c->stream));
  return check_status_word(c);
}

int gn_op_adam(gn_ctx* ctx, float* params, const float* grads, float* m1, float* v, int64_t n, float lr, float beta1, float beta2, float eps, int t, float grad_scale) {
  if (!ctx || !ctx->alive || !params || !grads || !m1 || !v || n <= 0) return fail(GN_ERR_INVALID_ARG, "op_adam: bad argument");
  Ctx* c = &ctx->c; std::lock_guard<std::mutex> run_lk(c->run_mu); GN_CUDA(cudaSetDevice(c->device));
  DevBuf dp, dg, dm, dv; size_t nn = (size_t)n; GN_TRY(dp.alloc(nn + 4)); GN_TRY(dg.alloc(nn + 4)); GN_TRY(dm.alloc(nn + 4)); GN_TRY(dv.alloc(nn + 4));
  GN_CUDA(copy_h2d(c, dp.p, params, nn * 4)); GN_CUDA(copy_h2d(c, dg.p, grads, nn * 4));
  GN_CUDA(copy_h2d(c, dm.p, m1, nn * 4)); GN_CUDA(copy_h2d(c, dv.p, v, nn * 4));
  GN_TRY(adam_launch(c, dp.p, dg.p, dm.p, dv.p, n, adam_args(lr, beta1, beta2, eps, t, grad_scale), nullptr, nullptr, nullptr, nullptr, nullptr));
  GN_CUDA(cudaStreamSynchronize(c->stream));
  GN_CUDA(copy_d2h(c, params, dp.p, nn * 4)); GN_CUDA(copy_d2h(c, m1, dm.p, nn * 4)); GN_CUDA(copy_d2h(c, v, dv.p, nn * 4));
  return GN_OK;
}

int gn_op_attention(gn_ctx* ctx, int engine, int B, int T, int D, int H, int causal, const float* Q, const float* K, const float* V, const float* dO,
                    float* O, float* M, float* L, float* dQ, float* dK, float* dV) {
  if (!ctx || !ctx->alive || !Q || !K || !V || !O || B <= 0 || T <= 0 || D <= 0 || H <= 0 || D % H) return fail(GN_ERR_INVALID_ARG, "op_attention: bad argument");
  if (dO && (!dQ || !dK || !dV)) return fail(GN_ERR_INVALID_ARG, "op_attention: dO given without dQ, dK, dV");
  Ctx* c = &ctx->c; std::lock_guard<std::mutex> run_lk(c->run_mu); GN_CUDA(cudaSetDevice(c->device));
  const int hd = D / H; const size_t n = (size_t)B * T * D, ns = (size_t)B * H * T;
  if (!attn_fused_supported(hd, D)) return fail(GN_ERR_UNSUPPORTED, "op_attention: head size %d", hd);
  if (engine == 1 && !attn_tc_supported(c, hd, T, B, H, D)) return fail(GN_ERR_UNSUPPORTED, "tcgen05 attention cannot run this shape (head size %d, T=%d)", hd, T);
  const AtKernel pick = engine == 2 ? AT_ROWS : engine == 3 ? AT_HEAD : AT_AUTO;
  DevBuf q, k, v, o, m, l, g, dv_, dq, dk, dvv;
  GN_TRY(q.alloc(n)); GN_TRY(k.alloc(n)); GN_TRY(v.alloc(n)); GN_TRY(o.alloc(n)); GN_TRY(m.alloc(ns)); GN_TRY(l.alloc(ns));
  GN_CUDA(copy_h2d(c, q.p, Q, n * 4)); GN_CUDA(copy_h2d(c, k.p, K, n * 4)); GN_CUDA(copy_h2d(c, v.p, V, n * 4));
  if (engine == 1) GN_TRY(attn_tc_fwd(c, q.p, k.p, v.p, o.p, m.p, l.p, B, T, D, H, causal));
  else GN_TRY(attn_fwd(c, hd, q.p, k.p, v.p, o.p, m.p, l.p, B, T, D, H, causal, pick));
  if (dO) {
    GN_TRY(g.alloc(n)); GN_TRY(dv_.alloc(ns)); GN_TRY(dq.alloc(n)); GN_TRY(dk.alloc(n)); GN_TRY(dvv.alloc(n));
    GN_CUDA(copy_h2d(c, g.p, dO, n * 4));
    if (engine == 1) GN_TRY(attn_tc_bwd(c, q.p, k.p, v.p, o.p, g.p, m.p, l.p, dv_.p, dq.p, dk.p, dvv.p, B, T, D, H, causal));
    else GN_TRY(attn_bwd(c, hd, q.p, k.p, v.p, o.p, g.p, m.p, l.p, dq.p, dk.p, dvv.p, B, T, D, H, causal, pick));
    GN_CUDA(copy_d2h(c, dQ, dq.p, n * 4)); GN_CUDA(copy_d2h(c, dK, dk.p, n * 4)); GN_CUDA(copy_d2h(c, dV, dvv.p, n * 4));
  }
  GN_CUDA(copy_d2h(c, O, o.p, n * 4));
  if (M) GN_CUDA(copy_d2h(c, M, m.p, ns * 4));
  if (L) GN_CUDA(copy_d2h(c, L, l.p, ns * 4));
  return check_status_word(c);
}

}  // extern "C"

#include "gemm_static.cuh"
#include "ops_tier.cuh"
