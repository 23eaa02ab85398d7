// common.cuh -- context, error handling and launch bookkeeping shared by all kernels.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <cstdlib>
#include <initializer_list>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/goneuron_cuda.h"
#include "graph_rec.cuh"

namespace gn {

// Per-thread message of the most recent failure (gn_last_error()).
inline std::string& last_error() { thread_local std::string e; return e; }
inline int fail(int code, const char* fmt, ...) {
  char buf[1024]; va_list ap; va_start(ap, fmt); vsnprintf(buf, sizeof buf, fmt, ap); va_end(ap);
  last_error() = buf; return code;
}

#define GN_CUDA(call)                                                                        \
  do { cudaError_t e_ = (call); if (e_ != cudaSuccess)                                       \
      return gn::fail(e_ == cudaErrorMemoryAllocation ? GN_ERR_OOM : GN_ERR_CUDA, "%s failed at %s:%d: %s", #call, __FILE__, __LINE__, cudaGetErrorString(e_)); } while (0)
#define GN_TRY(call) do { int rc_ = (call); if (rc_ != GN_OK) return rc_; } while (0)

struct NcclApi;   // resolved at run time from libnccl.so.2 (nccl_dl.cuh)

struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t comm_stream = nullptr;   // gradient all-reduces run here, overlapped with the rest of the backward pass
  cudaStream_t copy_stream = nullptr; cudaEvent_t copy_ev = nullptr;      // targets of a large host batch, copied under the forward pass
  cudaStream_t side_stream = nullptr; cudaEvent_t fork_ev = nullptr, join_ev = nullptr; bool side_pending = false;      // see side_run()
  int rank = 0, world = 1;
  void* comm = nullptr;            // ncclComm_t
  NcclApi* nccl = nullptr;
  int sm_count = 148;
  int sm_reserve = 0;              // SMs the persistent kernels leave free (for the collectives' CTAs when several ranks run); see persist_sms()
  int64_t launches = 0;            // kernels launched by this library on this context
  // contraction profiling (gn_model_set_profiling)
  int profile = 0;
  double gemm_flops = 0; float gemm_ms = 0; int64_t gemm_launches = 0;
  double gemm_bytes = 0, split_bytes = 0;   // algorithmic bytes of the step's contraction launches (operand planes + output + residual) / of its operand split passes
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_pool; size_t ev_used = 0;
  int* d_status = nullptr;         // device word set by kernels whose bounded waits gave up
  // pinned host memory of the context's calls (they run one at a time): results (loss sum | status word bits), a block for small
  // inputs, one for small outputs; d_ret / d_out: the device's addresses
  float *h_block = nullptr, *h_ret = nullptr, *h_stage = nullptr, *h_out = nullptr, *d_ret = nullptr, *d_out = nullptr;
  uint64_t epoch = 0;              // counts replacements of the context's scratch buffers
  GraphRec* rec = nullptr;         // set while a step is put together as a graph instead of being issued
  bool graph_conditions = true;    // conditional graph nodes can be made (until one is refused)
  bool tc_ok = false;              // tcgen05 engine usable (driver entry point for tensor maps found)
  void* encode_tiled = nullptr;    // cuTensorMapEncodeTiled
  unsigned spin_limit = 1u << 24;  // polls per bounded device-side wait (gn_ctx_set_spin_limit)
  bool tc_tile_queue = false;      // persistent contraction draws its tiles from a queue instead of a fixed share per CTA (GONEURON_CUDA_TC_TILE_QUEUE)
  int* tc_queue_pool = nullptr; int tc_queue_used = 0;      // zeroed counters for those queues
  bool tc_tail_split = true;       // left-over tiles of a short last round run as half tiles (GONEURON_CUDA_TC_TAIL_SPLIT=0 switches it off)
  int tc_force_bn = 0, tc_kslice = 0;   // experiment switches of the contraction engine (GONEURON_CUDA_TC_BN / _KSLICE); 0 = automatic
  void* tc_scratch = nullptr;      // operand planes of the contraction engine (TcScratch, owned)
  void* attn_scratch = nullptr;    // operand planes of the tcgen05 attention kernels (AttnTcScratch, owned)
  void* weight_planes = nullptr;         // the running model's table of prepared weight planes (WeightPlaneTable), or null
  std::mutex run_mu;               // serialises every entry point that launches work on this context (they share the scratch above)
  cudaEvent_t t0 = nullptr, t1 = nullptr;   // gn_timer_start / gn_timer_stop
  // Scratch objects created on demand for this context (operand planes of the contraction and attention engines),
  // all released by gn_shutdown.
  std::vector<std::pair<void*, void (*)(void*)>> owned; std::mutex owned_mu;
  template <class T> T* own(T* p) { std::lock_guard<std::mutex> lk(owned_mu); owned.push_back({p, [](void* q) { delete static_cast<T*>(q); }}); return p; }
  void release_owned() { std::lock_guard<std::mutex> lk(owned_mu); for (auto& e : owned) e.second(e.first); owned.clear(); }
};

inline unsigned cdiv(long a, long b) { return (unsigned)((a + b - 1) / b); }

// Runs `f` (launches on ctx->stream) on the side stream, beside what the main stream does next.  A parameter gradient is read by nothing
// before the update, while the gradient of the layer's input is the one thing the next layer waits for: a step of small
// kernels is a chain of those, and the parameter gradients need not be links of it.  `f` must not use the contraction
// engine's scratch or any buffer that the main stream writes before side_join(), which the backward pass calls after every layer.
template <class F> inline int side_run(Ctx* ctx, F&& f) {
  if (!ctx->side_stream || ctx->profile) return f();         // (profiling times the contractions one by one)
  if (ctx->rec) ctx->rec->join(ctx->side_stream, ctx->stream);
  else if (cudaEventRecord(ctx->fork_ev, ctx->stream) != cudaSuccess || cudaStreamWaitEvent(ctx->side_stream, ctx->fork_ev, 0) != cudaSuccess)
    return fail(GN_ERR_CUDA, "side stream: %s", cudaGetErrorString(cudaGetLastError()));
  cudaStream_t main = ctx->stream; ctx->stream = ctx->side_stream; ctx->side_pending = true;
  const int rc = f();
  ctx->stream = main; return rc;
}
inline int side_join(Ctx* ctx) {
  if (!ctx->side_pending) return GN_OK;
  ctx->side_pending = false;
  if (ctx->rec) { ctx->rec->join(ctx->stream, ctx->side_stream); return GN_OK; }
  if (cudaEventRecord(ctx->join_ev, ctx->side_stream) != cudaSuccess || cudaStreamWaitEvent(ctx->stream, ctx->join_ev, 0) != cudaSuccess)
    return fail(GN_ERR_CUDA, "side stream: %s", cudaGetErrorString(cudaGetLastError()));
  return GN_OK;
}

// Every kernel launch of the library goes through these macros, so that all are counted and a step can be recorded.  (A replayed step counts what was
// recorded, launches behind a condition among them whether they ran or not.)
// launch_kernel(): `cluster` > 0: that many neighbouring blocks of the grid's x dimension form a thread-block cluster; `early`: the
// blocks may be placed while the preceding kernel still runs (programmatic stream serialisation), which wants a kernel that calls
// pdl_wait() in every block before it touches anything its predecessors write, and pdl_launch() to let its own successor in.
// (Launching every kernel of a step that way, waiting at its first instruction, was measured: within a replayed graph it is
// slower than the ordinary edge, 78 -> 85 us for a step of 15 launches.  It pays where a kernel has something to fetch first.)
template <class... P, class... A>
inline cudaError_t launch_kernel(Ctx* ctx, cudaStream_t stream, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, int cluster, bool early, A&&... args) {
  ctx->launches++;
  if (ctx->rec) {
    GraphRec& rec = *ctx->rec;
    return rec.add(stream, true, [&](cudaGraphNode_t* node, const cudaGraphNode_t* deps, size_t n) -> cudaError_t {
      const bool edge = early && rec.tail(stream).kernel;
      auto make = [&](P... values) {
        void* pointers[] = {(void*)&values..., nullptr};
        cudaKernelNodeParams p{}; p.func = (void*)kernel; p.gridDim = grid; p.blockDim = block; p.sharedMemBytes = (unsigned)smem; p.kernelParams = pointers;
        return cudaGraphAddKernelNode(node, rec.graph, edge ? nullptr : deps, edge ? 0 : n, &p);
      };
      cudaError_t e = make(static_cast<P>(args)...);
      if (e == cudaSuccess && cluster > 0) {
        cudaLaunchAttributeValue v{}; v.clusterDim.x = cluster; v.clusterDim.y = v.clusterDim.z = 1;
        e = cudaGraphKernelNodeSetAttribute(*node, cudaLaunchAttributeClusterDimension, &v);
      }
      if (e == cudaSuccess && edge) {
        cudaGraphEdgeData d{}; d.from_port = cudaGraphKernelNodePortProgrammatic; d.type = cudaGraphDependencyTypeProgrammatic;
        e = cudaGraphAddDependencies_v2(rec.graph, deps, node, &d, 1);
      }
      return e;
    });
  }
  cudaLaunchConfig_t cfg{}; cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute at[2]; int n = 0;
  if (early) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n++].val.programmaticStreamSerializationAllowed = 1; }
  if (cluster > 0) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1; n++; }
  cfg.attrs = at; cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
// (an error of the first two is seen by the check_launch() behind them)
#define GN_LAUNCH(ctx, kernel, grid, block, smem, ...) GN_LAUNCH_ON(ctx, (ctx)->stream, kernel, grid, block, smem, __VA_ARGS__)
#define GN_LAUNCH_ON(ctx, stream, kernel, grid, block, smem, ...)              \
  do { (void)gn::launch_kernel(ctx, stream, kernel, dim3(grid), dim3(block), (size_t)(smem), 0, false, __VA_ARGS__); } while (0)
#define GN_CLUSTER_LAUNCH(ctx, kernel, grid, block, smem, cx, ...)             \
  do { GN_CUDA(gn::launch_kernel(ctx, (ctx)->stream, kernel, dim3(grid), dim3(block), (size_t)(smem), cx, false, __VA_ARGS__)); } while (0)
#define GN_EARLY_LAUNCH(ctx, kernel, grid, block, smem, ...)                   \
  do { GN_CUDA(gn::launch_kernel(ctx, (ctx)->stream, kernel, dim3(grid), dim3(block), (size_t)(smem), 0, true, __VA_ARGS__)); } while (0)
// `bytes` zeros at p / a copy, in stream order
inline cudaError_t stream_zero(Ctx* ctx, cudaStream_t stream, void* p, size_t bytes) {
  if (!ctx->rec) return cudaMemsetAsync(p, 0, bytes, stream);
  const unsigned es = ((uintptr_t)p | bytes) % 4 == 0 ? 4 : 1;
  cudaMemsetParams mp{}; mp.dst = p; mp.elementSize = es; mp.width = bytes / es; mp.height = 1;
  return ctx->rec->add(stream, false, [&](cudaGraphNode_t* node, const cudaGraphNode_t* deps, size_t n) { return cudaGraphAddMemsetNode(node, ctx->rec->graph, deps, n, &mp); });
}
inline cudaError_t stream_zero(Ctx* ctx, void* p, size_t bytes) { return stream_zero(ctx, ctx->stream, p, bytes); }
inline cudaError_t stream_copy(Ctx* ctx, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
  if (!ctx->rec) return cudaMemcpyAsync(dst, src, bytes, kind, ctx->stream);
  return ctx->rec->add(ctx->stream, false, [&](cudaGraphNode_t* node, const cudaGraphNode_t* deps, size_t n) { return cudaGraphAddMemcpyNode1D(node, ctx->rec->graph, deps, n, dst, src, bytes, kind); });
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(GN_ERR_CUDA, "kernel launch failed (%s): %s", what, cudaGetErrorString(e));
  return GN_OK;
}

// Host <-> device copies always go through the context's own stream and wait for it.  (The synchronous cudaMemcpy /
// cudaMemset run on the legacy default stream, which a non-blocking stream does not wait for, and may return before
// the transfer has landed: work issued that way can overtake, or be overtaken by, kernels of the context's stream.)
inline cudaError_t copy_h2d(Ctx* c, void* dst, const void* src, size_t bytes) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream); return e != cudaSuccess ? e : cudaStreamSynchronize(c->stream);
}
inline cudaError_t copy_d2h(Ctx* c, void* dst, const void* src, size_t bytes) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream); return e != cudaSuccess ? e : cudaStreamSynchronize(c->stream);
}

// Contraction profiling (gn_model_set_profiling): one CUDA-event pair around each contraction KERNEL launch (the operand
// split passes are separate, memory-bound kernels and are not inside the bracket).
struct ProfScope {
  Ctx* c; cudaEvent_t e1 = nullptr;
  explicit ProfScope(Ctx* ctx) : c(ctx) {
    if (!c->profile) return;
    if (c->ev_used == c->ev_pool.size()) { cudaEvent_t a, b; if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return; c->ev_pool.push_back({a, b}); }
    cudaEventRecord(c->ev_pool[c->ev_used].first, c->stream); e1 = c->ev_pool[c->ev_used].second; c->ev_used++;
  }
  ~ProfScope() { if (e1) cudaEventRecord(e1, c->stream); }
};

// Device memory of the library's buffers comes from one CUDA memory pool per GPU.  While a model lives there the pool keeps up to
// keep_limit() bytes of what models and scratch buffers have released (a model of the same size created later gets it back without
// going to the driver: Compile and first pass of a causal Transformer of width 256 take 0.2 and 1.4 ms instead of 1.9 and 9 with
// cudaMalloc); the rest, and everything once the GPU's last model or context is closed, goes back to the driver.
// (A list of cudaMalloc blocks by size, and parts of 128 MiB blocks, were as quick to prepare, but steps ran 0.4 to 1.4 % slower in them.)
// An allocation is usable on every stream when take() returns.  put() hands memory on only after every stream of the library on the GPU
// has finished what it held, as cudaFree waits for the device.  Not cudaDeviceSynchronize: that fails while any other thread has
// a stream in capture.  The pool's own stream orders its allocations and releases; nothing else runs there.
struct DeviceMemory {
  static constexpr int MAX = 64;
  struct Gpu { std::mutex mu; cudaMemPool_t pool = nullptr; cudaStream_t stream = nullptr; int models = 0, contexts = 0; std::vector<cudaStream_t> streams; };
  Gpu gpu[MAX];
  static DeviceMemory& get() { static DeviceMemory* p = new DeviceMemory(); return *p; }      // (lives until the process ends)
  static unsigned long long keep_limit() {
    static const unsigned long long n = [] { const char* e = getenv("GONEURON_CUDA_KEEP_BYTES"); return e ? strtoull(e, nullptr, 10) : 8ull << 30; }();
    return n;
  }
  // The functions below want `dev` to be the current device.
  static void set_keep(Gpu& g) { unsigned long long n = g.models > 0 && g.contexts > 0 ? keep_limit() : 0; cudaMemPoolSetAttribute(g.pool, cudaMemPoolAttrReleaseThreshold, &n); }
  static void trim(Gpu& g) { if (g.pool) { cudaStreamSynchronize(g.stream); cudaMemPoolTrimTo(g.pool, 0); } }
  static cudaError_t open(Gpu& g, int dev) {
    if (g.pool) return cudaSuccess;
    cudaMemPoolProps pr{}; pr.allocType = cudaMemAllocationTypePinned; pr.location.type = cudaMemLocationTypeDevice; pr.location.id = dev;
    cudaError_t e = g.stream ? cudaSuccess : cudaStreamCreateWithFlags(&g.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemPoolCreate(&g.pool, &pr);
    if (e != cudaSuccess) { g.pool = nullptr; return e; }
    set_keep(g); return cudaSuccess;
  }
  cudaError_t take(int dev, size_t bytes, void** p) {
    if (dev < 0 || dev >= MAX) return cudaErrorInvalidDevice;
    Gpu& g = gpu[dev]; std::lock_guard<std::mutex> lk(g.mu);
    cudaError_t e = open(g, dev);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, g.pool, g.stream);
    if (e == cudaErrorMemoryAllocation && g.pool) { cudaGetLastError(); trim(g); e = cudaMallocFromPoolAsync(p, bytes, g.pool, g.stream); }
    return e != cudaSuccess ? e : cudaStreamSynchronize(g.stream);
  }
  void put(int dev, void* p, bool idle) {                    // idle: the caller has waited for everything that uses the memory
    Gpu& g = gpu[dev]; std::lock_guard<std::mutex> lk(g.mu);
    if (!idle) for (auto s : g.streams) if (cudaStreamSynchronize(s) != cudaSuccess) return;      // (a broken context: nobody gets this memory any more)
    cudaFreeAsync(p, g.stream);
    if (g.models <= 0) cudaStreamSynchronize(g.stream);      // (where the pool gives back what it need not keep)
  }
  void count(int dev, int d_models, int d_contexts) {
    if (dev < 0 || dev >= MAX) return;
    Gpu& g = gpu[dev]; std::lock_guard<std::mutex> lk(g.mu);
    g.models += d_models; g.contexts += d_contexts;
    if (g.pool) set_keep(g);
    if (g.models <= 0 || g.contexts <= 0) trim(g);
  }
  void streams(int dev, std::initializer_list<cudaStream_t> list, bool there) {
    if (dev < 0 || dev >= MAX) return;
    Gpu& g = gpu[dev]; std::lock_guard<std::mutex> lk(g.mu);
    for (auto s : list) if (s) { if (there) g.streams.push_back(s); else g.streams.erase(std::remove(g.streams.begin(), g.streams.end(), s), g.streams.end()); }
  }
  // While one of these lives, buffers that its thread releases are known to be idle.
  struct Idle { static int& depth() { thread_local int d = 0; return d; } Idle() { depth()++; } ~Idle() { depth()--; } };
};

// Owning device buffer, or a view of part of another one.
struct DevBuf {
  float* p = nullptr; size_t n = 0; bool owner = true; int dev = 0;
  DevBuf() {}
  DevBuf(const DevBuf&) = delete; DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), owner(o.owner), dev(o.dev) { o.p = nullptr; o.n = 0; }
  DevBuf& operator=(DevBuf&& o) noexcept { release(); p = o.p; n = o.n; owner = o.owner; dev = o.dev; o.p = nullptr; o.n = 0; return *this; }
  ~DevBuf() { release(); }
  void release() {
    if (p && owner) {
      int cur = dev; cudaGetDevice(&cur);
      if (cur != dev) cudaSetDevice(dev);
      DeviceMemory::get().put(dev, p, DeviceMemory::Idle::depth() > 0);
      if (cur != dev) cudaSetDevice(cur);
    }
    p = nullptr; n = 0; owner = true;
  }
  void view(float* q, size_t count) { release(); p = q; n = count; owner = false; }
  int alloc(size_t count) {
    release(); if (count == 0) return GN_OK;
    cudaGetDevice(&dev);
    const cudaError_t e = DeviceMemory::get().take(dev, count * sizeof(float), (void**)&p);
    if (e != cudaSuccess) { cudaGetLastError(); p = nullptr; return fail(GN_ERR_OOM, "device allocation of %zu bytes failed: %s", count * sizeof(float), cudaGetErrorString(e)); }
    n = count; return GN_OK;
  }
};

// Asynchronous copies into shared memory (4 bytes; `ok` false: zero fill without reading; 16 bytes), and the wait for a thread's own.
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool ok = true) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async16_part(float* dst, const float* src, int n) {      // n floats from src, zeros behind them
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(4 * n) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum / max; every thread receives the result.  `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) { float t = lane < nw ? red[lane] : 0.f; t = warp_sum(t); if (lane == 0) red[32] = t; }
  __syncthreads();
  return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) { float t = lane < nw ? red[lane] : -INFINITY; t = warp_max(t); if (lane == 0) red[32] = t; }
  __syncthreads();
  return red[32];
}

}  // namespace gn
