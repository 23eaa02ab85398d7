// graph_rec.cuh -- a step put together as a CUDA graph, node by node.  Plain C++ over the runtime's graph calls.
#pragma once
#include <cuda_runtime_api.h>
#include <vector>

namespace gn {

// A run of launches and copies put together as a CUDA graph, node by node, while Ctx::rec points here: the helpers below then add a
// node behind what their stream holds so far instead of issuing the work.  (Capturing the stream gives the same graph but forbids
// other threads to synchronise the device, or to use the stream, for as long as it lasts -- theirs then fail, and the capture with
// them -- and a copy that another call queues meanwhile becomes part of it.)
struct GraphRec {
  cudaGraph_t graph = nullptr;
  bool* conditions = nullptr;                                 // may conditional nodes be made?  (null: yes); cleared where the driver refuses one
  struct Tail { cudaStream_t stream; std::vector<cudaGraphNode_t> nodes; bool kernel = false; };      // kernel: `nodes` is one kernel node
  std::vector<Tail> tails;
  GraphRec() {}
  GraphRec(const GraphRec&) = delete; GraphRec& operator=(const GraphRec&) = delete;
  ~GraphRec() { if (graph) cudaGraphDestroy(graph); }
  Tail& tail(cudaStream_t s) { for (auto& t : tails) if (t.stream == s) return t; tails.push_back(Tail{s, {}}); return tails.back(); }
  // what `from` holds so far comes before everything that `to` gets from now on
  void join(cudaStream_t to, cudaStream_t from) {
    const std::vector<cudaGraphNode_t> add = tail(from).nodes; Tail& t = tail(to);
    for (auto n : add) { bool have = false; for (auto q : t.nodes) have |= q == n; if (!have) { t.nodes.push_back(n); t.kernel = t.kernel && t.nodes.size() == 1; } }
  }
  template <class F> cudaError_t add(cudaStream_t s, bool kernel, F&& make) {      // make(node, dependencies, their number)
    Tail& t = tail(s); cudaGraphNode_t node;
    const cudaError_t e = make(&node, t.nodes.data(), t.nodes.size());
    if (e == cudaSuccess) { t.nodes.assign(1, node); t.kernel = kernel; }
    return e;
  }
  // Work on stream `s` that a replay leaves out unless a kernel before it has set `handle` to a non-zero value.  condition() is false, and the work is to be
  // recorded without one, where a driver does not make them; a driver that refuses the node behind the handle, or the graph with it, fails this recording
  // and the next goes without (record_graph).
  bool conditional = false;                                   // a handle has been made
  bool condition(cudaGraphConditionalHandle* handle) {
    if (conditions && !*conditions) return false;
    if (cudaGraphConditionalHandleCreate(handle, graph, 0, cudaGraphCondAssignDefault) != cudaSuccess) { cudaGetLastError(); if (conditions) *conditions = false; return false; }
    return conditional = true;
  }
  template <class F> cudaError_t only_if(cudaStream_t s, cudaGraphConditionalHandle handle, F&& body) {
    cudaGraphNodeParams p{}; p.type = cudaGraphNodeTypeConditional; p.conditional.handle = handle; p.conditional.type = cudaGraphCondTypeIf; p.conditional.size = 1;
    const cudaError_t e = add(s, false, [&](cudaGraphNode_t* node, const cudaGraphNode_t* deps, size_t n) { return cudaGraphAddNode(node, graph, deps, n, &p); });
    if (e != cudaSuccess) { if (conditions) *conditions = false; return e; }
    cudaGraph_t outer = graph; std::vector<Tail> outer_tails; outer_tails.swap(tails);
    graph = p.conditional.phGraph_out[0];                     // (belongs to the node)
    body();
    graph = outer; tails.swap(outer_tails); return cudaSuccess;
  }
};

// What `issue` (true: complete) records while `current` points to the recording, as an executable graph; null where that cannot be made.
// `conditions` outlives the recordings of a context.  A graph with conditional nodes that is refused for another reason than memory clears it.
template <class F> inline cudaGraphExec_t record_graph(GraphRec*& current, bool& conditions, F&& issue) {
  GraphRec rec; rec.conditions = &conditions; cudaGraphExec_t out = nullptr;
  if (cudaGraphCreate(&rec.graph, 0) != cudaSuccess) { rec.graph = nullptr; return nullptr; }
  current = &rec;
  struct Guard { GraphRec*& c; ~Guard() { c = nullptr; } } guard{current};
  if (!issue()) return nullptr;
  const cudaError_t e = cudaGraphInstantiate(&out, rec.graph, 0);
  if (e == cudaSuccess) return out;
  if (rec.conditional && e != cudaErrorMemoryAllocation) conditions = false;
  return nullptr;
}

}  // namespace gn
