"""Recorded steps on the CPU, with fakes of the runtime's graph calls that refuse: a driver that does not make conditional nodes costs the condition, not the
recording."""
import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r'''
#include <cstdio>
#include <cstring>
#include "goneuron_b200/csrc/graph_rec.cuh"
using namespace gn;
static int refuse = 0, conditional = 0, kernels = 0, graphs = 0;      // refuse: 1 the handle, 2 the node, 3 the finished graph, 4 it, for lack of memory
extern "C" {
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) { *g = (cudaGraph_t)(size_t)++graphs; conditional = kernels = 0; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { graphs--; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) { if (refuse == 1) return cudaErrorNotSupported; *h = 7; return cudaSuccess; }
static cudaGraph_t body = (cudaGraph_t)99;
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
  if (refuse == 2) return cudaErrorNotSupported;
  conditional++; *n = (cudaGraphNode_t)1; p->conditional.phGraph_out = &body; return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  if (conditional && refuse == 3) return cudaErrorNotSupported;
  if (refuse == 4) return cudaErrorMemoryAllocation;
  *x = (cudaGraphExec_t)5; return cudaSuccess;
}
}
int main() {
  GraphRec* rec = nullptr; int bad = 0;
  auto launch = [&] { rec->add(nullptr, true, [&](cudaGraphNode_t* n, const cudaGraphNode_t*, size_t) { kernels++; *n = (cudaGraphNode_t)2; return cudaSuccess; }); };
  auto step = [&]() -> bool {                                 // ten launches, eight of them behind a condition where there is one
    cudaGraphConditionalHandle h = 0; const bool skip = rec->condition(&h); bool ok = true;
    launch();
    if (skip) ok = rec->only_if(nullptr, h, [&] { for (int i = 0; i < 8; i++) launch(); }) == cudaSuccess; else for (int i = 0; i < 8; i++) launch();
    launch(); return ok;
  };
  auto check = [&](const char* what, bool is) { if (!is) { bad++; std::printf("%s (refuse %d)\n", what, refuse); } };
  for (refuse = 0; refuse <= 4; refuse++) {
    bool conditions = true;
    cudaGraphExec_t first = record_graph(rec, conditions, step);
    check("recorded at once", (first != nullptr) == (refuse < 2));
    check("conditional nodes of the first", conditional == (refuse == 1 || refuse == 2 ? 0 : 1));
    check("what is remembered", conditions == (refuse == 0 || refuse == 4));
    check("left alone", rec == nullptr && graphs == 0);
    if (refuse == 4) refuse = -4;                             // (there is memory again)
    cudaGraphExec_t second = record_graph(rec, conditions, step);
    if (refuse == -4) refuse = 4;
    check("recorded in the end", second != nullptr && kernels == 10);
    check("conditional nodes of the second", conditional == (refuse == 0 || refuse == 4 ? 1 : 0));
  }
  bool conditions = true;
  check("an incomplete step", record_graph(rec, conditions, [&]() -> bool { step(); return false; }) == nullptr && rec == nullptr && conditions);
  return bad;
}
'''


def test_a_driver_without_conditional_nodes_costs_the_condition_only():
    include = os.path.join(CUDA, "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(SRC)
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", ROOT, "-I", include, src, "-o", exe])
        r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stdout
