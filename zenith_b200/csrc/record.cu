// Launches into a stream or into a recording, and the recorded graphs (see launch.cuh).
#include "launch.cuh"
#include "../../include/zenith_b200.h"

namespace zen {

// What a thread records: a graph whose nodes follow one another within a branch.
struct Recording {
  cudaGraph_t graph;     // null: this thread does not record
  cudaGraphNode_t tail;  // last node of the branch, null in front of its first
  bool ok;
};
static thread_local Recording t_recording = {nullptr, nullptr, true};

bool recording() { return t_recording.graph != nullptr; }

// The node's edge is what the same two launches in a stream would get: full completion, or for an early launch the
// programmatic one (the kernel in front has released its dependents in every CTA).
static cudaError_t add_node(Recording& r, const void* kernel, const LaunchShape& sh, void** args) {
  cudaKernelNodeParams p = {};
  p.func = const_cast<void*>(kernel);
  p.gridDim = sh.grid;
  p.blockDim = sh.block;
  p.sharedMemBytes = unsigned(sh.smem);
  p.kernelParams = args;
  cudaGraphNode_t node;
  if (cudaError_t e = cudaGraphAddKernelNode(&node, r.graph, nullptr, 0, &p); e != cudaSuccess) return e;
  if (sh.cluster > 1) {
    cudaLaunchAttributeValue v = {};
    v.clusterDim.x = sh.cluster;
    v.clusterDim.y = 1;
    v.clusterDim.z = 1;
    if (cudaError_t e = cudaGraphKernelNodeSetAttribute(node, cudaLaunchAttributeClusterDimension, &v); e != cudaSuccess) return e;
  }
  if (r.tail != nullptr) {
    cudaGraphEdgeData edge = {};
    if (sh.early) {
      edge.from_port = cudaGraphKernelNodePortProgrammatic;
      edge.type = cudaGraphDependencyTypeProgrammatic;
    }
    if (cudaError_t e = cudaGraphAddDependencies_v2(r.graph, &r.tail, &node, &edge, 1); e != cudaSuccess) return e;
  }
  r.tail = node;
  return cudaSuccess;
}

int launch_args(const void* kernel, const LaunchShape& sh, cudaStream_t stream, void** args) {
  cudaError_t e;
  if (recording()) {
    e = add_node(t_recording, kernel, sh, args);
    t_recording.ok = t_recording.ok && e == cudaSuccess;
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = sh.grid;
    cfg.blockDim = sh.block;
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    if (sh.early) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (sh.cluster > 1) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attr[cfg.numAttrs].val.clusterDim.x = sh.cluster;
      attr[cfg.numAttrs].val.clusterDim.y = 1;
      attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    e = cudaLaunchKernelExC(&cfg, kernel, args);
  }
  if (e == cudaSuccess) return ZEN_OK;
  cudaGetLastError();
  return ZEN_ERR_LAUNCH;
}

}  // namespace zen

using namespace zen;

extern "C" {

int zen_record_begin(void) {
  if (recording()) return ZEN_ERR_INVALID_ARG;
  cudaGraph_t g = nullptr;
  if (cudaGraphCreate(&g, 0) != cudaSuccess) {
    cudaGetLastError();
    return ZEN_ERR_LAUNCH;
  }
  t_recording = {g, nullptr, true};
  return ZEN_OK;
}

int zen_record_branch(void) {
  if (!recording()) return ZEN_ERR_INVALID_ARG;
  t_recording.tail = nullptr;
  return ZEN_OK;
}

int zen_record_end(void** graph_host) {
  if (!recording()) return ZEN_ERR_INVALID_ARG;
  const Recording r = t_recording;
  t_recording = {nullptr, nullptr, true};
  int st = r.ok ? ZEN_OK : ZEN_ERR_LAUNCH;
  cudaGraphExec_t exec = nullptr;
  if (st == ZEN_OK && graph_host != nullptr && cudaGraphInstantiate(&exec, r.graph, 0) != cudaSuccess) st = ZEN_ERR_LAUNCH;
  cudaGraphDestroy(r.graph);
  cudaGetLastError();
  if (graph_host != nullptr) *graph_host = st == ZEN_OK ? exec : nullptr;
  return st;
}

int zen_graph_launch(void* graph, void* stream) {
  if (graph == nullptr) return ZEN_ERR_INVALID_ARG;
  if (recording()) return ZEN_ERR_UNSUPPORTED;
  if (cudaGraphLaunch(static_cast<cudaGraphExec_t>(graph), static_cast<cudaStream_t>(stream)) == cudaSuccess) return ZEN_OK;
  cudaGetLastError();
  return ZEN_ERR_LAUNCH;
}

int zen_graph_destroy(void* graph) {
  if (graph == nullptr) return ZEN_OK;
  if (cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(graph)) == cudaSuccess) return ZEN_OK;
  cudaGetLastError();
  return ZEN_ERR_LAUNCH;
}

}  // extern "C"
