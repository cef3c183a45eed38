// Kernel launches.  Every kernel of the library goes through launch_kernel(): into a stream, or, while the calling thread
// records (zen_record_begin), as a node of the graph that it records.
//
// A recording is built node by node with the graph functions of the runtime and not by capturing a stream: while any stream of
// the context is being captured, another thread's device synchronisation fails (and breaks the capture), and work that it
// issues on a pooled stream which happens to be the captured one disappears into the graph.  A pass that records itself
// behind a plain call must not do that to a program.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace zen {

struct LaunchShape {
  dim3 grid, block;
  size_t smem = 0;
  bool early = false;    // may start before the kernel in front of it has ended (programmatic dependent launch)
  unsigned cluster = 1;  // CTAs of a cluster (along x)
};

// record.cu: launches, or adds to this thread's recording.  `args`: one pointer per kernel parameter.
__attribute__((visibility("hidden"))) int launch_args(const void* kernel, const LaunchShape& shape, cudaStream_t stream, void** args);

// Whether the calling thread records.
__attribute__((visibility("hidden"))) bool recording();

template <typename... KArgs, typename... Args>
inline int launch_kernel(void (*kernel)(KArgs...), const LaunchShape& shape, cudaStream_t stream, Args&&... args) {
  return [&](KArgs... held) {
    void* ptrs[] = {const_cast<void*>(static_cast<const void*>(&held))...};
    return launch_args(reinterpret_cast<const void*>(kernel), shape, stream, ptrs);
  }(std::forward<Args>(args)...);
}

}  // namespace zen
