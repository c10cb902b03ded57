// common.cuh — shared helpers of libpfsim: status/error plumbing, device
// error words, launch-shape constants and small vector math.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdlib>
#include <string>

#include "pfsim.h"

namespace pf {

// Thread-local error text behind pf_last_error().
void set_error(const std::string& msg);
const std::string& get_error();

// PFSIM_VERBOSE set: host-side events (grid window growth, graph captures,
// the phases of a serving tick) and their times go to stderr.
inline bool verbose() {
  static const bool v = std::getenv("PFSIM_VERBOSE") != nullptr;
  return v;
}

// Returns a pf_status and records msg.
inline pf_status fail(pf_status s, const std::string& msg) {
  set_error(msg);
  return s;
}

// CUDA call check inside functions returning pf_status.
#define PF_CUDA(call)                                                                      \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return ::pf::fail(PF_ERR_CUDA, std::string("CUDA: ") + #call + ": " +                \
                                         cudaGetErrorString(e_));                          \
  } while (0)

#define PF_TRY(expr)                \
  do {                              \
    pf_status s_ = (expr);          \
    if (s_ != PF_OK) return s_;     \
  } while (0)

// Number of SMs on the current device (148 on B200), cached per device.
int sm_count();

// Device-side error word bits, written by kernels that give up a bounded
// wait or find an inconsistent input; read back by the host after a call.
enum DeviceError : uint32_t {
  DEV_ERR_LOOKBACK_TIMEOUT = 1u << 0,
};

// Upper bound on spins of a decoupled look-back before it reports
// DEV_ERR_LOOKBACK_TIMEOUT and returns (forward progress is guaranteed by
// tile ids taken in launch order, so this only triggers on a bug).
constexpr uint32_t kLookbackSpinLimit = 1u << 24;

// ------------------------------------------------- linked launches ----
// A stage of a step or a sort is a few microseconds of kernel, and a plain
// launch adds a microsecond or two of starting it after the kernel before
// has completed. Kernels launched one after the other on a stream inside a
// LinkedLaunches scope are therefore linked (programmatic dependent launch):
// the next kernel's blocks are placed once the blocks of the one before have
// exited, and wait in pdl_begin(), their first statement, until its writes
// are visible. Nothing of a kernel runs before its pdl_begin(), apart from the
// cloth's colours, which read what no kernel just before them writes; so the
// order of the work is that of plain launches. Only those colours signal their
// dependents before they end: blocks placed beside a running kernel crowded on
// the SMs that it left first, which made the soft-body passes 7 % slower (24
// mixed scenes: 2.67 ms a step plain, 2.87 signalled at the start, 2.64 at the
// exit), and signalled from small grids alone, nothing got faster.
// Plain and linked, each with the kernels of its time: a sort of 20,011
// particles 57 and 40 us (25 now, in one cluster), of 1,000,003 103 and 72, a
// 256 x 256 cloth's step (190 launches) 0.86 and 0.81 ms (0.64 now, see
// k_cloth), a 30,000-particle fluid's with surface effects 2.31 and 2.24
// (1.78 now, for other reasons).
__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets the next kernel's blocks be placed while this one runs: only after
// this kernel's own pdl_begin(), so that what the next one reads before its
// wait is safe from every kernel but this.
__device__ __forceinline__ void pdl_signal() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The calling thread's state: linking is on inside a scope, and the last
// operation issued there was a kernel on `last`.
struct LinkState {
  bool on = false, linked = false;
  cudaStream_t last = nullptr;
};
inline thread_local LinkState t_link;

// Links the launches of its lifetime; what came before is waited for in full.
class LinkedLaunches {
 public:
  LinkedLaunches() : was_(t_link) { t_link = LinkState{true, false, nullptr}; }
  ~LinkedLaunches() { t_link = was_; }
  LinkedLaunches(const LinkedLaunches&) = delete;
  LinkedLaunches& operator=(const LinkedLaunches&) = delete;

 private:
  LinkState was_;
};
// To be called after any operation other than launch_kernel (a copy, a
// memset, a wait for another stream's event): the next kernel is launched
// plainly, after all of the stream's work before it.
inline void break_link() { t_link.linked = false; }

inline cudaLaunchAttribute cluster_attribute(uint32_t blocks) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = blocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  return at;
}
// kernel<<<grid, block, smem, st>>>(args...) in clusters of `cluster` blocks
// (0: none), linked where the operation before it on this thread was a kernel
// on the same stream. Every kernel launched through it starts with pdl_begin().
template <typename... P, typename... A>
inline cudaError_t launch_cluster(void (*kernel)(P...), uint32_t cluster, dim3 grid, dim3 block, size_t smem,
                                  cudaStream_t st, A... args) {
  cudaLaunchAttribute at[2] = {};
  unsigned attrs = 0;
  if (t_link.on && t_link.linked && t_link.last == st) {
    at[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[attrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster) at[attrs++] = cluster_attribute(cluster);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = attrs;
  t_link.linked = true;
  t_link.last = st;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  return launch_cluster(kernel, 0, grid, block, smem, st, args...);
}

__host__ __device__ inline uint32_t div_up(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

}  // namespace pf
