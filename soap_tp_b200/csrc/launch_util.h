// Host-side launch helpers shared by the kernels of this library.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

namespace soapb200 {

// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device attribute of a kernel: a process that
// drives several GPUs has to raise it on each of them before the first launch there.  One instance of
// this struct per kernel (a function-local static at the launch site) remembers which devices are done.
struct PerDeviceOnce {
  static constexpr int kMaxDevices = 64;
  bool done[kMaxDevices] = {};
};

inline void allow_dynamic_smem(const void* kernel, size_t bytes, PerDeviceOnce& once, const char* what) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + ": cudaGetDevice: " + cudaGetErrorString(err));
  const bool tracked = device >= 0 && device < PerDeviceOnce::kMaxDevices;
  if (tracked && once.done[device]) return;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + " attribute: " + cudaGetErrorString(err));
  if (tracked) once.done[device] = true;
}

// An event for ordering streams, given back when the scope ends (work that waits for it keeps what it needs).
class ScopedEvent {
 public:
  ScopedEvent() { check(cudaEventCreateWithFlags(&event_, cudaEventDisableTiming)); }
  ~ScopedEvent() { cudaEventDestroy(event_); }
  ScopedEvent(const ScopedEvent&) = delete;
  ScopedEvent& operator=(const ScopedEvent&) = delete;
  void record(cudaStream_t stream) { check(cudaEventRecord(event_, stream)); }
  void hold(cudaStream_t stream) { check(cudaStreamWaitEvent(stream, event_, 0)); }

 private:
  static void check(cudaError_t err) {
    if (err != cudaSuccess) throw std::runtime_error(std::string("event: ") + cudaGetErrorString(err));
  }
  cudaEvent_t event_ = nullptr;
};

// The blocks of up to N problems that share a launch, one problem's after another's.
template <int N>
class GroupBlocks {
 public:
  void add(int blocks) {
    ends_[count_] = (count_ ? ends_[count_ - 1] : 0) + blocks;
    ++count_;
  }
  int total() const { return ends_[count_ - 1]; }
#ifdef __CUDACC__
  __device__ __forceinline__ int member(int block) const {
    int i = 0;
    if constexpr (N > 1) {
      while (i + 1 < count_ && block >= ends_[i]) ++i;
    }
    return i;
  }
  __device__ __forceinline__ int first(int member) const { return N > 1 && member ? ends_[member - 1] : 0; }
  __device__ __forceinline__ int count(int member) const { return ends_[member] - first(member); }
#endif

 private:
  int ends_[N];
  int count_ = 0;
};

// Launch that may begin before the kernel ahead of it in the stream has ended (programmatic dependent launch): what a kernel
// does before `wait_for_predecessor` -- barriers, TMEM, descriptor prefetch -- overlaps the tail of the one before, and the
// gap between two launches closes (a step of eight dependent launches: 118 -> 106 us at 256 x 512, 193 -> 181 us at
// 1000 x 1501).  Everything that touches global memory comes after that wait, which lasts until the
// predecessor has ended and its writes are visible.
template <typename... Parameters, typename... Arguments>
cudaError_t launch_dependent(void (*kernel)(Parameters...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Arguments&&... arguments) {
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &overlap;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Parameters>(arguments)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// From here on the next kernel's CTAs may take the SMs that this one leaves free.
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace soapb200
