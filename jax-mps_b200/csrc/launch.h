// The one way in which kernels and device copies of a plan are issued. Usually that is the runtime's launch; while a plan
// is recorded, or a recording is given other memory, the thread's LaunchObserver gets the launch instead. So the
// parameters that a recording's node is given later are made by the code that launches the kernel, tensor maps and
// alignment-dependent choices included.
#pragma once
#include <cuda_runtime.h>

#include <tuple>
#include <type_traits>
#include <utility>

namespace b200 {

struct LaunchObserver {
  virtual cudaError_t kernel(const void* func, const cudaLaunchConfig_t& cfg, void** args) = 0;
  virtual cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) = 0;

 protected:
  ~LaunchObserver() = default;
};
inline thread_local LaunchObserver* launch_observer = nullptr;

template <typename... P, typename... A>
cudaError_t launch_kernel(const cudaLaunchConfig_t& cfg, void (*kernel)(P...), A&&... args) {
  if (!launch_observer) return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  std::tuple<std::decay_t<P>...> values(std::forward<A>(args)...);
  return std::apply(
      [&](auto&... v) {
        void* ptrs[] = {(void*)&v...};
        return launch_observer->kernel((const void*)kernel, cfg, ptrs);
      },
      values);
}

// Without launch attributes.
template <typename... P, typename... A>
cudaError_t launch_plain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return launch_kernel(cfg, kernel, std::forward<A>(args)...);
}

inline cudaError_t copy_on_device(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  if (launch_observer) return launch_observer->copy(dst, src, bytes, stream);
  return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream);
}

}  // namespace b200
