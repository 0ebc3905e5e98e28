// Host-side helpers shared by the kernel launchers: per-device status word, tensor-map encoding
// through the driver entry point (no link-time dependency on libcuda), launch-error plumbing.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace lt {

// Device int that kernels write an error code to (0 = ok). One per device, created on first use.
int* device_status_word();

// Number of SMs of the current device (cached per device).
int sm_count();

// Encode a 2-D row-major tensor map. `inner` is the contiguous extent (elements), `outer` the number
// of rows, `row_stride_bytes` the pitch. Returns 0 on success, a CUresult otherwise.
int encode_tmap_2d(CUtensorMap* out, const void* base, int elem_bytes, uint64_t inner, uint64_t outer,
                   uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, int swizzle_128b);

// 3-D variant: dims/strides listed innermost first; stride[0] is implied by elem_bytes.
int encode_tmap_3d(CUtensorMap* out, const void* base, int elem_bytes, uint64_t d0, uint64_t d1, uint64_t d2,
                   uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1, uint32_t b2,
                   int swizzle_128b);

// 4-D variant.
int encode_tmap_4d(CUtensorMap* out, const void* base, int elem_bytes, uint64_t d0, uint64_t d1, uint64_t d2,
                   uint64_t d3, uint64_t stride1_bytes, uint64_t stride2_bytes, uint64_t stride3_bytes,
                   uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, int swizzle_128b);

// Every translation unit with bounded waits registers a function that stores the two wait budgets (SM cycles) into
// its own device globals; lt_set_wait_budget_cycles() calls them all for the current device.
void register_wait_budget_setter(int (*fn)(long long local_cycles, long long peer_cycles));

// Work that is due once on every device, such as the opt-in to more than 48 KB of shared memory for a kernel, which belongs to the device that
// is current.  Doing it twice is harmless: threads may race for it.
class OncePerDevice {
 public:
  bool pending() const { return (done_.load(std::memory_order_acquire) & bit()) == 0; }
  void finish() { done_.fetch_or(bit(), std::memory_order_release); }

 private:
  static uint64_t bit() {   // none: work stays due
    int dev = -1;
    return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;
  }
  std::atomic<uint64_t> done_{0};
};

// Launch of a kernel that calls pdl_wait() ahead of its first access to global memory: it may take its place on the SMs and set up its shared and
// tensor memory while the kernel ahead of it in the stream ends (from that one's pdl_launch_dependents() on; a kernel with tensor memory calls that
// after its own allocation, so that a successor cannot take the columns that it still needs).  What the kernels ahead may have written it reads by plain
// loads: no __ldg, ld.global.nc or inputs declared "const ... __restrict__", which are for memory that nobody writes while the kernel lives, and which the
// compiler may move across the wait.  Between kernels of a stream 2.2 us pass otherwise, 0.4 in
// a recorded graph, and set-up comes on top.  Training step of 1.1B layers over 2 x 2000 tokens (506 kernels) 18.4 -> 17.7 ms, four 8B layers over 8192
// tokens 82.9 -> 80.5 (1 % of it the norms), prompt of 4096 tokens 11.7 -> 11.4, decode step of the 1.1B model 1038 -> 956 us, latent decode step 510 -> 470.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// The same with CTAs in clusters of `cluster` along x.
template <class... P, class... A>
inline cudaError_t launch_chained_clusters(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

inline int cuda_ok(cudaError_t e) { return e == cudaSuccess ? 0 : int(e); }

}  // namespace lt

#define LT_RETURN_IF_CUDA(expr)                      \
  do {                                               \
    cudaError_t _e = (expr);                         \
    if (_e != cudaSuccess) return int(_e);           \
  } while (0)

#define LT_LAUNCH_CHECK()                            \
  do {                                               \
    cudaError_t _e = cudaGetLastError();             \
    if (_e != cudaSuccess) return int(_e);           \
  } while (0)
