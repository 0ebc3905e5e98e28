// Product of 1 to 8 rows with a weight matrix: y[M, N] = x[M, K] @ W[N, K]^T (+ residual).
//
// weight_stream.cu does it; the kernel here takes what its copies can not, rows that overlap in memory (an expanded or sliding view), one row of
// x at a time: a warp owns one output column, its lanes walk the row of W in 16-byte steps, four loads in flight per lane, and a shuffle
// reduction finishes the column.  The reference runs every Linear through cublasSgemm whatever the row count (src/ops/linear.cpp:176-192).
#include "lt_cuda.h"
#include "common/host.h"
#include "common/ptx.cuh"
#include "weight_stream.h"

namespace lt {

constexpr int kGemvMaxM = 8;
constexpr int kGemvWarps = 8;

__global__ void __launch_bounds__(kGemvWarps * 32)
gemv_bf16_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, long long ldw, __nv_bfloat16* __restrict__ y,
                 const __nv_bfloat16* __restrict__ residual, int N, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int n = blockIdx.x * kGemvWarps + warp; n < N; n += gridDim.x * kGemvWarps) {
    const __nv_bfloat16* wr = w + (long long)n * ldw;
    float v = 0.f;
    // K is a multiple of 8; a lane takes 8 elements per step, the warp 256
    for (int k0 = lane * 8; k0 < K; k0 += 4 * 256) {
      uint4 wv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u * 256;
        wv[u] = (k < K) ? ld_nc_v4(wr + k) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u * 256;
        if (k >= K) break;
        const float2 w0 = unpack_bf16x2(wv[u].x), w1 = unpack_bf16x2(wv[u].y), w2 = unpack_bf16x2(wv[u].z), w3 = unpack_bf16x2(wv[u].w);
        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + k));
        const float2 x0 = unpack_bf16x2(xv.x), x1 = unpack_bf16x2(xv.y), x2 = unpack_bf16x2(xv.z), x3 = unpack_bf16x2(xv.w);
        v += w0.x * x0.x + w0.y * x0.y + w1.x * x1.x + w1.y * x1.y + w2.x * x2.x + w2.y * x2.y + w3.x * x3.x + w3.y * x3.y;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) {
      if (residual) v += __bfloat162float(residual[n]);
      y[n] = __float2bfloat16(v);
    }
  }
}

}  // namespace lt

extern "C" {

// y[M, N] = x[M, K] @ w[N, K]^T (+ residual[M, N]); 1 <= M <= 8, K a multiple of 8, rows 16-byte aligned.
int lt_gemv_bf16(const void* x, long long ldx, const void* w, long long ldw, void* y, long long ldy, const void* residual,
                 long long ldr, int M, int N, int K, void* stream) {
  using namespace lt;
  if (M < 1 || M > kGemvMaxM || N <= 0 || K <= 0 || (K & 7) || (ldx & 7) || (ldw & 7) ||
      (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15))
    return -int(kStatusBadArgument);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto W = static_cast<const __nv_bfloat16*>(w);
  auto Y = static_cast<__nv_bfloat16*>(y);
  auto R = static_cast<const __nv_bfloat16*>(residual);
  const StreamProduct p{X, ldx, W, ldw, Y, ldy, R, ldr, M, N, K, 0};
  if (stream_takes(p)) return launch_stream(p, st);
  const int sms = sm_count();
  int blocks = (N + kGemvWarps - 1) / kGemvWarps;
  if (blocks > sms * 8) blocks = sms * 8;
  for (int m = 0; m < M; ++m)
    gemv_bf16_kernel<<<blocks, kGemvWarps * 32, 0, st>>>(X + m * ldx, W, ldw, Y + m * ldy, R ? R + m * ldr : nullptr, N, K);
  LT_LAUNCH_CHECK();
  return 0;
}

}  // extern "C"
