// Products of a few rows with a weight matrix that is read once (weight_stream.cu), for the launchers in gemv.cu and gemm_skinny.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace lt {

constexpr int kStreamMaxRows = 64, kStreamNormRows = 16, kStreamNormK = 8192;

// y[M, N] = x[M, K] @ w[N, K]^T (+ residual[M, N]); act != 0: y = act(gate) * up with w [2 N, K] = gate rows, then up rows (1: GELU in
// its tanh form, 2: SiLU; no residual).  1 <= M <= kStreamMaxRows, K a multiple of 8, rows of x and w 16-byte aligned; y and residual
// need the alignment of their elements only.
struct StreamProduct {
  const __nv_bfloat16* x;
  long long ldx;
  const __nv_bfloat16* w;
  long long ldw;
  __nv_bfloat16* y;
  long long ldy;
  const __nv_bfloat16* residual;
  long long ldr;
  int M, N, K, act;
  // x is normalised first: x / rms(x) * gain, rms over the K columns with eps (nullptr: taken as it is); M <= kStreamNormRows, K <= kStreamNormK
  const __nv_bfloat16* gain;
  float eps;
  float* y32;   // 32-bit results instead of y, pitch ldy (nullptr: y)
  int early;   // the kernel starts under the one before it in the stream and fetches weights meanwhile, which that one must not write
};
// Rows of x or w that overlap (a pitch below K) are not taken.
bool stream_takes(const StreamProduct& p);
int launch_stream(StreamProduct p, cudaStream_t st);

}  // namespace lt
