// Product of 1 to 64 rows with a weight matrix, bound by reading the matrix once.
//
// A CTA of eight warps owns R rows of W at a time (output columns); the warps take turns along K, 64 elements each.  Every warp
// keeps a ring of stages in shared memory (R rows of W and the rows of x, 128 bytes of each) that its first lane fills by TMA, across
// the ends of tiles too, so that loads need neither registers nor addresses, no warp waits for another before the end of a tile, and
// 60 to 130 KB of weights a SM stay in flight (latency times bandwidth is about 45 KB a SM).  The products go through the
// warp-level tensor-core instruction (mma.sync m16n8k16: 16 rows of x by 8 rows of W; the 128-row tiles of tcgen05 need a set-up
// longer than many of these kernels run).  Inside a stage the K dimension is permuted the same way for both operands, so that 16
// contiguous bytes are a lane's fragments of two instructions and eight lanes read from all banks.  The warps' partial sums meet in
// shared memory in a fixed order.
//
// Where the caller vouches for the weights (a step of serving), the kernel is launched to start under the one before it and fills its rings
// with weights meanwhile: decode steps of six 8B layers 1343 -> 1312 us (32 sequences) and 963 -> 935 (8 on an 8-bit cache), of the 1.1B
// model 1020 -> 1004 (1030 to 1042 on other cards).
//
// Measured (graph replay over different weights, us; before: CUDA-core dot products for up to 8 rows, register-fed mma.sync beyond; bytes of W at
// the copy rate in brackets): 28672 x 4096 [35.8]: 1 row 40.5 -> 37.9, 8 rows 121 -> 39, 16 rows 81 -> 42, 32 rows 100 -> 53, 64 rows
// 163 -> 87; 4096 x 14336 [17.9]: 24 -> 21, 74 -> 21, 41 -> 21, 47 -> 24, 71 -> 36; 2048 x 2048 [1.3]: 4.7 -> 4.3, 8.2 -> 4.3, 8.0 -> 4.4,
// 10.0 -> 5.2, 16.4 -> 8.5.  Additions with rounding, up to 16 rows (see the loop), were added since: 38.7 -> 38.8, 39.6 -> 39.9, 42.2 -> 42.6 and
// 4.79 -> 4.88 (2048 x 2048, 8 rows).  With 32 rows and more it is bound by x, which every tile reads again from L2; small matrices by the start.
//
// With up to 16 rows the kernel can normalise x on the way: the fragments are multiplied by the gains and rounded, as normalised rows would be, the
// squares are summed beside them, and 1 / rms multiplies the results.  A kernel in front of the product takes 2 to 3 us of a step's chain: decode
// steps of the 1.1B model 956 -> 880 us (one sequence), six 8B layers 943 -> 930 (8 sequences on an 8-bit cache).
//
// Rings of half the size, so that the next product lies beside this one and has all of its first weights early, are slower (1.1B step 880 -> 1037 us, tiles of
// 16 rows with 8 rows of x as well 1069): its copies queue ahead of this kernel's own.  Deeper rings with 8 rows of x: 880 -> 911.
#include "lt_cuda.h"
#include "common/host.h"
#include "common/ptx.cuh"
#include "common/scalar.cuh"
#include "weight_stream.h"

namespace lt {

__device__ __forceinline__ void ws_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same from zero.
__device__ __forceinline__ void ws_mma_0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// Eight bf16 values of x times eight gains, rounded to bf16; their squares join `sq`.
__device__ __forceinline__ void ws_times(uint4& x, const uint4& gain, float& sq) {
  uint32_t* xw = &x.x;
  const uint32_t* gw = &gain.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = unpack_bf16x2(xw[j]), b = unpack_bf16x2(gw[j]);
    sq = fmaf(a.x, a.x, fmaf(a.y, a.y, sq));
    xw[j] = pack_bf16x2(a.x * b.x, a.y * b.y);
  }
}
__device__ __forceinline__ uint4 lds_16(uint32_t src) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
  return v;
}

// XR: rows of x that a stage holds (8 or a multiple of 16); R: rows of W of a tile.
template <int XR, int R>
struct WsCfg {
  static constexpr int kWarps = 8;
  static constexpr int kStage = (R + XR) * 128;
  static constexpr int kCtas = XR == 8 && R == 32 ? 2 : 1;                              // a SM
  static constexpr int kRing = (kCtas == 2 ? 96 : 192) * 1024;
  static constexpr int kStages = kRing / (kWarps * kStage) < 6 ? kRing / (kWarps * kStage) : 6;
  static constexpr int kOffPart = kWarps * kStages * kStage;                            // [warp][16 rows of x][R] partial sums
  static constexpr int kOffBar = kOffPart + kWarps * R * 64;
  static constexpr int kSmem = kOffBar + kWarps * kStages * 8 + 16 + 1024;
  static_assert(kStages >= 2 && kSmem * kCtas <= 227 * 1024 - (kCtas - 1) * 1024, "does not fit");
};

template <int XR, int R, bool GLU, bool NORM>
__global__ void __launch_bounds__(WsCfg<XR, R>::kWarps * 32, WsCfg<XR, R>::kCtas)
weight_stream_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap tx, const StreamProduct p, const int tiles, const int cols, int* status) {
  using Cfg = WsCfg<XR, R>;
  constexpr int W = Cfg::kWarps, S = Cfg::kStages, MT = (XR + 15) / 16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const uint32_t ring = smem_u32(smem) + warp * (S * Cfg::kStage);
  const uint32_t bars = smem_u32(smem) + Cfg::kOffBar + warp * (S * 8);
  float* part = reinterpret_cast<float*>(smem + Cfg::kOffPart);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kOffBar + W * S * 8);
  // with NORM: [warp][16 rows] sums of squares, then the gains, zero past K
  float* squares = reinterpret_cast<float*>(smem + Cfg::kOffBar + W * S * 8 + 16);
  const uint32_t gains = smem_u32(smem) + Cfg::kOffBar + W * S * 8 + 16 + W * 64;
  if (threadIdx.x == 0) *abort_flag = 0;
  if (lane == 0) {
    for (int s = 0; s < S; ++s) mbar_init(bars + s * 8, 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  __syncthreads();
  const int N = p.N, M = p.M;
  const int chunks = (p.K + 63) / 64;
  const int mine = chunks > warp ? (chunks - warp + W - 1) / W : 0;    // of every tile

  // copies run ahead of the products by S stages, into the next tiles
  int at_tile = blockIdx.x, at = 0, at_slot = 0;
  auto load = [&](bool weights, bool xs) {
    if (mine > 0 && at_tile < tiles) {
      if (lane == 0) {
        const uint32_t to = ring + at_slot * Cfg::kStage, bar = bars + at_slot * 8;
        const int k0 = (warp + at * W) * 64;
        if (weights) {
          mbar_expect_tx(bar, ((GLU ? 2 * cols : cols) + XR) * 128);
          tma_load_2d(to, &tw, bar, k0, at_tile * cols);
          if (GLU) tma_load_2d(to + R * 64, &tw, bar, k0, N + at_tile * cols);
        }
        if (xs) tma_load_2d(to + R * 128, &tx, bar, k0, 0);
      }
      at_slot = at_slot + 1 == S ? 0 : at_slot + 1;
      if (++at == mine) { at = 0; at_tile += gridDim.x; }
    }
  };
  pdl_launch_dependents();
  if (!p.early) pdl_wait();
  if constexpr (NORM) {   // (a weight like w)
    for (int k = threadIdx.x * 8; k < chunks * 64; k += W * 32 * 8) {
      const uint4 v = k < p.K ? *reinterpret_cast<const uint4*>(p.gain + k) : make_uint4(0u, 0u, 0u, 0u);
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(gains + k * 2), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
    __syncthreads();
  }
#pragma unroll
  for (int s = 0; s < S; ++s) load(true, false);
  if (p.early) pdl_wait();
  at_tile = blockIdx.x; at = 0; at_slot = 0;
#pragma unroll
  for (int s = 0; s < S; ++s) load(false, true);

  // lane (g, q) reads units 2 q and 2 q + 1 of rows g, g + 8, ...; TMA's swizzle puts unit u of row r at u ^ (r & 7)
  const uint32_t from0 = ring + g * 128 + (((2 * q) ^ g) << 4), from1 = ring + g * 128 + (((2 * q + 1) ^ g) << 4);
  int slot = 0;
  uint32_t phase = 0;
  bool ok = true;
  [[maybe_unused]] float sq_lo = 0.f, sq_hi = 0.f;   // this lane's share of the sums of squares of rows g and g + 8
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    float acc[MT][R / 8][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int f = 0; f < R / 8; ++f)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[m][f][r] = 0.f;
    for (int i = 0; i < mine && ok; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(bars + slot * 8, phase, abort_flag, status, kStatusTimeoutFull));
      if (!ok) break;
      // The instruction cuts off what it adds to its accumulator.  With one block of rows, four of them start from zero for every stage and
      // ordinary additions take the sums on (products of up to 8 rows were such additions throughout; 14336 deep, one result in a thousand came
      // out a unit off in the 16 bits that leave, now one in ten thousand, as before).
      float sum[MT == 1 ? R / 8 : 1][4];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t from = (c ? from1 : from0) + slot * Cfg::kStage;
        uint4 xv[MT][2];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          xv[m][0] = lds_16(from + R * 128 + m * 2048);
          xv[m][1] = XR == 8 ? make_uint4(0u, 0u, 0u, 0u) : lds_16(from + R * 128 + m * 2048 + 1024);
        }
        if constexpr (NORM) {
          // the rows times the gains, rounded to 16 bits as normalised rows would be; their common factor 1 / rms waits for the sums
          const uint4 gn = lds_16(gains + ((warp + i * W) * 64 + (2 * q + c) * 8) * 2);
          ws_times(xv[0][0], gn, sq_lo);
          if constexpr (XR != 8) ws_times(xv[0][1], gn, sq_hi);
        }
#pragma unroll
        for (int f = 0; f < R / 8; ++f) {
          const uint4 wv = lds_16(from + f * 1024);
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            if constexpr (MT == 1) {
              if (c == 0) ws_mma_0(sum[f], xv[m][0].x, xv[m][1].x, xv[m][0].y, xv[m][1].y, wv.x, wv.y);
              else ws_mma(sum[f], xv[m][0].x, xv[m][1].x, xv[m][0].y, xv[m][1].y, wv.x, wv.y);
              ws_mma(sum[f], xv[m][0].z, xv[m][1].z, xv[m][0].w, xv[m][1].w, wv.z, wv.w);
            } else {
              ws_mma(acc[m][f], xv[m][0].x, xv[m][1].x, xv[m][0].y, xv[m][1].y, wv.x, wv.y);
              ws_mma(acc[m][f], xv[m][0].z, xv[m][1].z, xv[m][0].w, xv[m][1].w, wv.z, wv.w);
            }
          }
        }
      }
      if constexpr (MT == 1) {
#pragma unroll
        for (int f = 0; f < R / 8; ++f)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[0][f][r] += sum[f][r];
      }
      __syncwarp();
      load(true, true);
      if (++slot == S) { slot = 0; phase ^= 1u; }
    }

    if constexpr (NORM) {
      if (tile == blockIdx.x) {   // the first tile has met every column; its sums serve all of them
        sq_lo += __shfl_xor_sync(0xffffffffu, sq_lo, 1); sq_lo += __shfl_xor_sync(0xffffffffu, sq_lo, 2);
        sq_hi += __shfl_xor_sync(0xffffffffu, sq_hi, 1); sq_hi += __shfl_xor_sync(0xffffffffu, sq_hi, 2);
        if (q == 0) { squares[warp * 16 + g] = sq_lo; squares[warp * 16 + g + 8] = sq_hi; }
      }
    }
    constexpr int F = R / 8 / (GLU ? 2 : 1);   // fragments of results
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      __syncthreads();   // the sums before have been read
#pragma unroll
      for (int f = 0; f < R / 8; ++f)
#pragma unroll
        for (int r = 0; r < 4; ++r) part[warp * (R * 16) + (f * 4 + r) * 32 + lane] = acc[m][f][r];
      __syncthreads();
      for (int e = threadIdx.x; e < F * 64; e += W * 32) {
        const int f = e >> 6, h = (e >> 5) & 1, l = e & 31;
        const int row = m * 16 + h * 8 + (l >> 2), at_col = f * 8 + (l & 3) * 2, col = tile * cols + at_col;
        if (row >= M || at_col >= cols) continue;   // cols is even
        float v[2];
        float factor = 1.f;
        if constexpr (NORM) {
          float sq = 0.f;
#pragma unroll
          for (int w = 0; w < W; ++w) sq += squares[w * 16 + row];
          factor = rsqrtf(sq / p.K + p.eps);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int from = (f * 4 + h * 2 + b) * 32 + l;
          float s = 0.f, up = 0.f;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            s += part[w * (R * 16) + from];
            if constexpr (GLU) up += part[w * (R * 16) + from + F * 128];
          }
          if constexpr (NORM) { s *= factor; up *= factor; }
          if constexpr (GLU) s = (p.act == 1 ? gelu_tanh_f(s) : silu_quick_f(s)) * up;
          else if (p.residual && col + b < N) s += __bfloat162float(p.residual[(long long)row * p.ldr + col + b]);
          v[b] = s;
        }
        if (p.y32) {
          if (col < N) p.y32[(long long)row * p.ldy + col] = v[0];
          if (col + 1 < N) p.y32[(long long)row * p.ldy + col + 1] = v[1];
          continue;
        }
        __nv_bfloat16* to = p.y + (long long)row * p.ldy + col;
        if (col + 1 < N && !(reinterpret_cast<uintptr_t>(to) & 3)) {
          *reinterpret_cast<uint32_t*>(to) = pack_bf16x2(v[0], v[1]);
        } else {
          if (col < N) to[0] = __float2bfloat16(v[0]);
          if (col + 1 < N) to[1] = __float2bfloat16(v[1]);
        }
      }
    }
  }
  if (!ok)
    for (int spin = 0; spin < 2000; ++spin) __nanosleep(100);  // bounded grace period for copies in flight
}

// Shared memory that normalising takes beside kSmem: sums of squares and gains.
template <class Cfg>
static int norm_bytes(int K) { return Cfg::kWarps * 64 + (K + 63) / 64 * 128; }

template <int XR, int R, bool GLU, bool NORM = false>
static int launch_ws(const StreamProduct& p, cudaStream_t st) {
  using Cfg = WsCfg<XR, R>;
  if constexpr (!NORM && XR <= 16) {
    if (p.gain) return launch_ws<XR, R, GLU, true>(p, st);
  }
  static OncePerDevice configured;
  auto kern = weight_stream_kernel<XR, R, GLU, NORM>;
  const int smem = Cfg::kSmem + (NORM ? norm_bytes<Cfg>(p.K) : 0);
  if (configured.pending()) {
    LT_RETURN_IF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem + (NORM ? norm_bytes<Cfg>(kStreamNormK) : 0)));
    configured.finish();
  }
  // As many tiles as CTAs, or a multiple of that, so that none ends in a round of a few tiles: tiles get as wide as that takes, and
  // the copies fetch that many rows.
  constexpr int most = GLU ? R / 2 : R;
  const int room = sm_count() * Cfg::kCtas, rounds = (p.N + most * room - 1) / (most * room);
  int cols = (p.N + rounds * room - 1) / (rounds * room);
  cols = cols + (cols & 1);
  CUtensorMap tw, tx;
  int r = encode_tmap_2d(&tw, p.w, 2, p.K, GLU ? 2ull * p.N : p.N, (uint64_t)p.ldw * 2, 64, cols, 1);
  if (r) return 1000 + r;
  r = encode_tmap_2d(&tx, p.x, 2, p.K, p.M, (uint64_t)p.ldx * 2, 64, XR, 1);
  if (r) return 2000 + r;
  const int tiles = (p.N + cols - 1) / cols;
  LT_RETURN_IF_CUDA(launch_chained(kern, dim3(tiles < room ? tiles : room), dim3(Cfg::kWarps * 32), smem, st, tw, tx, p, tiles, cols, device_status_word()));
  return 0;
}

// Tiles of 16 rows where they give every SM one, else of 32: 2048 columns 4.3 against 4.7 us, 4096 columns 13.9 against 8.3.  Up to
// 8 rows of x and more columns than SMs have tiles, two CTAs an SM and a stage for 8 rows of x (28672 x 4096, 8 rows: 39 against 42 us); with
// 17 to 32 rows and that many columns, tiles of 64, which read x half as often (53 against 55 us, 32000 x 2048 34.7 against 37.7).  Gains of more than 7808
// columns leave no room for the second CTA: its tiles would come after the first one's (10240 x 8192, 8 rows: 49 us, with 16 rows of x 31).
template <bool GLU>
static int stream_by_size(const StreamProduct& p, cudaStream_t st) {
  const long long rows = GLU ? 2ll * p.N : p.N, sms = sm_count();
  const bool narrow = rows <= 16 * sms, wide = rows > 32 * sms;
  if (p.M <= 16) {
    if (narrow) return launch_ws<16, 16, GLU>(p, st);
    const bool two = !p.gain || 2 * (WsCfg<8, 32>::kSmem + norm_bytes<WsCfg<8, 32>>(p.K) + 1024) <= 228 * 1024;
    return wide && p.M <= 8 && two ? launch_ws<8, 32, GLU>(p, st) : launch_ws<16, 32, GLU>(p, st);
  }
  if (p.M <= 32) {
    if (narrow) return launch_ws<32, 16, GLU>(p, st);
    return wide ? launch_ws<32, 64, GLU>(p, st) : launch_ws<32, 32, GLU>(p, st);
  }
  return launch_ws<64, 32, GLU>(p, st);
}

bool stream_takes(const StreamProduct& p) {
  if (p.gain && (p.M > kStreamNormRows || p.K > kStreamNormK || (p.K & 7) || (reinterpret_cast<uintptr_t>(p.gain) & 15))) return false;
  return p.M >= 1 && p.M <= kStreamMaxRows && p.ldw >= p.K && (p.M == 1 || p.ldx >= p.K);
}

int launch_stream(StreamProduct p, cudaStream_t st) {
  if (p.M == 1) p.ldx = (p.K + 7) / 8 * 8;
  return p.act ? stream_by_size<true>(p, st) : stream_by_size<false>(p, st);
}

}  // namespace lt

extern "C" {

// The product of weight_stream.h by itself.  early: the kernel may start before the one ahead of it in the stream has ended and reads w (and gain)
// then, so that one must not write them; x, residual and y are touched only after it.  gain (or nullptr), eps: x is normalised.  fp32: y holds 32-bit results.
int lt_weight_stream_norm(const void* x, long long ldx, const void* gain, float eps, const void* w, long long ldw, void* y, long long ldy, int fp32,
                          const void* residual, long long ldr, int M, int N, int K, int act, int early, void* stream) {
  using namespace lt;
  StreamProduct p{static_cast<const __nv_bfloat16*>(x), ldx, static_cast<const __nv_bfloat16*>(w), ldw, static_cast<__nv_bfloat16*>(y), ldy,
                  static_cast<const __nv_bfloat16*>(residual), ldr, M, N, K, act};
  p.gain = static_cast<const __nv_bfloat16*>(gain);
  p.eps = eps;
  p.early = early;
  if (fp32) p.y32 = static_cast<float*>(y);
  if (N <= 0 || K <= 0 || (K & 7) || (ldx & 7) || (ldw & 7) || act < 0 || act > 2 || (act && residual) || !stream_takes(p) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
    return -int(kStatusBadArgument);
  return launch_stream(p, static_cast<cudaStream_t>(stream));
}
int lt_weight_stream(const void* x, long long ldx, const void* w, long long ldw, void* y, long long ldy, const void* residual, long long ldr, int M,
                     int N, int K, int act, int early, void* stream) {
  return lt_weight_stream_norm(x, ldx, nullptr, 0.f, w, ldw, y, ldy, 0, residual, ldr, M, N, K, act, early, stream);
}

}  // extern "C"
