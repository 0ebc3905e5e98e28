// Memory-bound bf16 kernels of the transformer block: RoPE (interleaved pairs), SwiGLU, GELU(tanh),
// residual add, embedding gather / scatter-add, dtype casts, fills.
//
// Reference counterparts: rope_forward/backward (src/backend/gpu_native/nn/nn_kernels.cu:1204-1254),
// gelu_forward/backward (:1118-1146), embedding_forward/backward (:1148-1188), elementwise family
// (src/backend/gpu_native/elementwise/elementwise_ops.cu:3-98), cast kernels (:362-430).
// The reference has no SiLU/SwiGLU; it is added because the Llama-style configurations need it.
// Every kernel moves 16 bytes per thread per access and grid-strides.
#include "lt_cuda.h"

#include <cuda_fp8.h>
#include "common/host.h"
#include "common/ptx.cuh"
#include "common/scalar.cuh"

namespace lt {

__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ---------------------------------------------------------------------------------------------- RoPE
// In-place rotation of `heads` heads of width `hd` inside rows of pitch `row_stride` (elements).
// Row r belongs to position (r % T) + pos_offset... positions are given explicitly when pos != nullptr.
// Pair convention: (x[2i], x[2i+1]) rotated by angle pos * theta^(-2i/hd)  (interleaved, as the reference).
// cos/sin tables are [max_pos, hd/2] fp32. sign = +1 forward, -1 backward (inverse rotation).
// IDX: 32 bits where the count of 8-element pieces fits (64-bit divisions cost more than the bytes: 8192 rows of 32 heads of 64, 20 us).
template <typename IDX>
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, const int* pos, IDX rows, IDX T,
                            IDX heads, IDX hd, long long row_stride, float sign) {
  pdl_launch_dependents();
  pdl_wait();
  const IDX vec_per_head = hd / 8, per_row = heads * vec_per_head;
  const IDX total = rows * per_row;
  for (IDX i = IDX(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += IDX(gridDim.x) * blockDim.x) {
    const IDX r = i / per_row, c = i - r * per_row, v = c % vec_per_head;
    const int t = pos ? pos[r] : int(r % T);
    __nv_bfloat16* p = x + r * row_stride + (long long)c * 8;
    float f[8];
    ld8(p, f);
    const float4 c4 = *reinterpret_cast<const float4*>(cos_t + (long long)t * (hd / 2) + v * 4);
    const float4 s4 = *reinterpret_cast<const float4*>(sin_t + (long long)t * (hd / 2) + v * 4);
    const float cs[4] = {c4.x, c4.y, c4.z, c4.w};
    const float s[4] = {s4.x * sign, s4.y * sign, s4.z * sign, s4.w * sign};
    float o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = f[2 * j] * cs[j] - f[2 * j + 1] * s[j];
      o[2 * j + 1] = f[2 * j] * s[j] + f[2 * j + 1] * cs[j];
    }
    st8(p, o);
  }
}

// Rotation of queries and keys and the write of keys and values into a paged cache, in one pass over the rows [q | k | v] of a product.
// Queries go to q_out, packed, or stay where they are (q_out nullptr: keys are then rotated in place too, for a prompt's own attention).
// A launch for each of these (two rotations, two or three copies, the write) took 9 to 16 us a layer of a decode step, this one 2.  Items are counted
// in 32 bits where they fit: three 64-bit divisions an item were most of a prompt's time here (12 us a layer of 4096 tokens, 8 without).
template <bool FP8, typename IDX>
__global__ void rope_append_kernel(__nv_bfloat16* __restrict__ qkv, long long ld, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                   const int* pos, const int* slots, __nv_bfloat16* __restrict__ q_out,
                                   void* __restrict__ k_cache, void* __restrict__ v_cache, IDX rows, int Hq, int Hkv, int hd, int block_size,
                                   float k_inv, float v_inv) {
  pdl_launch_dependents();
  pdl_wait();
  const int vph = hd / 8, heads = Hq + 2 * Hkv;
  const IDX per_row = IDX(heads) * vph, total = rows * per_row;
  for (IDX i = IDX(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += IDX(gridDim.x) * blockDim.x) {
    const long long r = i / per_row;
    const int c = int(i - IDX(r) * per_row), h = c / vph, v = c - h * vph;
    __nv_bfloat16* p = qkv + r * ld + (long long)h * hd + v * 8;
    float f[8];
    ld8(p, f);
    if (h < Hq + Hkv) {
      const int t = pos[r];
      const float4 c4 = *reinterpret_cast<const float4*>(cos_t + (long long)t * (hd / 2) + v * 4);
      const float4 s4 = *reinterpret_cast<const float4*>(sin_t + (long long)t * (hd / 2) + v * 4);
      const float c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = f[2 * j], b = f[2 * j + 1];
        f[2 * j] = a * c[j] - b * s[j];
        f[2 * j + 1] = a * s[j] + b * c[j];
      }
      if (h < Hq && q_out) st8(q_out + (r * Hq + h) * (long long)hd + v * 8, f);
      else if (!q_out) st8(p, f);
      if (h < Hq) continue;
    }
    const int slot = slots[r];
    if (slot < 0) continue;
    const bool is_k = h < Hq + Hkv;
    const int g = h - Hq - (is_k ? 0 : Hkv);
    const long long dst = (((long long)(slot / block_size) * Hkv + g) * block_size + slot % block_size) * hd + v * 8;
    if (FP8) {
      alignas(8) uint8_t out[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)   // what is cached is the value as 16 bits hold it
        out[j] = __nv_fp8_e4m3(__bfloat162float(__float2bfloat16(f[j])) * (is_k ? k_inv : v_inv)).__x;
      *reinterpret_cast<uint2*>(static_cast<uint8_t*>(is_k ? k_cache : v_cache) + dst) = *reinterpret_cast<const uint2*>(out);
    } else {
      st8(static_cast<__nv_bfloat16*>(is_k ? k_cache : v_cache) + dst, f);
    }
  }
}

// ---------------------------------------------------------------------------------------------- SwiGLU
// gu: [M, 2F] with gate in columns [0,F) and up in [F,2F).  h = silu(gate) * up.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* __restrict__ h, long long M, int F) {
  pdl_launch_dependents();
  pdl_wait();
  const int vpr = F / 8;
  const long long total = M * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = int(i % vpr) * 8;
    float g[8], u[8], o[8];
    ld8(gu + r * 2 * F + c, g);
    ld8(gu + r * 2 * F + F + c, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    st8(h + r * F + c, o);
  }
}
// dgu may alias gu (written in place).
// h = g sigmoid(slope g) (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit); gu rows are [gate | up].
template <typename T>
__global__ void clamped_glu_kernel(const T* __restrict__ gu, T* __restrict__ h, long long M, int F, float limit, float slope) {
  const long long total = M * F;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / F, c = i % F;
    const float g = fminf(ldf(gu + r * 2 * F + c), limit);
    const float u = fminf(fmaxf(ldf(gu + r * 2 * F + F + c), -limit), limit);
    stf(h + i, g * sigmoid_f(slope * g) * (u + 1.f));
  }
}

// The same for bf16, eight columns per thread.
__global__ void clamped_glu8_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h, long long M, int F,
                                    float limit, float slope) {
  const int fu = F / 8;
  const long long total = M * fu;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / fu, c = (i % fu) * 8;
    const uint4 gv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + c), uv = *reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c);
    const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 g2 = unpack_bf16x2(gw[k]), u2 = unpack_bf16x2(uw[k]);
      const float g0 = fminf(g2.x, limit), g1 = fminf(g2.y, limit);
      const float u0 = fminf(fmaxf(u2.x, -limit), limit), u1 = fminf(fmaxf(u2.y, -limit), limit);
      o[k] = pack_bf16x2(g0 * sigmoid_f(slope * g0) * (u0 + 1.f), g1 * sigmoid_f(slope * g1) * (u1 + 1.f));
    }
    *reinterpret_cast<uint4*>(h + r * F + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// h = act(gate) * up; act 1: GELU (tanh form), 2: SiLU.  `live` (nullptr: all M rows) counts blocks of block_rows rows in use.
// V: columns per thread (1, or 8 for bf16).
template <typename T, int V>
__global__ void act_glu_kernel(const T* __restrict__ gu, T* __restrict__ h, long long M, int F, int act, const int* __restrict__ live,
                               int block_rows) {
  if (live) M = min(M, (long long)*live * block_rows);
  const int fv = F / V;
  const long long total = M * fv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / fv;
    const int c = int(i - r * fv) * V;
    float g[V], u[V];
    if constexpr (V == 8) {
      ldf8(gu + r * 2 * F + c, g);
      ldf8(gu + r * 2 * F + F + c, u);
    } else {
      g[0] = ldf(gu + r * 2 * F + c);
      u[0] = ldf(gu + r * 2 * F + F + c);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) g[k] = (act == 1 ? gelu_tanh_f(g[k]) : g[k] * sigmoid_f(g[k])) * u[k];
    if constexpr (V == 8) {
      *reinterpret_cast<uint4*>(h + r * F + c) =
          make_uint4(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3]), pack_bf16x2(g[4], g[5]), pack_bf16x2(g[6], g[7]));
    } else {
      stf(h + r * F + c, g[0]);
    }
  }
}

// out[n, c] = gelu(g[n, c]) * table[tokens[n], off + c] for c < dim, zero up to ld: a token's own input, gated.  A thread takes V columns (8 where all
// pieces are aligned: one load each instead of eight, and a division a piece; 4096 x 256: 5.8 us a column at a time, 3.4 so).
template <typename T, int V>
__global__ void token_gate_kernel(const T* g, const int* tokens, const T* table, long long ldt,
                                  int off, int dim, int ld, T* __restrict__ out, long long total) {
  pdl_launch_dependents();
  pdl_wait();
  const int pieces = ld / V;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = total < (1ll << 31) ? int(i) / pieces : i / pieces;
    const int c = int(i - n * pieces) * V;
    if constexpr (V == 8) {
      float a[8], t[8];
      if (c < dim) {
        ldf8(table + tokens[n] * ldt + off + c, t);
        ldf8(g + i * 8, a);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = c < dim ? gelu_tanh_f(a[j]) * t[j] : 0.f;
      stf4(out + i * 8, make_float4(a[0], a[1], a[2], a[3]));
      stf4(out + i * 8 + 4, make_float4(a[4], a[5], a[6], a[7]));
    } else {
      stf(out + i, c < dim ? gelu_tanh_f(ldf(g + i)) * ldf(table + tokens[n] * ldt + off + c) : 0.f);
    }
  }
}

__global__ void swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* dh, __nv_bfloat16* dgu,
                                  long long M, int F) {
  pdl_launch_dependents();
  pdl_wait();
  const int vpr = F / 8;
  const long long total = M * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = int(i % vpr) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    ld8(gu + r * 2 * F + c, g);
    ld8(gu + r * 2 * F + F + c, u);
    ld8(dh + r * F + c, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * sg;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (sg + silu * (1.f - sg));
    }
    st8(dgu + r * 2 * F + c, dg);
    st8(dgu + r * 2 * F + F + c, du);
  }
}

// ---------------------------------------------------------------------------------------------- GELU / add / scale
__global__ void gelu_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n8) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float f[8];
    ld8(x + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = gelu_tanh(f[j]);
    st8(y + i * 8, f);
  }
}
__global__ void gelu_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                __nv_bfloat16* __restrict__ dx, long long n8) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float f[8], g[8];
    ld8(x + i * 8, f);
    ld8(dy + i * 8, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      const float xx = f[j];
      const float t = tanhf(k0 * (xx + k1 * xx * xx * xx));
      const float dt = (1.f - t * t) * k0 * (1.f + 3.f * k1 * xx * xx);
      g[j] *= 0.5f * (1.f + t) + 0.5f * xx * dt;
    }
    st8(dx + i * 8, g);
  }
}
// out = a * alpha + b * beta  (b may be null)
__global__ void axpby_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, float alpha, float beta, long long n8) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float f[8];
    ld8(a + i * 8, f);
    if (b) {
      float g[8];
      ld8(b + i * 8, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * alpha + g[j] * beta;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] *= alpha;
    }
    st8(out + i * 8, f);
  }
}

// ---------------------------------------------------------------------------------------------- cached rows
// Rows [pos0, pos0 + n) of one sequence out of its blocks into [n, G, D] arrays.
__global__ void kv_gather_kernel(const uint4* k_cache, const uint4* v_cache, uint4* __restrict__ k_lin,
                                 uint4* __restrict__ v_lin, const int* table, int pos0, int G, int ku, int vu,
                                 int block_size) {
  pdl_launch_dependents();
  pdl_wait();
  const int pos = pos0 + blockIdx.x;
  const long long blk = table[pos / block_size];
  const int off = pos % block_size;
  for (int i = threadIdx.x; i < G * (ku + vu); i += blockDim.x) {
    const bool is_k = i < G * ku;
    const int j = is_k ? i : i - G * ku, w = is_k ? ku : vu;
    const int g = j / w, u = j % w;
    const long long src = ((blk * G + g) * block_size + off) * w + u, dst = ((long long)blockIdx.x * G + g) * w + u;
    if (is_k) k_lin[dst] = k_cache[src];
    else v_lin[dst] = v_cache[src];
  }
}

// ---------------------------------------------------------------------------------------------- greedy tokens
// Whether a at index i goes before b at j as the largest of a row: a NaN is the largest, of equals the first.
template <typename T>
__device__ __forceinline__ bool goes_before(T a, int i, T b, int j) {
  const bool na = a != a, nb = b != b;
  if (na || nb) return na && (!nb || i < j);
  return a > b || (a == b && i < j);
}
// Index of the largest element of every row.  (A conversion to fp32 and a library reduction took 13 us of a decode step.)  A cluster of 1 << log_parts CTAs
// takes a row and its first one compares their candidates: few long rows leave a CTA a row waiting for one load after the other.  A CTA a row / this:
// 8 x 32000 5.1 / 3.6 us, 8 x 128256 14.1 / 5.0, 64 x 128256 21.3 / 7.2; more rows than that keep a CTA a row (256 x 32000 7.7 / 5.1: one
// comparison an element instead of three).
template <bool F32, int NT>
__global__ void __launch_bounds__(NT) argmax_rows_kernel(const void* x, long long* __restrict__ out, int V, long long ld, int log_parts) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float bv[32];
  __shared__ int bi[32];
  const int parts = 1 << log_parts, part = blockIdx.x & (parts - 1);
  const long long row = blockIdx.x >> log_parts;
  const int len = log_parts ? (V / parts + 8) / 8 * 8 : V;
  const int from = part * len, end = from + len < V ? from + len : V;      // (from beyond V: nothing)
  float best = -INFINITY;
  int at = V;
  // a thread's elements come in order: a later one goes before only if it is larger, or the first NaN
  auto see = [&](float v, int i) { if (!(v <= best) && best == best) { best = v; at = i; } };
  auto take = [&](float v, int i) { if (goes_before(v, i, best, at)) { best = v; at = i; } };
  if (F32) {
    const float* r = static_cast<const float*>(x) + row * ld;
    if ((reinterpret_cast<uintptr_t>(r) & 15) == 0) {
      for (int c = from + threadIdx.x * 4; c + 3 < end; c += 4 * NT) {
        const float4 f = *reinterpret_cast<const float4*>(r + c);
        see(f.x, c); see(f.y, c + 1); see(f.z, c + 2); see(f.w, c + 3);
      }
      for (int c = end / 4 * 4 + threadIdx.x; c < end; c += NT) see(r[c], c);
    } else {
      for (int c = from + threadIdx.x; c < end; c += NT) see(r[c], c);
    }
  } else {
    const __nv_bfloat16* r = static_cast<const __nv_bfloat16*>(x) + row * ld;
    if ((reinterpret_cast<uintptr_t>(r) & 15) == 0) {
      for (int c = from + threadIdx.x * 8; c + 7 < end; c += 8 * NT) {
        float f[8];
        ld8(r + c, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) see(f[j], c + j);
      }
      for (int c = end / 8 * 8 + threadIdx.x; c < end; c += NT) see(__bfloat162float(r[c]), c);
    } else {
      for (int c = from + threadIdx.x; c < end; c += NT) see(__bfloat162float(r[c]), c);
    }
  }
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, at, o);
      take(v, i);
    }
  };
  reduce();
  if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = at; }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool there = threadIdx.x * 32 < NT;
    best = there ? bv[threadIdx.x] : -INFINITY;
    at = there ? bi[threadIdx.x] : V;
    reduce();
    if (threadIdx.x == 0) { bv[0] = best; bi[0] = at; }
  }
  if (parts > 1) {
    cluster_sync_all();
    if (part == 0 && threadIdx.x == 0)
      for (int i = 1; i < parts; ++i) take(ld_cluster_f32(smem_u32(bv), i), __float_as_int(ld_cluster_f32(smem_u32(bi), i)));
    cluster_sync_all();                  // a CTA's shared memory is read until here
  }
  if (part == 0 && threadIdx.x == 0) out[row] = at < V ? at : 0;
}

// ---------------------------------------------------------------------------------------------- embedding
template <typename IDX>
__global__ void embedding_fwd_kernel(const IDX* __restrict__ idx, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, long long n_tok, int D, int V) {
  pdl_launch_dependents();
  pdl_wait();
  const int vpr = D / 8;
  const long long total = n_tok * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = int(i % vpr) * 8;
    long long t = idx[r];
    t = t < 0 ? 0 : (t >= V ? V - 1 : t);
    *reinterpret_cast<uint4*>(out + r * D + c) = __ldg(reinterpret_cast<const uint4*>(table + t * D + c));
  }
}
// dtable[idx[r]] += dout[r]   (bf16x2 atomics; dtable must be zeroed or hold the running gradient)
__global__ void embedding_bwd_kernel(const long long* idx, const __nv_bfloat16* dout,
                                     __nv_bfloat16* __restrict__ dtable, long long n_tok, int D, int V) {
  pdl_launch_dependents();
  pdl_wait();
  const int ppr = D / 2;
  const long long total = n_tok * ppr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / ppr;
    const int c = int(i % ppr) * 2;
    long long t = idx[r];
    if (t < 0 || t >= V) continue;
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(dout + r * D + c);
    atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtable + t * D + c), v);
  }
}

// ---------------------------------------------------------------------------------------------- casts / fills
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n) {
  const long long n8 = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    const float4 a = *reinterpret_cast<const float4*>(in + i * 8);
    const float4 b = *reinterpret_cast<const float4*>(in + i * 8 + 4);
    uint4 u;
    u.x = pack_bf16x2(a.x, a.y); u.y = pack_bf16x2(a.z, a.w);
    u.z = pack_bf16x2(b.x, b.y); u.w = pack_bf16x2(b.z, b.w);
    *reinterpret_cast<uint4*>(out + i * 8) = u;
  }
  const long long tail = n8 * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (tail < n) out[tail] = __float2bfloat16(in[tail]);
}
__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, long long n) {
  const long long n8 = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float f[8];
    ld8(in + i * 8, f);
    *reinterpret_cast<float4*>(out + i * 8) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(out + i * 8 + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
  const long long tail = n8 * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (tail < n) out[tail] = __bfloat162float(in[tail]);
}

inline int grid_for(long long work, int threads) {
  long long g = (work + threads - 1) / threads;
  const long long cap = (long long)sm_count() * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return int(g);
}

}  // namespace lt

extern "C" {

int lt_rope(void* x, const float* cos_t, const float* sin_t, const int* pos, long long rows, int T, int heads, int hd,
            long long row_stride, int backward, void* stream) {
  using namespace lt;
  if (hd % 8 != 0 || row_stride % 8 != 0) return -int(kStatusBadArgument);
  const long long work = rows * heads * (hd / 8);
  if (work == 0) return 0;
  auto X = static_cast<__nv_bfloat16*>(x);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float sign = backward ? -1.f : 1.f;
  const int grid = grid_for(work, 256);
  if (work + (long long)grid * 256 < (1ll << 32))
    LT_RETURN_IF_CUDA(launch_chained(rope_kernel<unsigned>, grid, 256, 0, st, X, cos_t, sin_t, pos, rows, T, heads, hd, row_stride, sign));
  else
    LT_RETURN_IF_CUDA(launch_chained(rope_kernel<long long>, grid, 256, 0, st, X, cos_t, sin_t, pos, rows, T, heads, hd, row_stride, sign));
  LT_LAUNCH_CHECK();
  return 0;
}

// qkv: rows [Hq | Hkv | Hkv heads of hd] at pitch ld; pos, slots [rows] int32; q_out [rows, Hq, hd] or nullptr; caches as in
// lt_kv_append.  hd and ld are multiples of 8, qkv, q_out and the caches 16-byte aligned.
int lt_rope_append(void* qkv, long long ld, const float* cos_t, const float* sin_t, const int* pos, const int* slots, void* q_out, void* k_cache,
                   void* v_cache, long long rows, int Hq, int Hkv, int hd, int block_size, int kv_fp8, float k_scale, float v_scale, void* stream) {
  using namespace lt;
  if (hd % 8 != 0 || ld % 8 != 0 || block_size < 1 ||
      ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15))
    return -int(kStatusBadArgument);
  const long long work = rows * (Hq + 2 * Hkv) * (hd / 8);
  if (work == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto X = static_cast<__nv_bfloat16*>(qkv);
  auto Q = static_cast<__nv_bfloat16*>(q_out);
  const int grid = grid_for(work, 256);
  const bool small = work + (long long)grid * 256 < (1ll << 32);     // (see rope_kernel)
  const float ki = kv_fp8 ? 1.f / k_scale : 1.f, vi = kv_fp8 ? 1.f / v_scale : 1.f;
#define LT_ROPE_APPEND(F8, IDX) \
  LT_RETURN_IF_CUDA(launch_chained(rope_append_kernel<F8, IDX>, grid, 256, 0, st, X, ld, cos_t, sin_t, pos, slots, Q, k_cache, v_cache, rows, Hq, Hkv, hd, block_size, ki, vi))
  if (kv_fp8) { if (small) LT_ROPE_APPEND(true, unsigned); else LT_ROPE_APPEND(true, long long); }
  else { if (small) LT_ROPE_APPEND(false, unsigned); else LT_ROPE_APPEND(false, long long); }
#undef LT_ROPE_APPEND
  LT_LAUNCH_CHECK();
  return 0;
}

int lt_swiglu_fwd(const void* gu, void* h, long long M, int F, void* stream) {
  using namespace lt;
  if (F % 8 != 0) return -int(kStatusBadArgument);
  if (M == 0) return 0;
  LT_RETURN_IF_CUDA(launch_chained(swiglu_fwd_kernel, grid_for(M * (F / 8), 256), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(h), M, F));
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_clamped_glu(int fp32, const void* gu, void* h, long long M, int F, float limit, float slope, void* stream) {
  using namespace lt;
  if (M == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (fp32) clamped_glu_kernel<float><<<grid_for(M * F, 256), 256, 0, st>>>(static_cast<const float*>(gu), static_cast<float*>(h), M, F, limit, slope);
  else if (F % 8 == 0) clamped_glu8_kernel<<<grid_for(M * (F / 8), 256), 256, 0, st>>>(static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(h), M, F, limit, slope);
  else clamped_glu_kernel<__nv_bfloat16><<<grid_for(M * F, 256), 256, 0, st>>>(static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(h), M, F, limit, slope);
  LT_LAUNCH_CHECK();
  return 0;
}
// act(gate) * up for rows [gate | up] of gu [M, 2 F]; act 1: GELU (tanh form), 2: SiLU; live nullptr, or the number of blocks of
// block_rows rows to do (on the device).
int lt_act_glu(int fp32, const void* gu, void* h, long long M, int F, int act, const int* live, int block_rows, void* stream) {
  using namespace lt;
  if (act < 1 || act > 2) return -int(kStatusBadArgument);
  if (M == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  using bf = __nv_bfloat16;
  const bool v8 = !fp32 && F % 8 == 0 && ((reinterpret_cast<uintptr_t>(gu) | reinterpret_cast<uintptr_t>(h)) & 15) == 0;
  if (fp32) act_glu_kernel<float, 1><<<grid_for(M * F, 256), 256, 0, st>>>(static_cast<const float*>(gu), static_cast<float*>(h), M, F, act, live, block_rows);
  else if (v8) act_glu_kernel<bf, 8><<<grid_for(M * (F / 8), 256), 256, 0, st>>>(static_cast<const bf*>(gu), static_cast<bf*>(h), M, F, act, live, block_rows);
  else act_glu_kernel<bf, 1><<<grid_for(M * F, 256), 256, 0, st>>>(static_cast<const bf*>(gu), static_cast<bf*>(h), M, F, act, live, block_rows);
  LT_LAUNCH_CHECK();
  return 0;
}
// g [n, ld] -> out [n, ld]; table [vocab, ldt].
int lt_token_gate(int fp32, const void* g, const int* tokens, const void* table, long long ldt, int off, int dim, int ld, void* out,
                  int n, void* stream) {
  using namespace lt;
  if (dim > ld) return -int(kStatusBadArgument);
  if ((long long)n * ld == 0) return 0;
  const bool wide = ((dim | ld | off | ldt) & 7) == 0 &&
                    ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const long long total = (long long)n * (wide ? ld / 8 : ld);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  using bf = __nv_bfloat16;
#define LT_TOKEN_GATE(T, V) \
  LT_RETURN_IF_CUDA(launch_chained(token_gate_kernel<T, V>, grid_for(total, 256), 256, 0, st, static_cast<const T*>(g), tokens, static_cast<const T*>(table), ldt, off, dim, ld, static_cast<T*>(out), total))
  if (fp32) { if (wide) LT_TOKEN_GATE(float, 8); else LT_TOKEN_GATE(float, 1); }
  else { if (wide) LT_TOKEN_GATE(bf, 8); else LT_TOKEN_GATE(bf, 1); }
#undef LT_TOKEN_GATE
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_swiglu_bwd(const void* gu, const void* dh, void* dgu, long long M, int F, void* stream) {
  using namespace lt;
  if (F % 8 != 0) return -int(kStatusBadArgument);
  if (M == 0) return 0;
  LT_RETURN_IF_CUDA(launch_chained(swiglu_bwd_kernel, grid_for(M * (F / 8), 256), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dh), static_cast<__nv_bfloat16*>(dgu), M, F));
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_gelu_fwd(const void* x, void* y, long long n, void* stream) {
  using namespace lt;
  if (n % 8 != 0) return -int(kStatusBadArgument);
  if (n == 0) return 0;
  gelu_fwd_kernel<<<grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), n / 8);
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_gelu_bwd(const void* x, const void* dy, void* dx, long long n, void* stream) {
  using namespace lt;
  if (n % 8 != 0) return -int(kStatusBadArgument);
  if (n == 0) return 0;
  gelu_bwd_kernel<<<grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dx), n / 8);
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_axpby(const void* a, const void* b, void* out, float alpha, float beta, long long n, void* stream) {
  using namespace lt;
  if (n % 8 != 0) return -int(kStatusBadArgument);
  if (n == 0) return 0;
  axpby_kernel<<<grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b), static_cast<__nv_bfloat16*>(out), alpha, beta, n / 8);
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_embedding_fwd(const long long* idx, const void* table, void* out, long long n_tok, int D, int V, void* stream) {
  return lt_embedding_fwd_idx(idx, 0, table, out, n_tok, D, V, stream);
}
// idx32: the tokens are 32-bit.
int lt_embedding_fwd_idx(const void* idx, int idx32, const void* table, void* out, long long n_tok, int D, int V, void* stream) {
  using namespace lt;
  if (D % 8 != 0) return -int(kStatusBadArgument);
  if (n_tok == 0) return 0;
  // (a full stop: what was launched before it is complete, and the kernels of a step behind it count on that for its tables)
  auto tb = static_cast<const __nv_bfloat16*>(table);
  auto to = static_cast<__nv_bfloat16*>(out);
  const int grid = grid_for(n_tok * (D / 8), 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (idx32) embedding_fwd_kernel<int><<<grid, 256, 0, st>>>(static_cast<const int*>(idx), tb, to, n_tok, D, V);
  else embedding_fwd_kernel<long long><<<grid, 256, 0, st>>>(static_cast<const long long*>(idx), tb, to, n_tok, D, V);
  LT_LAUNCH_CHECK();
  return 0;
}
// Head sizes here are bytes of one (token, head) row; multiples of 16.
int lt_kv_gather(const void* k_cache, const void* v_cache, void* k_lin, void* v_lin, const int* table, int pos0, int n, int G,
                 int k_bytes, int v_bytes, int block_size, void* stream) {
  using namespace lt;
  if (n <= 0) return 0;
  if ((k_bytes & 15) || (v_bytes & 15)) return -4;
  LT_RETURN_IF_CUDA(launch_chained(kv_gather_kernel, n, 128, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(k_cache),
                                   static_cast<const uint4*>(v_cache), static_cast<uint4*>(k_lin), static_cast<uint4*>(v_lin), table, pos0, G, k_bytes / 16,
                                   v_bytes / 16, block_size));
  return 0;
}

// out[r] (64-bit) = index of the largest of the V elements of row r (bf16, or fp32) at pitch ld; a NaN is the largest, of equals the first.
int lt_argmax_rows(const void* x, int fp32, long long* out, int rows, int V, long long ld, void* stream) {
  using namespace lt;
  if (rows == 0) return 0;
  if (V < 1) return -int(kStatusBadArgument);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // two CTAs of 1024 threads fit an SM; a part of 4096 elements is one load a thread (fp32)
  int parts = 3;
  while (parts > 0 && (((long long)rows << parts) > 2 * sm_count() || (V >> parts) < 4096)) --parts;
  // short rows: fewer threads that have nothing to load (1024 x 512 fp32: 1024 threads a row 7.6 us, 256 2.8)
  const bool few = V >> parts <= (fp32 ? 2048 : 4096);
  const int threads = few ? 256 : 1024;
  auto kernel = few ? (fp32 ? argmax_rows_kernel<true, 256> : argmax_rows_kernel<false, 256>) : (fp32 ? argmax_rows_kernel<true, 1024> : argmax_rows_kernel<false, 1024>);
  if (parts > 0) LT_RETURN_IF_CUDA(launch_chained_clusters(kernel, rows << parts, threads, 0, 1 << parts, st, x, out, V, ld, parts));
  else LT_RETURN_IF_CUDA(launch_chained(kernel, rows, threads, 0, st, x, out, V, ld, 0));
  return 0;
}
int lt_embedding_bwd(const long long* idx, const void* dout, void* dtable, long long n_tok, int D, int V, void* stream) {
  using namespace lt;
  if (D % 2 != 0) return -int(kStatusBadArgument);
  if (n_tok == 0) return 0;
  LT_RETURN_IF_CUDA(launch_chained(embedding_bwd_kernel, grid_for(n_tok * (D / 2), 256), 256, 0, static_cast<cudaStream_t>(stream), idx, static_cast<const __nv_bfloat16*>(dout), static_cast<__nv_bfloat16*>(dtable), n_tok, D, V));
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_cast_f32_to_bf16(const float* in, void* out, long long n, void* stream) {
  using namespace lt;
  if (n == 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n / 8 + 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(in, static_cast<__nv_bfloat16*>(out), n);
  LT_LAUNCH_CHECK();
  return 0;
}
int lt_cast_bf16_to_f32(const void* in, float* out, long long n, void* stream) {
  using namespace lt;
  if (n == 0) return 0;
  cast_bf16_to_f32_kernel<<<grid_for(n / 8 + 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(in), out, n);
  LT_LAUNCH_CHECK();
  return 0;
}

}  // extern "C"
