// Paged-KV decode attention (one query token per sequence) with split-K, grouped-query heads and bf16 or
// e4m3 KV caches, plus the KV-append kernel that fills the cache.
//
// Reference: paged_attention_forward runs one THREAD per (sequence, head) with a 2048-float local score
// array and float block tables (src/backend/gpu_native/nn/nn_kernels.cu:1256-1312), flash-decoding exists
// only on the CPU (src/ops/flash_decoding.cpp:13-115), and nothing writes the cache.  Here a CTA owns a
// (sequence, KV head, split) and its warps stream chunks of 32 keys through an online softmax, each byte read once
// for the whole group of query heads: on the warp-level tensor-core instruction for caches in blocks of 8 keys or more (bf16 and
// e4m3), on CUDA cores for bf16 caches in smaller blocks, and, where neither applies, a warp a query head.  The splits' (max, sum,
// partial output) triples meet in a cluster or in a merge kernel.  Decode is bound by the cache's bytes.
// Cache layout: [num_blocks, Hkv, block_size, D] as in the reference.
#include "lt_cuda.h"
#include <cuda_fp8.h>
#include <initializer_list>

#include "common/host.h"
#include "common/ptx.cuh"
#include "common/scalar.cuh"

namespace lt {

// Plain (non-multicast) bulk asynchronous copy global -> this CTA's shared memory; bytes a multiple of 16, both
// addresses 16-byte aligned; completion is counted on the mbarrier.
__device__ __forceinline__ void bulk_g2s_pd(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(gsrc), "r"(bytes), "r"(bar) : "memory");
}

template <int D, bool FP8>
__device__ __forceinline__ void load_row(const void* base, long long elem_off, int lane, float (&out)[D / 32]) {
  constexpr int E = D / 32;
  if (FP8) {
    const __nv_fp8_e4m3* p = static_cast<const __nv_fp8_e4m3*>(base) + elem_off + lane * E;
#pragma unroll
    for (int i = 0; i < E; ++i) out[i] = float(p[i]);
  } else {
    const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(base) + elem_off + lane * E;
#pragma unroll
    for (int i = 0; i < E; i += 2) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + i));
      out[i] = f.x;
      out[i + 1] = f.y;
    }
  }
}

// part: [S, Hq, splits, D + 2] fp32 = (partial output normalised by its own sum, max, sum)
template <int D, bool FP8>
__global__ void paged_decode_kernel(const __nv_bfloat16* __restrict__ q, const void* __restrict__ k_cache,
                                    const void* __restrict__ v_cache, const int* __restrict__ block_tables,
                                    const int* __restrict__ context_lens, float* __restrict__ part, int S, int Hq, int Hkv,
                                    int block_size, int max_blocks, int splits, float scale, float k_scale, float v_scale, int window) {
  constexpr int E = D / 32;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int total = S * Hq * splits;
  if (warp_global >= total) return;
  const int sp = warp_global % splits;
  const int h = (warp_global / splits) % Hq;
  const int s = warp_global / (splits * Hq);
  const int hkv = h / (Hq / Hkv);
  const int ctx = context_lens[s];
  const int lo = window > 0 ? max(0, ctx - window) : 0;              // first visible key
  const int per = (ctx - lo + splits - 1) / splits;
  const int t0 = lo + sp * per, t1 = min(ctx, t0 + per);
  float qv[E];
  {
    const __nv_bfloat16* qp = q + ((long long)s * Hq + h) * D + lane * E;
#pragma unroll
    for (int i = 0; i < E; ++i) qv[i] = __bfloat162float(qp[i]) * scale * k_scale;
  }
  float m = -INFINITY, l = 0.f, acc[E];
#pragma unroll
  for (int i = 0; i < E; ++i) acc[i] = 0.f;
  for (int t = t0; t < t1; ++t) {
    const int blk = block_tables[(long long)s * max_blocks + t / block_size];
    const long long off = (((long long)blk * Hkv + hkv) * block_size + (t % block_size)) * D;
    float kv[E];
    load_row<D, FP8>(k_cache, off, lane, kv);
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < E; ++i) d += qv[i] * kv[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    const float nm = fmaxf(m, d);
    const float a = __expf(m - nm), p = __expf(d - nm);
    load_row<D, FP8>(v_cache, off, lane, kv);
    l = l * a + p;
#pragma unroll
    for (int i = 0; i < E; ++i) acc[i] = acc[i] * a + p * kv[i];
    m = nm;
  }
  float* out = part + (((long long)s * Hq + h) * splits + sp) * (D + 2);
  const float inv = l > 0.f ? v_scale / l : 0.f;
#pragma unroll
  for (int i = 0; i < E; ++i) out[lane * E + i] = acc[i] * inv;
  if (lane == 0) { out[D] = m; out[D + 1] = l; }
}


// ---------------------------------------------------------------------------------------------- grouped-query decode
// One CTA of four warps owns one (sequence, KV head, split): every K / V byte of its key range is read once for the
// whole group of G = Hq / Hkv query heads (the warp-per-query-head kernel above reads it G times and walks the keys
// one at a time).  A warp takes 32 keys at a time, and the K and V rows of the chunks ahead are already on their way:
//   loads    the rows of one cache block are contiguous, so a chunk is one or two bulk asynchronous copies each for K
//            and V (cp.async.bulk global -> shared with an mbarrier per stage); one lane requests chunk i + kStages - 1
//            before the warp starts on chunk i, so several KB per warp are in flight whatever the occupancy;
//   scores   lane = key: the lane reads its key row from shared memory 16 bytes at a time, starting at a unit rotated
//            by its lane number (rows are 128 / 256 bytes apart, so unrotated reads would all hit the same banks), and
//            forms the dot products with the G query vectors, which sit in shared memory pre-scaled;
//   softmax  per head, one max and one sum reduction per 32 keys; running (max, sum) kept per warp;
//   P V      lane = pair (D 64) or quad (D 128) of output columns: the probabilities of the chunk go through shared
//            memory, each V row is read as one conflict-free line and every lane updates its G x E accumulators.
// The warps' partial results are merged in shared memory and written in the (normalised output, max, sum) form that
// the merge kernel below combines across splits.  bf16 caches only; block_size must
// divide 32 or be a multiple of it.
constexpr int kPdWarps = 4;
constexpr int kPdMaxG = 8;

template <int D>
struct PdCfg {
  static constexpr int kStages = (D == 64) ? 3 : 2;
  static constexpr int kRowBytes = D * 2;
  static constexpr int kTileBytes = 32 * kRowBytes;                       // 32 keys of K (or V)
  static constexpr int kWarpBytes = kStages * 2 * kTileBytes;             // K and V tiles of every stage
  static constexpr int kOffQ = kPdWarps * kWarpBytes;                     // float q_s[G][D]
  static constexpr int kQUnitStride = kPdMaxG * 8 + 4;                    // floats per 8-column unit of q (all heads) + pad
  static constexpr int kOffP = kOffQ + (D / 8) * kQUnitStride * 4;       // float p_s[warps][G][32]
  static constexpr int kOffBar = kOffP + kPdWarps * 32 * kPdMaxG * 4;     // mbarriers [warps][stages]
  static constexpr int kSmemBytes = kOffBar + kPdWarps * kStages * 8 + 16;
};

template <int D>
__global__ void __launch_bounds__(kPdWarps * 32)
paged_decode_gqa_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                        const __nv_bfloat16* __restrict__ v_cache, const int* __restrict__ block_tables,
                        const int* __restrict__ context_lens, float* __restrict__ part, int S, int Hq, int Hkv, int block_size,
                        int max_blocks, int splits, float scale, int* status) {
  using Cfg = PdCfg<D>;
  constexpr int E = D / 32;
  constexpr int ST = Cfg::kStages;
  constexpr int UNITS = D / 8;                     // 16-byte units per row
  extern __shared__ __align__(128) uint8_t pd_smem[];
  const int G = Hq / Hkv;
  const int sp = blockIdx.x % splits;
  const int hkv = (blockIdx.x / splits) % Hkv;
  const int s = blockIdx.x / (splits * Hkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* q_s = reinterpret_cast<float*>(pd_smem + Cfg::kOffQ);                       // [D / 8][kQUnitStride]
  float* p_s = reinterpret_cast<float*>(pd_smem + Cfg::kOffP) + warp * 32 * kPdMaxG; // [G][32] of this warp
  uint8_t* my_tiles = pd_smem + warp * Cfg::kWarpBytes;
  const uint32_t bar0 = smem_u32(pd_smem + Cfg::kOffBar) + warp * ST * 8;
  __shared__ int abort_s, drain_s;
  // the reduction at the end reuses the tile area (all copies have been consumed by then)
  // q_s[unit j][head g][8 columns], units kQUnitStride floats apart: a lane that starts at unit (lane & 7) reads 32-byte
  // pieces whose 16-byte halves fall into distinct bank groups across its quarter-warp
  for (int i = threadIdx.x; i < G * D; i += blockDim.x) {
    const int g = i / D, d = i % D;
    q_s[(d >> 3) * Cfg::kQUnitStride + g * 8 + (d & 7)] = __bfloat162float(q[((long long)s * Hq + hkv * G + g) * D + d]) * scale;
  }
  if (threadIdx.x == 0) { abort_s = 0; drain_s = 0; }
  if (lane == 0) {
    for (int st = 0; st < ST; ++st) mbar_init(bar0 + 8u * st, 1);
    fence_barrier_init();
  }
  __syncthreads();
  volatile int* abort_flag = &abort_s;
  const int ctx = context_lens[s];
  const int per = ((ctx + splits - 1) / splits + 31) / 32 * 32;      // whole 32-key chunks per split
  const int t0 = sp * per, t1 = min(ctx, t0 + per);
  const int* bt = block_tables + (long long)s * max_blocks;
  const int n_chunks = t1 > t0 ? (t1 - t0 + 31) / 32 : 0;
  const int my_n = n_chunks > warp ? (n_chunks - warp + kPdWarps - 1) / kPdWarps : 0;   // chunks warp, warp + 4, ...

  // one lane requests the K and V rows of this warp's i-th chunk into stage i % ST
  auto request = [&](int i) {
    const int c0 = t0 + (warp + i * kPdWarps) * 32;
    const uint32_t bar = bar0 + 8u * (i % ST);
    uint8_t* kt = my_tiles + (i % ST) * 2 * Cfg::kTileBytes;
    uint8_t* vt = kt + Cfg::kTileBytes;
    // rows [c0, c0 + 32) clipped to the blocks the sequence owns (the last block is allocated whole)
    const int last_row = ((t1 - 1) / block_size + 1) * block_size;            // end of the last block holding a live key
    const int r_end = min(c0 + 32, last_row);
    mbar_expect_tx(bar, uint32_t(2 * (r_end - c0) * Cfg::kRowBytes));
    for (int r = c0; r < r_end;) {
      const int blk = bt[r / block_size];
      const int in_blk = r % block_size;
      const int n = min(block_size - in_blk, r_end - r);
      const long long src = (((long long)blk * Hkv + hkv) * block_size + in_blk) * D;
      bulk_g2s_pd(smem_u32(kt + (r - c0) * Cfg::kRowBytes), k_cache + src, uint32_t(n * Cfg::kRowBytes), bar);
      bulk_g2s_pd(smem_u32(vt + (r - c0) * Cfg::kRowBytes), v_cache + src, uint32_t(n * Cfg::kRowBytes), bar);
      r += n;
    }
  };

  float m[kPdMaxG], l[kPdMaxG], acc[kPdMaxG][E];
#pragma unroll
  for (int g = 0; g < kPdMaxG; ++g) {
    m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) acc[g][e] = 0.f;
  }
  if (lane == 0)
    for (int i = 0; i < ST - 1 && i < my_n; ++i) request(i);
  bool ok = true;
  for (int i = 0; i < my_n; ++i) {
    if (lane == 0 && i + ST - 1 < my_n) request(i + ST - 1);      // its stage was consumed in iteration i - 1
    ok = __all_sync(0xffffffffu, mbar_wait(bar0 + 8u * (i % ST), uint32_t(i / ST) & 1u, abort_flag, status, kStatusTimeoutFull));
    if (!ok) {
      // a copy never arrived: give the other requested stages one more bounded wait each, so that no copy of this
      // warp is still writing shared memory when the CTA leaves, then drop out (the result of the CTA is discarded)
      for (int r = i + 1; r < my_n && r < i + ST; ++r)
        mbar_wait(bar0 + 8u * (r % ST), uint32_t(r / ST) & 1u, &drain_s, status, kStatusTimeoutFull);
      break;
    }
    const int c0 = t0 + (warp + i * kPdWarps) * 32;
    const uint8_t* kt = my_tiles + (i % ST) * 2 * Cfg::kTileBytes;
    const uint8_t* vt = kt + Cfg::kTileBytes;
    // ---- scores of this lane's key for every head of the group
    const bool live = c0 + lane < t1;
    float sc[kPdMaxG];
#pragma unroll
    for (int g = 0; g < kPdMaxG; ++g) sc[g] = 0.f;
    if (live) {
      const uint4* kr = reinterpret_cast<const uint4*>(kt + lane * Cfg::kRowBytes);
#pragma unroll
      for (int jj = 0; jj < UNITS; ++jj) {
        const int j = (jj + lane) & (UNITS - 1);                  // rotated start: conflict-free across the quarter-warp
        const uint4 u = kr[j];
        const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
#pragma unroll
        for (int g = 0; g < kPdMaxG; ++g) {
          if (g < G) {
            const float4 q0 = *reinterpret_cast<const float4*>(q_s + j * Cfg::kQUnitStride + g * 8);
            const float4 q1 = *reinterpret_cast<const float4*>(q_s + j * Cfg::kQUnitStride + g * 8 + 4);
            sc[g] += a.x * q0.x + a.y * q0.y + b.x * q0.z + b.y * q0.w + c.x * q1.x + c.y * q1.y + d.x * q1.z + d.y * q1.w;
          }
        }
      }
    }
    // ---- online softmax per head over the 32 keys of the chunk
#pragma unroll
    for (int g = 0; g < kPdMaxG; ++g) {
      if (g < G) {
        float mx = live ? sc[g] : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float nm = fmaxf(m[g], mx);
        const float top = nm == -INFINITY ? 0.f : nm;      // (no score above minus infinity: weights of zero, or of NaN for NaN scores)
        const float a = (m[g] == -INFINITY) ? 0.f : __expf(m[g] - nm);
        const float pv = live ? __expf(sc[g] - top) : 0.f;
        float ps = pv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        l[g] = l[g] * a + ps;
        m[g] = nm;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[g][e] *= a;
        p_s[g * 32 + lane] = pv;
      }
    }
    __syncwarp();
    // ---- P V: lane = E output columns; V rows come from shared memory, one conflict-free line per key
    const int nk = min(32, t1 - c0);
#pragma unroll 4
    for (int kk = 0; kk < nk; ++kk) {
      const __nv_bfloat16* vr = reinterpret_cast<const __nv_bfloat16*>(vt + kk * Cfg::kRowBytes) + lane * E;
      float vv[E];
      if (E == 2) {
        const float2 f = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(vr));
        vv[0] = f.x; vv[1] = f.y;
      } else {
        const uint2 w2 = *reinterpret_cast<const uint2*>(vr);
        const float2 f0 = unpack_bf16x2(w2.x), f1 = unpack_bf16x2(w2.y);
        vv[0] = f0.x; vv[1] = f0.y; vv[E - 2] = f1.x; vv[E - 1] = f1.y;
      }
#pragma unroll
      for (int g = 0; g < kPdMaxG; ++g)
        if (g < G) {
          const float pgk = p_s[g * 32 + kk];              // same address for every lane: a broadcast
#pragma unroll
          for (int e = 0; e < E; ++e) acc[g][e] += pgk * vv[e];
        }
    }
    __syncwarp();            // every lane is done with this stage and with p_s before lane 0 requests into it again
  }
  // ---- merge the four warps (the tile area is free now: every requested copy has been waited for), write the partial result
  __syncthreads();
  float* red_m = reinterpret_cast<float*>(pd_smem);                 // [warps][G]
  float* red_l = red_m + kPdWarps * kPdMaxG;                         // [warps][G]
  float* red_o = red_l + kPdWarps * kPdMaxG;                         // [warps][G][D]
#pragma unroll
  for (int g = 0; g < kPdMaxG; ++g)
    if (g < G) {
      if (lane == 0) { red_m[warp * kPdMaxG + g] = ok ? m[g] : -INFINITY; red_l[warp * kPdMaxG + g] = ok ? l[g] : 0.f; }
#pragma unroll
      for (int e = 0; e < E; ++e) red_o[(warp * kPdMaxG + g) * D + lane * E + e] = acc[g][e];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += blockDim.x) {
    const int g = i / D, d = i % D;
    float gm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kPdWarps; ++w) gm = fmaxf(gm, red_m[w * kPdMaxG + g]);
    float lsum = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < kPdWarps; ++w) {
      const float lw = red_l[w * kPdMaxG + g];
      if (lw == 0.f) continue;                           // no keys; a NaN goes on
      const float a = __expf(red_m[w * kPdMaxG + g] - gm);
      lsum += lw * a;
      o += red_o[(w * kPdMaxG + g) * D + d] * a;
    }
    float* out = part + (((long long)s * Hq + hkv * G + g) * splits + sp) * (D + 2);
    out[d] = lsum == 0.f ? 0.f : o / lsum;
    if (d == 0) { out[D] = gm; out[D + 1] = lsum; }
  }
}

// ------------------------------------------------------------------------------------------------------------
// Grouped-query decode with the scores and the P V product on the warp-level tensor-core instruction.
//
// Same split of the work as paged_decode_gqa_kernel (one CTA of four warps, or six, per sequence, KV head and context split;
// a warp streams chunks of 32 keys through its own shared-memory stages), but the tiles arrive as TMA tensor copies in
// the 128-byte-swizzled layout, so that ldmatrix reads them without bank conflicts.  Both products are made transposed: keys (and then
// value columns) are the 16 rows of mma.sync m16n8k16, the group's query heads its 8 columns, so that groups of up to 8 heads, which is
// what models have, waste half or nothing instead of half to three quarters (heads as the 16 rows: twice the instructions, of the softmax too).
// The scores stay in registers; an 8 x 8 transpose in registers turns their fragments into those of the second product.  tcgen05 is not the tool
// here: its smallest tile is 64 rows and the kernel is bound by the K / V stream and by issue.  Six warps where heads have 128 columns (a CTA an SM),
// block tables read a chunk ahead by the lanes that request its runs: 32 sequences of 2048 to 4096 tokens, 8 KV heads of 128, 97 -> 72 us (61 at the copy rate).
template <int D>
struct PdMmaCfg {
  static constexpr int kWarps = (D == 64) ? 4 : 6;
  static constexpr int kStages = (D == 64) ? 3 : 2;
  static constexpr int kTileBytes = 32 * D * 2;                           // 32 keys of K (or V); D = 128: two 4 KB halves of 64 columns
  static constexpr int kWarpBytes = kStages * 2 * kTileBytes;
  static constexpr int kOffBar = kWarps * kWarpBytes;
  static constexpr int kSmemBytes = kOffBar + kWarps * kStages * 8 + 16 + 1024;   // + slack to align the tiles to 1024 bytes
};
constexpr int kPdMmaMaxG = 16;

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 8 x 8 matrix of 16-bit values, a row in four lanes, transposed.
__device__ __forceinline__ uint32_t movmatrix(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

// End of a CTA of the tensor-core decode kernels: shared memory (the tile area: every requested copy has been waited for) takes
// the warps' maxima, sums and outputs, [warps][16], [warps][16] and [warps][16][D] floats; the last one is returned.  m, l: of heads
// 8 n + 2 (lane % 4) + e, l this lane's share.
template <int W, int NT>
__device__ __forceinline__ float* pd_row_sums(uint8_t* smem, int warp, int lane, bool ok, const float (&m)[NT][2], float (&l)[NT][2]) {
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) l[n][e] += __shfl_xor_sync(0xffffffffu, l[n][e], o);
  __syncthreads();
  float* red_m = reinterpret_cast<float*>(smem);
  float* red_l = red_m + W * kPdMmaMaxG;
  if (lane < 4) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        red_m[warp * kPdMmaMaxG + n * 8 + lane * 2 + e] = ok ? m[n][e] : -INFINITY;
        red_l[warp * kPdMmaMaxG + n * 8 + lane * 2 + e] = ok ? l[n][e] : 0.f;
      }
  }
  return red_l + W * kPdMmaMaxG;
}
// What the maxima start from: below all scores but those of minus infinity, whose weights are zero then.
constexpr float kPdLowest = -3.402823466e38f;
// Scores of a chunk of 32 keys, [16-key block][fragment] for every 8 heads: rows are keys g and g + 8, columns heads 2 qd and 2 qd + 1.  They become
// weights; maxima m and sums l go on, and `a` is what the outputs so far are multiplied by.  factor: of the scores of this lane's heads.
template <int NT>
__device__ __forceinline__ void pd_softmax(float (&s)[NT][2][4], const float (&factor)[NT][2], float (&m)[NT][2], float (&l)[NT][2], float (&a)[NT][2], int g,
                                           int nk, int c0, int lo) {
  bool live[4];   // keys g, g + 8, g + 16, g + 24
#pragma unroll
  for (int i = 0; i < 4; ++i) live[i] = i * 8 + g < nk && c0 + i * 8 + g >= lo;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float& x = s[n][i >> 1][(i & 1) * 2 + e];
        x = live[i] ? x * factor[n][e] : -INFINITY;
        mx = fmaxf(mx, x);
      }
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float nm = fmaxf(m[n][e], mx);   // finite from the start (kPdLowest); fmaxf passes NaN over: a NaN score shows in the sum alone
      a[n][e] = __expf(m[n][e] - nm);
      m[n][e] = nm;
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float& x = s[n][i >> 1][(i & 1) * 2 + e];
        x = __expf(x - nm);
        sum += x;
      }
      l[n][e] = l[n][e] * a[n][e] + sum;
    }
}
// part: the group's rows [G][splits][D + 2]; out_scale multiplies the outputs.
template <int D, int W>
__device__ __forceinline__ void pd_write_partial(uint8_t* smem, float* part, int G, int splits, int sp, float out_scale) {
  const float* red_m = reinterpret_cast<const float*>(smem);
  const float* red_l = red_m + W * kPdMmaMaxG;
  const float* red_o = red_l + W * kPdMmaMaxG;
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += blockDim.x) {
    const int gg = i / D, d = i % D;
    float gm = -INFINITY;
#pragma unroll
    for (int w = 0; w < W; ++w) gm = fmaxf(gm, red_m[w * kPdMmaMaxG + gg]);
    float lsum = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float lw = red_l[w * kPdMmaMaxG + gg];
      if (lw == 0.f) continue;                                     // no keys; a NaN goes on
      const float a = __expf(red_m[w * kPdMmaMaxG + gg] - gm);
      lsum += lw * a;
      o += red_o[(w * kPdMmaMaxG + gg) * D + d] * a;
    }
    float* out = part + ((long long)gg * splits + sp) * (D + 2);   // (in shared memory: splits 1, sp 0)
    out[d] = lsum == 0.f ? 0.f : o / lsum * out_scale;
    if (d == 0) { out[D] = gm; out[D + 1] = lsum; }
  }
}

// A decode step's attention in one launch (STEP): the kernel reads the rows [q | k | v] of the product in front of it as they lie, turns queries and
// the newest key by the angles of their positions, writes the newest key and value to their cache slots and puts them into its own tile, and the
// splits of a (sequence, KV head), a cluster, merge their results through each other's shared memory.  Rotation and cache write, and the merge,
// were launches of their own: 2.6 and 3 to 5 us of a chain in which every kernel waits for the one before it.
struct PdStep {
  const __nv_bfloat16* qkv;      // [S, ld], 16-byte aligned rows
  long long ld;
  const float *cos_t, *sin_t;    // [positions, D / 2]
  const int *pos, *slots;        // [S]; a sequence's newest token is the last of its context; slot < 0: not written
  void *k_cache, *v_cache;
  float k_inv, v_inv;            // what 8-bit keys and values are multiplied by
  __nv_bfloat16* out;            // [S, Hq, D]
  int early;                     // block tables, lengths and all cached rows but the newest were complete before the kernels that may still run
};
constexpr int kPdMaxCluster = 16;

// Lane `lane` < D / 4 holds eight columns of the newest key (lane < D / 8) or value of (s, hkv), turned and rounded to bf16.
template <int D>
__device__ __forceinline__ uint4 pd_newest(const PdStep& f, int s, int hkv, int Hq, int Hkv, int lane) {
  if (lane >= D / 4) return make_uint4(0u, 0u, 0u, 0u);
  const bool is_k = lane < D / 8;
  const int u = is_k ? lane : lane - D / 8;
  uint4 w = *reinterpret_cast<const uint4*>(f.qkv + s * f.ld + (long long)(Hq + (is_k ? 0 : Hkv) + hkv) * D + u * 8);
  if (is_k) {
    const long long at = (long long)f.pos[s] * (D / 2) + u * 4;
    const float4 c = *reinterpret_cast<const float4*>(f.cos_t + at), n = *reinterpret_cast<const float4*>(f.sin_t + at);
    const float cc[4] = {c.x, c.y, c.z, c.w}, nn[4] = {n.x, n.y, n.z, n.w};
    uint32_t* p = &w.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = unpack_bf16x2(p[j]);
      p[j] = pack_bf16x2(a.x * cc[j] - a.y * nn[j], a.x * nn[j] + a.y * cc[j]);
    }
  }
  return w;
}
// Element offset of this lane's eight columns in its cache; negative: not cached.
template <int D>
__device__ __forceinline__ long long pd_newest_at(const PdStep& f, int s, int hkv, int Hkv, int block_size, int lane) {
  const int slot = f.slots[s];
  if (slot < 0 || lane >= D / 4) return -1;
  return (((long long)(slot / block_size) * Hkv + hkv) * block_size + slot % block_size) * D + (lane % (D / 8)) * 8;
}
// The cluster's splits (their rows [G][D + 2] at `mine` in each one's shared memory) merged and written, every CTA a share of the G * D results.
template <int D>
__device__ __forceinline__ void pd_merge_cluster(const float* mine, __nv_bfloat16* out, int G, int splits, int sp) {
  cluster_sync_all();
  const uint32_t base = smem_u32(mine);
  for (int e = sp * blockDim.x + threadIdx.x; e < G * D; e += splits * blockDim.x) {
    const int gg = e / D, d = e % D;
    float gm = -INFINITY, sum = 0.f, acc = 0.f;
    // eight splits at a time, their loads under way together
    for (int i0 = 0; i0 < splits; i0 += 8) {
      float m[8], l[8], o[8], top = gm;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        m[i] = -INFINITY; l[i] = 0.f; o[i] = 0.f;
        if (i0 + i < splits) {
          m[i] = ld_cluster_f32(base + (gg * (D + 2) + D) * 4, i0 + i);
          l[i] = ld_cluster_f32(base + (gg * (D + 2) + D + 1) * 4, i0 + i);
          o[i] = ld_cluster_f32(base + (gg * (D + 2) + d) * 4, i0 + i);
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) top = fmaxf(top, m[i]);
      const float before = gm == -INFINITY ? 0.f : __expf(gm - top);
      sum *= before; acc *= before; gm = top;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float w = !(l[i] <= 0.f) ? l[i] * __expf(m[i] - gm) : 0.f;     // a split without keys has outputs of zero
        sum += w;
        acc += w * o[i];
      }
    }
    out[e] = __float2bfloat16(sum == 0.f ? 0.f : acc / sum);       // zeros only where there is no key at all: a NaN goes out as one
  }
  cluster_sync_all();   // nobody leaves while its rows are read
}

// tmK / tmV: the caches seen as [num_blocks * Hkv * block_size rows, D] bf16, box 64 columns x min(block_size, 32) rows,
// 128-byte swizzle.  block_size is a multiple of 8 and divides 32 or is a multiple of it.
// NT: blocks of 8 query heads.
template <int D, int NT, bool STEP>
__global__ void __launch_bounds__(PdMmaCfg<D>::kWarps * 32)
paged_decode_mma_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                        const __nv_bfloat16* q, const int* block_tables,
                        const int* context_lens, float* __restrict__ part, int S, int Hq, int Hkv, int block_size,
                        int max_blocks, int splits, float scale, int window, int* status, const __grid_constant__ PdStep step) {
  using Cfg = PdMmaCfg<D>;
  constexpr int ST = Cfg::kStages;
  constexpr int KS = D / 16;     // k-steps of the score product
  constexpr int NU = D / 16;     // blocks of 16 value columns
  extern __shared__ uint8_t pd_raw[];
  uint8_t* pd_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pd_raw) + 1023) & ~uintptr_t(1023));
  const int G = Hq / Hkv;
  const int sp = blockIdx.x % splits;
  const int hkv = (blockIdx.x / splits) % Hkv;
  const int s = blockIdx.x / (splits * Hkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, qd = lane & 3;
  uint8_t* my_tiles = pd_smem + warp * Cfg::kWarpBytes;
  const uint32_t bar0 = smem_u32(pd_smem + Cfg::kOffBar) + warp * ST * 8;
  __shared__ int abort_s, drain_s;
  if (threadIdx.x == 0) { abort_s = 0; drain_s = 0; }
  if (lane == 0) {
    for (int st = 0; st < ST; ++st) mbar_init(bar0 + 8u * st, 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  pdl_launch_dependents();
  const bool early = STEP && step.early;
  if (!early) pdl_wait();
  __syncthreads();   // (each warp waits on barriers of its own; the flags are shared)
  volatile int* abort_flag = &abort_s;
  const int ctx = context_lens[s];
  const int lo = window > 0 ? max(0, ctx - window) : 0;              // first visible key
  const int base = lo & ~31;                                         // chunks start on multiples of 32 keys
  const int per = ((ctx - base + splits - 1) / splits + 31) / 32 * 32;      // whole 32-key chunks per split
  const int t0 = base + sp * per, t1 = min(ctx, t0 + per);
  const int* bt = block_tables + (long long)s * max_blocks;
  const int n_chunks = t1 > t0 ? (t1 - t0 + 31) / 32 : 0;
  const int my_n = n_chunks > warp ? (n_chunks - warp + Cfg::kWarps - 1) / Cfg::kWarps : 0;   // chunks warp, warp + kWarps, ...
  const int run = block_size < 32 ? block_size : 32;                 // rows per tensor copy

  // The copies of a chunk, a lane for every run of rows; its block, read from the table a chunk ahead, is in `next_blk`.
  const int last_row = t1 > t0 ? ((t1 - 1) / block_size + 1) * block_size : 0;   // end of the last block holding a live key
  int next_blk = 0;
  auto look_up = [&](int i) {
    const int r = t0 + (warp + i * Cfg::kWarps) * 32 + lane * run;
    if (i < my_n && lane * run < 32 && r < last_row) next_blk = bt[r / block_size];
  };
  auto request = [&](int i) {
    const int c0 = t0 + (warp + i * Cfg::kWarps) * 32;
    const uint32_t bar = bar0 + 8u * (i % ST);
    const int r_end = min(c0 + 32, last_row), r = c0 + lane * run;
    if (lane == 0) mbar_expect_tx(bar, uint32_t(2 * (r_end - c0) * D * 2));
    if (r < r_end) {
      const int row = (next_blk * Hkv + hkv) * block_size + r % block_size;
      uint8_t* kt = my_tiles + (i % ST) * 2 * Cfg::kTileBytes + (r - c0) * 128;
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        tma_load_2d(smem_u32(kt + h * 4096), &tmK, bar, h * 64, row);
        tma_load_2d(smem_u32(kt + Cfg::kTileBytes + h * 4096), &tmV, bar, h * 64, row);
      }
    }
    look_up(i + 1);
  };

  float m[NT][2], l[NT][2], factor[NT][2];   // of heads 8 n + 2 qd + e; l: this lane's share of the sums
  float oacc[NT][NU][4];                     // rows = value columns 16 u + g and + 8, columns = heads
#pragma unroll
  for (int n = 0; n < NT; ++n) {
#pragma unroll
    for (int e = 0; e < 2; ++e) { m[n][e] = kPdLowest; l[n][e] = 0.f; factor[n][e] = scale; }
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r) oacc[n][u][r] = 0.f;
  }

  look_up(0);
  for (int i = 0; i < ST - 1 && i < my_n; ++i) request(i);
  if (early) pdl_wait();
  // B fragments of the query block, transposed: columns = heads of the group (8 n + g), zero past G
  uint32_t qb[NT][KS][2];
  {
    const __nv_bfloat16* rows = STEP ? step.qkv + s * step.ld + (long long)hkv * G * D : q + ((long long)s * Hq + hkv * G) * D;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const bool there = n * 8 + g < G;
      const __nv_bfloat16* row = rows + (there ? n * 8 + g : 0) * D + qd * 2;
#pragma unroll
      for (int kk = 0; kk < KS; ++kk)
#pragma unroll
        for (int half = 0; half < 2; ++half) qb[n][kk][half] = there ? *reinterpret_cast<const uint32_t*>(row + kk * 16 + half * 8) : 0u;
    }
    if constexpr (STEP) {
      const long long at = (long long)step.pos[s] * (D / 2) + qd;
#pragma unroll
      for (int kk = 0; kk < KS; ++kk)
#pragma unroll
        for (int half = 0; half < 2; ++half) {     // columns kk * 16 + 8 half + 2 qd and the next
          const float c = step.cos_t[at + kk * 8 + half * 4], w = step.sin_t[at + kk * 8 + half * 4];
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const float2 a = unpack_bf16x2(qb[n][kk][half]);
            qb[n][kk][half] = pack_bf16x2(a.x * c - a.y * w, a.x * w + a.y * c);
          }
        }
    }
  }
  // the newest token's row, for the warp whose last chunk it ends
  const int newest = STEP && t1 == ctx && my_n > 0 && (n_chunks - 1) % Cfg::kWarps == warp ? my_n - 1 : -1;
  [[maybe_unused]] uint4 fresh;
  [[maybe_unused]] long long fresh_at = -1;
  if constexpr (STEP) {
    if (newest >= 0) {
      fresh = pd_newest<D>(step, s, hkv, Hq, Hkv, lane);
      fresh_at = pd_newest_at<D>(step, s, hkv, Hkv, block_size, lane);
    }
  }
  bool ok = true;
  const int lj = lane >> 3, lr = lane & 7;   // ldmatrix: this lane addresses row lr of matrix lj
  for (int i = 0; i < my_n; ++i) {
    if (i + ST - 1 < my_n) request(i + ST - 1);      // its stage was consumed in iteration i - 1
    ok = __all_sync(0xffffffffu, mbar_wait(bar0 + 8u * (i % ST), uint32_t(i / ST) & 1u, abort_flag, status, kStatusTimeoutFull));
    if (!ok) {
      // a copy never arrived: give the other requested stages one more bounded wait each, so that no copy of this
      // warp is still writing shared memory when the CTA leaves, then drop out (the result of the CTA is discarded)
      for (int r = i + 1; r < my_n && r < i + ST; ++r)
        mbar_wait(bar0 + 8u * (r % ST), uint32_t(r / ST) & 1u, &drain_s, status, kStatusTimeoutFull);
      break;
    }
    const int c0 = t0 + (warp + i * Cfg::kWarps) * 32;
    uint8_t* kt = my_tiles + (i % ST) * 2 * Cfg::kTileBytes;
    uint8_t* vt = kt + Cfg::kTileBytes;
    const uint32_t kt_addr = smem_u32(kt), vt_addr = smem_u32(vt);
    const int nk = min(32, t1 - c0);
    if constexpr (STEP) {
      if (i == newest) {
        if (lane < D / 4) {
          const int r = nk - 1, u = lane % (D / 8);
          *reinterpret_cast<uint4*>((lane < D / 8 ? kt : vt) + (u >> 3) * 4096 + r * 128 + (((u & 7) ^ (r & 7)) << 4)) = fresh;
          if (fresh_at >= 0) *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(lane < D / 8 ? step.k_cache : step.v_cache) + fresh_at) = fresh;
        }
        __syncwarp();
      }
    }
    if (nk < 32) {
      // rows past the context (the tail of the last block, or never copied) may hold anything: zero them in V so that
      // their zero probabilities do not meet a NaN
      if (lane >= nk) {
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {
          uint4* row = reinterpret_cast<uint4*>(vt + h * 4096 + lane * 128);
#pragma unroll
          for (int u = 0; u < 8; ++u) row[u] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      __syncwarp();
    }
    // ---- S^T = K Q^T: two blocks of 16 keys, which take turns (an instruction that adds to what the one before it makes waits for it)
    float sacc[NT][2][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int r = 0; r < 4; ++r) sacc[n][t][r] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      const int u = kk * 2 + (lj >> 1);                             // 16-byte unit of the row: columns 8 u .. 8 u + 7
      uint32_t ka[2][4];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int key = t * 16 + (lj & 1) * 8 + lr;
        ldsm_x4(kt_addr + (u >> 3) * 4096 + key * 128 + (((u & 7) ^ (key & 7)) << 4), ka[t][0], ka[t][1], ka[t][2], ka[t][3]);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int t = 0; t < 2; ++t) mma_16816(sacc[n][t], ka[t], qb[n][kk][0], qb[n][kk][1]);
    }
    float a[NT][2];
    pd_softmax<NT>(sacc, factor, m, l, a, g, nk, c0, lo);
    uint32_t pb[NT][4];                                             // weights of 8 keys each, heads as columns
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) pb[n][i] = movmatrix(pack_bf16x2(sacc[n][i >> 1][(i & 1) * 2], sacc[n][i >> 1][(i & 1) * 2 + 1]));
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        oacc[n][u][0] *= a[n][0]; oacc[n][u][1] *= a[n][1];
        oacc[n][u][2] *= a[n][0]; oacc[n][u][3] *= a[n][1];
      }
    // ---- O^T += V^T P^T: two steps of 16 keys, transposed loads of V
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const int key = ks * 16 + (lj >> 1) * 8 + lr;
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int w = u * 2 + (lj & 1);
        uint32_t va[4];
        ldsm_x4_trans(vt_addr + (w >> 3) * 4096 + key * 128 + (((w & 7) ^ (key & 7)) << 4), va[0], va[1], va[2], va[3]);
#pragma unroll
        for (int n = 0; n < NT; ++n) mma_16816(oacc[n][u], va, pb[n][2 * ks], pb[n][2 * ks + 1]);
      }
    }
    __syncwarp();            // every lane is done with this stage before the next copies into it are requested
  }
  // ---- merge the warps (the tile area is free now: every requested copy has been waited for), write the partial result
  float* red_o = pd_row_sums<Cfg::kWarps, NT>(pd_smem, warp, lane, ok, m, l);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r) red_o[(warp * kPdMmaMaxG + n * 8 + qd * 2 + (r & 1)) * D + u * 16 + g + (r >> 1) * 8] = oacc[n][u][r];
  if (STEP && !part) {
    float* mine = red_o + Cfg::kWarps * kPdMmaMaxG * D;
    pd_write_partial<D, Cfg::kWarps>(pd_smem, mine, G, 1, 0, 1.f);
    pd_merge_cluster<D>(mine, step.out + ((long long)s * Hq + hkv * G) * D, G, splits, sp);
  } else {
    pd_write_partial<D, Cfg::kWarps>(pd_smem, part + ((long long)s * Hq + hkv * G) * splits * (D + 2), G, splits, sp, 1.f);
  }
}

// The same split of the work for e4m3 caches.  What was a warp per query head that walked the keys one at a time (968 us for 8
// sequences of 4500 to 9000 tokens, 8 KV heads of 128 and 4 query heads each, where the cache streams in 18 us) reads every byte once for
// the whole group.  8-bit keys and values are exact as fp16 operands (one conversion for two of them):
//   scores   a lane takes 16 contiguous bytes of a key row, which are its fragments of four instructions when the columns of
//            the query are permuted alike; the query's rows are scaled by a power of two so that fp16 holds all of their bits;
//   P V      ldmatrix transposes pairs of bytes, so that a lane gets two neighbouring columns of two neighbouring keys; even and odd
//            columns are the upper and the lower eight rows of an instruction.  2^14 times a softmax weight is the sum of two fp16 parts (22 bits or more), each
//            with an instruction of its own.
// 8 sequences of 4500 to 9000 tokens: 60 us with heads as the instruction's 16 rows, 37 with heads as its 8 columns (1270 against about 600
// instructions a chunk of 8 KB; the table read a chunk ahead), bytes at the copy rate 17.
// Against 64 bits the 32-bit results are 1.3e-7 to 4.2e-7 off (2-norm; 32 to 16384 keys, one split or as many as a step takes, queries of
// size 0.1 to 4), those of the kernel before 1.5e-7 to 7.7e-6.
template <int D>
struct PdF8Cfg {
  static constexpr int kWarps = 4;
  static constexpr int kStages = (D == 64) ? 4 : 3;
  static constexpr int kTileBytes = 32 * D;                               // 32 keys of K (or V)
  static constexpr int kWarpBytes = kStages * 2 * kTileBytes;
  static constexpr int kOffBar = kWarps * kWarpBytes;
  static constexpr int kSmemBytes = kOffBar + kWarps * kStages * 8 + 16 + 1024;   // + slack to align the tiles to 1024 bytes
  static_assert(kOffBar >= (kWarps + 1) * kPdMmaMaxG * (D + 2) * 4, "the reduction at the end reuses the tile area");
};
constexpr float kPdWeightScale = 16384.f;   // weights are at most 1: the largest fp16 part is 2^14, the smallest 2^-24 stands for 2^-38

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero.
__device__ __forceinline__ void mma_f16_16816_0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// Four e4m3 values (low byte first) -> two fp16 pairs, exactly.
__device__ __forceinline__ void e4m3x4_to_f16(uint32_t four, uint32_t& lo, uint32_t& hi) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}" : "=r"(lo), "=r"(hi) : "r"(four));
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// x = hi + lo as two fp16 pairs.
__device__ __forceinline__ void split_f16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_f16x2(x0 - f.x, x1 - f.y);
}

// tmK / tmV: the caches seen as [num_blocks * Hkv * block_size rows, D] bytes, box D columns x min(block_size, 32) rows; rows of 128
// bytes arrive with the 128-byte swizzle, rows of 64 as they are.
template <int D, int NT, bool STEP>
__global__ void __launch_bounds__(PdF8Cfg<D>::kWarps * 32)
paged_decode_f8_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                       const __nv_bfloat16* q, const int* block_tables,
                       const int* context_lens, float* __restrict__ part, int S, int Hq, int Hkv, int block_size,
                       int max_blocks, int splits, float scale, float v_scale, int window, int* status, const __grid_constant__ PdStep step) {
  using Cfg = PdF8Cfg<D>;
  constexpr int ST = Cfg::kStages;
  constexpr int KS = D / 16;     // k-steps of the score product
  constexpr int NU = D / 16;     // 16-byte units of a value row
  extern __shared__ uint8_t pd_raw[];
  uint8_t* pd_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pd_raw) + 1023) & ~uintptr_t(1023));
  const int G = Hq / Hkv;
  const int sp = blockIdx.x % splits;
  const int hkv = (blockIdx.x / splits) % Hkv;
  const int s = blockIdx.x / (splits * Hkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, qd = lane & 3;
  uint8_t* my_tiles = pd_smem + warp * Cfg::kWarpBytes;
  const uint32_t bar0 = smem_u32(pd_smem + Cfg::kOffBar) + warp * ST * 8;
  __shared__ int abort_s, drain_s;
  if (threadIdx.x == 0) { abort_s = 0; drain_s = 0; }
  if (lane == 0) {
    for (int st = 0; st < ST; ++st) mbar_init(bar0 + 8u * st, 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  pdl_launch_dependents();
  const bool early = STEP && step.early;
  if (!early) pdl_wait();
  // offset of 16-byte unit u of row r inside a tile
  auto unit = [](int r, int u) { return D == 128 ? r * 128 + ((u ^ (r & 7)) << 4) : r * 64 + (u << 4); };
  __syncthreads();   // (each warp waits on barriers of its own; the flags are shared)
  volatile int* abort_flag = &abort_s;
  const int ctx = context_lens[s];
  const int lo = window > 0 ? max(0, ctx - window) : 0;              // first visible key
  const int base = lo & ~31;                                         // chunks start on multiples of 32 keys
  const int per = ((ctx - base + splits - 1) / splits + 31) / 32 * 32;      // whole 32-key chunks per split
  const int t0 = base + sp * per, t1 = min(ctx, t0 + per);
  const int* bt = block_tables + (long long)s * max_blocks;
  const int n_chunks = t1 > t0 ? (t1 - t0 + 31) / 32 : 0;
  const int my_n = n_chunks > warp ? (n_chunks - warp + Cfg::kWarps - 1) / Cfg::kWarps : 0;   // chunks warp, warp + kWarps, ...
  const int run = block_size < 32 ? block_size : 32;                 // rows per tensor copy

  // The copies of a chunk, a lane for every run of rows; its block, read from the table a chunk ahead, is in `next_blk`.
  const int last_row = t1 > t0 ? ((t1 - 1) / block_size + 1) * block_size : 0;   // end of the last block holding a live key
  int next_blk = 0;
  auto look_up = [&](int i) {
    const int r = t0 + (warp + i * Cfg::kWarps) * 32 + lane * run;
    if (i < my_n && lane * run < 32 && r < last_row) next_blk = bt[r / block_size];
  };
  auto request = [&](int i) {
    const int c0 = t0 + (warp + i * Cfg::kWarps) * 32;
    const uint32_t bar = bar0 + 8u * (i % ST);
    const int r_end = min(c0 + 32, last_row), r = c0 + lane * run;
    if (lane == 0) mbar_expect_tx(bar, uint32_t(2 * (r_end - c0) * D));
    if (r < r_end) {
      const int row = (next_blk * Hkv + hkv) * block_size + r % block_size;
      const uint32_t kt = smem_u32(my_tiles + (i % ST) * 2 * Cfg::kTileBytes) + (r - c0) * D;
      tma_load_2d(kt, &tmK, bar, 0, row);
      tma_load_2d(kt + Cfg::kTileBytes, &tmV, bar, 0, row);
    }
    look_up(i + 1);
  };

  float m[NT][2], l[NT][2], factor[NT][2];   // of heads 8 n + 2 qd + e; l: this lane's share of the sums
  float oacc[NT][NU][4];                     // rows = value columns 16 u + 2 g and the next, columns = heads
#pragma unroll
  for (int n = 0; n < NT; ++n) {
#pragma unroll
    for (int e = 0; e < 2; ++e) { m[n][e] = kPdLowest; l[n][e] = 0.f; }
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r) oacc[n][u][r] = 0.f;
  }

  look_up(0);
  for (int i = 0; i < ST - 1 && i < my_n; ++i) request(i);
  if (early) pdl_wait();
  // B fragments of the query block, transposed, its columns permuted: step kk = 4 h + r takes columns 64 h + 16 qd + 4 r + {0 .. 3}.  Columns =
  // heads of the group (8 n + g), zero past G, scaled by a power of two to a largest value in [2^14, 2^15).
  uint32_t qb[NT][KS][2];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    uint2 raw[KS];
    float top = 0.f;
    const bool there = n * 8 + g < G;
    const __nv_bfloat16* rows = STEP ? step.qkv + s * step.ld + (long long)hkv * G * D : q + ((long long)s * Hq + hkv * G) * D;
    const __nv_bfloat16* row = rows + (there ? n * 8 + g : 0) * D + qd * 16;
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      raw[kk] = there ? *reinterpret_cast<const uint2*>(row + (kk >> 2) * 64 + (kk & 3) * 4) : make_uint2(0u, 0u);
      if constexpr (STEP) {
        const long long at = (long long)step.pos[s] * (D / 2) + (kk >> 2) * 32 + qd * 8 + (kk & 3) * 2;
        const float2 c = *reinterpret_cast<const float2*>(step.cos_t + at), w = *reinterpret_cast<const float2*>(step.sin_t + at);
        const float2 x = unpack_bf16x2(raw[kk].x), y = unpack_bf16x2(raw[kk].y);
        raw[kk] = make_uint2(pack_bf16x2(x.x * c.x - x.y * w.x, x.x * w.x + x.y * c.x), pack_bf16x2(y.x * c.y - y.y * w.y, y.x * w.y + y.y * c.y));
      }
      const float2 a = unpack_bf16x2(raw[kk].x), b = unpack_bf16x2(raw[kk].y);
      top = fmaxf(top, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
    }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    // (a row of zeros or with an infinity stays as it is)
    const int e = top > 0.f && top <= 3.4e38f ? max(-120, min(100, 14 - ilogbf(top))) : 0;
    const float up = ldexpf(1.f, e), down = scale * ldexpf(1.f, -e);
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      const float2 a = unpack_bf16x2(raw[kk].x), b = unpack_bf16x2(raw[kk].y);
      qb[n][kk][0] = pack_f16x2(a.x * up, a.y * up);
      qb[n][kk][1] = pack_f16x2(b.x * up, b.y * up);
    }
    // scores lie in other lanes than their query: those of heads 2 qd and 2 qd + 1 here
    factor[n][0] = __shfl_sync(0xffffffffu, down, qd * 8);
    factor[n][1] = __shfl_sync(0xffffffffu, down, qd * 8 + 4);
  }
  // the newest token's row, for the warp whose last chunk it ends
  const int newest = STEP && t1 == ctx && my_n > 0 && (n_chunks - 1) % Cfg::kWarps == warp ? my_n - 1 : -1;
  [[maybe_unused]] uint4 fresh;
  [[maybe_unused]] long long fresh_at = -1;
  if constexpr (STEP) {
    if (newest >= 0) {
      fresh = pd_newest<D>(step, s, hkv, Hq, Hkv, lane);
      fresh_at = pd_newest_at<D>(step, s, hkv, Hkv, block_size, lane);
    }
  }
  bool ok = true;
  const int lj = lane >> 3, lr = lane & 7;   // ldmatrix: this lane addresses row lr of matrix lj
  for (int i = 0; i < my_n; ++i) {
    if (i + ST - 1 < my_n) request(i + ST - 1);      // its stage was consumed in iteration i - 1
    ok = __all_sync(0xffffffffu, mbar_wait(bar0 + 8u * (i % ST), uint32_t(i / ST) & 1u, abort_flag, status, kStatusTimeoutFull));
    if (!ok) {
      // a copy never arrived: give the other requested stages one more bounded wait each, so that no copy of this
      // warp is still writing shared memory when the CTA leaves, then drop out (the result of the CTA is discarded)
      for (int r = i + 1; r < my_n && r < i + ST; ++r)
        mbar_wait(bar0 + 8u * (r % ST), uint32_t(r / ST) & 1u, &drain_s, status, kStatusTimeoutFull);
      break;
    }
    const int c0 = t0 + (warp + i * Cfg::kWarps) * 32;
    uint8_t* kt = my_tiles + (i % ST) * 2 * Cfg::kTileBytes;
    uint8_t* vt = kt + Cfg::kTileBytes;
    const uint32_t vt_addr = smem_u32(vt);
    const int nk = min(32, t1 - c0);
    if constexpr (STEP) {
      if (i == newest) {
        if (lane < D / 4) {
          const int r = nk - 1, u = lane % (D / 8);
          const float inv = lane < D / 8 ? step.k_inv : step.v_inv;
          alignas(8) uint8_t eight[8];
          const uint32_t* p = &fresh.x;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 a = unpack_bf16x2(p[j]);
            eight[2 * j] = __nv_fp8_e4m3(a.x * inv).__x;
            eight[2 * j + 1] = __nv_fp8_e4m3(a.y * inv).__x;
          }
          const uint2 two = *reinterpret_cast<const uint2*>(eight);
          *reinterpret_cast<uint2*>((lane < D / 8 ? kt : vt) + unit(r, u >> 1) + (u & 1) * 8) = two;
          if (fresh_at >= 0) *reinterpret_cast<uint2*>(static_cast<uint8_t*>(lane < D / 8 ? step.k_cache : step.v_cache) + fresh_at) = two;
        }
        __syncwarp();
      }
    }
    if (nk < 32 || c0 < lo) {
      // rows past the context or before the window may hold anything: zero them in V so that their zero weights do not meet a NaN
      // (a window starts in a warp's first chunk, whose stage a later copy fills again: that copy has to come after these stores)
      if (lane >= nk || c0 + lane < lo) {
#pragma unroll
        for (int u = 0; u < NU; ++u) *reinterpret_cast<uint4*>(vt + lane * D + u * 16) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
      }
      __syncwarp();
    }
    // ---- S^T = K Q^T: two blocks of 16 keys, which take turns
    float sacc[NT][2][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int r = 0; r < 4; ++r) sacc[n][t][r] = 0.f;
#pragma unroll
    for (int h = 0; h < D / 64; ++h) {
      uint4 w[2][2];                                         // [block][keys g / g + 8]
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int half = 0; half < 2; ++half) w[t][half] = *reinterpret_cast<const uint4*>(kt + unit(t * 16 + half * 8 + g, h * 4 + qd));
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          uint32_t ka[4];
#pragma unroll
          for (int half = 0; half < 2; ++half) e4m3x4_to_f16(r == 0 ? w[t][half].x : r == 1 ? w[t][half].y : r == 2 ? w[t][half].z : w[t][half].w, ka[half], ka[2 + half]);
#pragma unroll
          for (int n = 0; n < NT; ++n) mma_f16_16816(sacc[n][t], ka, qb[n][h * 4 + r][0], qb[n][h * 4 + r][1]);
        }
    }
    float a[NT][2];
    pd_softmax<NT>(sacc, factor, m, l, a, g, nk, c0, lo);
    uint32_t ph[NT][4], pl[NT][4];                           // weights of 8 keys each, heads as columns
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t hi, low;
        split_f16x2(sacc[n][i >> 1][(i & 1) * 2] * kPdWeightScale, sacc[n][i >> 1][(i & 1) * 2 + 1] * kPdWeightScale, hi, low);
        ph[n][i] = movmatrix(hi);
        pl[n][i] = movmatrix(low);
      }
    // ---- O^T += V^T P^T: two steps of 16 keys.  A chunk's products start from zero and are added with rounding: the instruction cuts off what it
    // adds to its accumulator, which over hundreds of chunks would add up.
#pragma unroll
    for (int u2 = 0; u2 < NU / 2; ++u2) {
      float pv[NT][2][4];                                    // [unit][fragment]
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const int key = ks * 16 + (lj & 1) * 8 + lr;
        uint32_t b[2][2];                                    // [unit][keys 0 .. 7 / 8 .. 15 of the step]
        ldsm_x4_trans(vt_addr + unit(key, u2 * 2 + (lj >> 1)), b[0][0], b[0][1], b[1][0], b[1][1]);
        uint32_t va[2][4];                                   // rows 2 g (registers 0, 2) and 2 g + 1 (1, 3) of the unit
#pragma unroll
        for (int uu = 0; uu < 2; ++uu)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t ka, kb;                                 // both columns of a key, and of the next
            e4m3x4_to_f16(b[uu][h], ka, kb);
            va[uu][2 * h] = __byte_perm(ka, kb, 0x5410);
            va[uu][2 * h + 1] = __byte_perm(ka, kb, 0x7632);
          }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int uu = 0; uu < 2; ++uu) {
            if (ks == 0) mma_f16_16816_0(pv[n][uu], va[uu], ph[n][0], ph[n][1]);
            else mma_f16_16816(pv[n][uu], va[uu], ph[n][2], ph[n][3]);
          }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int uu = 0; uu < 2; ++uu) mma_f16_16816(pv[n][uu], va[uu], pl[n][2 * ks], pl[n][2 * ks + 1]);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int uu = 0; uu < 2; ++uu)
#pragma unroll
          for (int r = 0; r < 4; ++r) oacc[n][u2 * 2 + uu][r] = fmaf(oacc[n][u2 * 2 + uu][r], a[n][r & 1], pv[n][uu][r]);
    }
    __syncwarp();            // every lane is done with this stage before the next copies into it are requested
  }
  float* red_o = pd_row_sums<Cfg::kWarps, NT>(pd_smem, warp, lane, ok, m, l);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float2*>(red_o + (warp * kPdMmaMaxG + n * 8 + qd * 2 + e) * D + u * 16 + g * 2) = make_float2(oacc[n][u][e], oacc[n][u][2 + e]);
  if (STEP && !part) {
    float* mine = red_o + Cfg::kWarps * kPdMmaMaxG * D;
    pd_write_partial<D, Cfg::kWarps>(pd_smem, mine, G, 1, 0, v_scale / kPdWeightScale);
    pd_merge_cluster<D>(mine, step.out + ((long long)s * Hq + hkv * G) * D, G, splits, sp);
  } else {
    pd_write_partial<D, Cfg::kWarps>(pd_smem, part + ((long long)s * Hq + hkv * G) * splits * (D + 2), G, splits, sp, v_scale / kPdWeightScale);
  }
}

template <int D>
__global__ void paged_decode_merge_kernel(const float* part, __nv_bfloat16* __restrict__ o, int rows, int splits,
                                          const __nv_bfloat16* gate, long long ldg, int Hq, int vdim) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  constexpr int E = D / 32;
  // A lane reads maximum and sum of one split, so that their loads are under way together, as are then those of the outputs (one split
  // after another: 5.4 us for 32 rows of 16 splits, two thirds of them waiting).
  const float* p0 = part + (long long)row * splits * (D + 2);
  float gm = -INFINITY;
  for (int sp = lane; sp < splits; sp += 32) gm = fmaxf(gm, p0[(long long)sp * (D + 2) + D]);
  gm = warp_max(gm);
  float wsum = 0.f, acc[E];
#pragma unroll
  for (int i = 0; i < E; ++i) acc[i] = 0.f;
  for (int s0 = 0; s0 < splits; s0 += 32) {
    const float* p = p0 + (long long)s0 * (D + 2);
    const int n = min(32, splits - s0);
    float w = 0.f;
    if (lane < n) {
      const float l = p[(long long)lane * (D + 2) + D + 1];
      if (!(l <= 0.f)) w = l * __expf(p[(long long)lane * (D + 2) + D] - gm);
    }
    wsum += w;
#pragma unroll 8
    for (int j = 0; j < n; ++j) {
      const float wj = __shfl_sync(0xffffffffu, w, j);
      // a split without keys has outputs of zero
#pragma unroll
      for (int i = 0; i < E; ++i) acc[i] += wj * p[(long long)j * (D + 2) + lane * E + i];
    }
  }
  wsum = warp_sum(wsum);
  float inv = wsum > 0.f ? 1.f / wsum : 0.f;
  if (gate) inv /= 1.f + expf(-__bfloat162float(gate[(row / Hq) * ldg + row % Hq]));     // times sigmoid(gate) of this head
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (lane * E + i < vdim) o[(long long)row * vdim + lane * E + i] = __float2bfloat16(acc[i] * inv);
}

// slot = block * block_size + offset for each new token.
template <bool FP8>
__global__ void kv_append_kernel(const __nv_bfloat16* __restrict__ k_new, const __nv_bfloat16* __restrict__ v_new,
                                 void* __restrict__ k_cache, void* __restrict__ v_cache, const int* __restrict__ slots,
                                 long long n_tok, int Hkv, int D, int block_size, float k_inv_scale, float v_inv_scale) {
  const long long total = n_tok * Hkv * D;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int d = int(i % D);
    const int h = int((i / D) % Hkv);
    const long long t = i / ((long long)D * Hkv);
    const int slot = slots[t];
    if (slot < 0) continue;
    const long long dst = (((long long)(slot / block_size) * Hkv + h) * block_size + (slot % block_size)) * D + d;
    if (FP8) {
      static_cast<__nv_fp8_e4m3*>(k_cache)[dst] = __nv_fp8_e4m3(__bfloat162float(k_new[i]) * k_inv_scale);
      static_cast<__nv_fp8_e4m3*>(v_cache)[dst] = __nv_fp8_e4m3(__bfloat162float(v_new[i]) * v_inv_scale);
    } else {
      static_cast<__nv_bfloat16*>(k_cache)[dst] = k_new[i];
      static_cast<__nv_bfloat16*>(v_cache)[dst] = v_new[i];
    }
  }
}

template <class K>
static int configure_clustered(K kernel, int smem, OncePerDevice& configured) {
  if (configured.pending()) {
    LT_RETURN_IF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    LT_RETURN_IF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    configured.finish();
  }
  return 0;
}
// Clusters of `cluster` CTAs that an empty GPU holds at once; negative: an error.
template <class K>
static int clusters_at_once(K kernel, int warps, int smem, int cluster) {
  OncePerDevice configured;
  if (const int rc = configure_clustered(kernel, smem, configured)) return -rc;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  return e == cudaSuccess ? n : -int(e);
}
// One of the tensor-core decode kernels, by cache type, head size and heads of a group; cluster: CTAs of a cluster.
template <class K, class... A>
static int launch_clustered(K kernel, int warps, int smem, OncePerDevice& configured, int ctas, int cluster, cudaStream_t st, A... args) {
  if (const int rc = configure_clustered(kernel, smem, configured)) return rc;
  LT_RETURN_IF_CUDA(launch_chained_clusters(kernel, ctas, warps * 32, smem, cluster, st, args...));
  LT_LAUNCH_CHECK();
  return 0;
}
template <bool STEP, int D, int NT>
static int launch_tensor_decode_by(const CUtensorMap& tmK, const CUtensorMap& tmV, const __nv_bfloat16* q, const int* bt, const int* ctx, float* part, int S,
                                   int Hq, int Hkv, int block_size, int max_blocks, int splits, float scale, int kv_fp8, float v_scale, int window, int* status,
                                   const PdStep& step, int ctas, int cluster, cudaStream_t st) {
  static OncePerDevice done8, done16;
  if (kv_fp8)
    return launch_clustered(paged_decode_f8_kernel<D, NT, STEP>, PdF8Cfg<D>::kWarps, PdF8Cfg<D>::kSmemBytes, done8, ctas, cluster, st, tmK, tmV, q, bt, ctx, part, S, Hq, Hkv, block_size,
                            max_blocks, splits, scale, v_scale, window, status, step);
  return launch_clustered(paged_decode_mma_kernel<D, NT, STEP>, PdMmaCfg<D>::kWarps, PdMmaCfg<D>::kSmemBytes, done16, ctas, cluster, st, tmK, tmV, q, bt, ctx, part, S, Hq, Hkv, block_size,
                          max_blocks, splits, scale, window, status, step);
}
template <bool STEP>
static int launch_tensor_decode(const CUtensorMap& tmK, const CUtensorMap& tmV, const __nv_bfloat16* q, const int* bt, const int* ctx, float* part, int S, int Hq,
                                int Hkv, int D, int block_size, int max_blocks, int splits, float scale, int kv_fp8, float v_scale, int window, int* status,
                                const PdStep& step, int ctas, int cluster, cudaStream_t st) {
#define LT_PD(DD, NT) \
  launch_tensor_decode_by<STEP, DD, NT>(tmK, tmV, q, bt, ctx, part, S, Hq, Hkv, block_size, max_blocks, splits, scale, kv_fp8, v_scale, window, status, step, ctas, cluster, st)
  if (Hq / Hkv <= 8) return D == 64 ? LT_PD(64, 1) : LT_PD(128, 1);
  return D == 64 ? LT_PD(64, 2) : LT_PD(128, 2);
#undef LT_PD
}

static int merge_splits(const float* part, __nv_bfloat16* o, int rows, int splits, int D, const __nv_bfloat16* gate, long long ldg, int Hq, int vdim,
                        cudaStream_t st) {
  const int mb = (rows + 3) / 4;
  if (D == 64) LT_RETURN_IF_CUDA(launch_chained(paged_decode_merge_kernel<64>, mb, 128, 0, st, part, o, rows, splits, gate, ldg, Hq, vdim));
  else LT_RETURN_IF_CUDA(launch_chained(paged_decode_merge_kernel<128>, mb, 128, 0, st, part, o, rows, splits, gate, ldg, Hq, vdim));
  return 0;
}

}  // namespace lt

extern "C" {

// q: [S, Hq, D] bf16; caches [num_blocks, Hkv, block_size, D] bf16 (kv_fp8 = 0) or e4m3 (kv_fp8 = 1, with the
// dequantisation scales k_scale / v_scale); block_tables [S, max_blocks] int32; context_lens [S] int32;
// part: scratch [S, Hq, splits, D + 2] fp32; o: [S, Hq, D] bf16.  num_blocks: blocks in the caches (0: not known, which
// rules out the tensor-copy kernel).
int lt_paged_decode(const void* q, const void* k_cache, const void* v_cache, const int* block_tables, const int* context_lens,
                    float* part, void* o, int S, int Hq, int Hkv, int D, int block_size, int max_blocks, int num_blocks,
                    int splits, float scale, int kv_fp8, float k_scale, float v_scale, void* stream) {
  return lt_paged_decode_window(q, k_cache, v_cache, block_tables, context_lens, part, o, S, Hq, Hkv, D, block_size, max_blocks,
                                num_blocks, splits, scale, kv_fp8, k_scale, v_scale, 0, nullptr, 0, D, stream);
}

// The same over the newest `window` keys of every sequence (0: all of them), with an optional gate per head (logits
// gate[s * ldg + h]; the head's output is multiplied by its sigmoid) and only the first vdim of the D value columns
// written: o is [S, Hq, vdim].
int lt_paged_decode_window(const void* q, const void* k_cache, const void* v_cache, const int* block_tables,
                           const int* context_lens, float* part, void* o, int S, int Hq, int Hkv, int D, int block_size,
                           int max_blocks, int num_blocks, int splits, float scale, int kv_fp8, float k_scale, float v_scale,
                           int window, const void* gate, long long ldg, int vdim, void* stream) {
  using namespace lt;
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || splits < 1 || window < 0 || vdim < 1 || vdim > D) return -int(kStatusBadArgument);
  if (S == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int warps = S * Hq * splits;
  const int threads = 128;
  const int blocks = (warps * 32 + threads - 1) / threads;
  auto Q = static_cast<const __nv_bfloat16*>(q);
#define LT_PD(DD, F8) \
  paged_decode_kernel<DD, F8><<<blocks, threads, 0, st>>>(Q, k_cache, v_cache, block_tables, context_lens, part, S, Hq, Hkv, \
                                                          block_size, max_blocks, splits, scale, k_scale, v_scale, window)
  const int G = Hq / Hkv;
  const bool bs_ok = block_size > 0 && (32 % block_size == 0 || block_size % 32 == 0);
  // (the tensor-core kernels read two query values at a time, for 8-bit caches four)
  const bool aligned = (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 && (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0 &&
                       (reinterpret_cast<uintptr_t>(q) & (kv_fp8 ? 7 : 3)) == 0;
  if (G <= kPdMmaMaxG && bs_ok && block_size % 8 == 0 && num_blocks > 0 && aligned && (long long)num_blocks * Hkv * block_size < (1ll << 31)) {
    // caches in blocks of 8 keys or more: tiles by TMA, scores and P V on mma.sync
    const int ctas = S * Hkv * splits;
    const uint64_t rows = uint64_t(num_blocks) * Hkv * block_size;
    const uint32_t run = block_size < 32 ? block_size : 32;
    const int bytes = kv_fp8 ? 1 : 2;
    CUtensorMap tmK, tmV;
    int r = encode_tmap_2d(&tmK, k_cache, bytes, D, rows, uint64_t(D) * bytes, kv_fp8 ? D : 64, run, !kv_fp8 || D == 128);
    if (r == 0) r = encode_tmap_2d(&tmV, v_cache, bytes, D, rows, uint64_t(D) * bytes, kv_fp8 ? D : 64, run, !kv_fp8 || D == 128);
    if (r) return r > 0 ? 1000 + r : r;
    int* status = device_status_word();
    const int rc = launch_tensor_decode<false>(tmK, tmV, Q, block_tables, context_lens, part, S, Hq, Hkv, D, block_size, max_blocks, splits,
                                               kv_fp8 ? scale * k_scale : scale, kv_fp8, v_scale, window, status, PdStep{}, ctas, 1, st);
    if (rc) return rc;
  } else if (!kv_fp8 && window == 0 && G <= kPdMaxG && bs_ok && (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 && (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0) {
    // bf16 caches: every K / V byte is read once for the whole group of query heads, through a shared-memory pipeline
    const int ctas = S * Hkv * splits;
    auto KC = static_cast<const __nv_bfloat16*>(k_cache);
    auto VC = static_cast<const __nv_bfloat16*>(v_cache);
    static OncePerDevice configured;
    if (configured.pending()) {
      LT_RETURN_IF_CUDA(cudaFuncSetAttribute(paged_decode_gqa_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, PdCfg<64>::kSmemBytes));
      LT_RETURN_IF_CUDA(cudaFuncSetAttribute(paged_decode_gqa_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, PdCfg<128>::kSmemBytes));
      configured.finish();
    }
    int* status = device_status_word();
    if (D == 64) paged_decode_gqa_kernel<64><<<ctas, kPdWarps * 32, PdCfg<64>::kSmemBytes, st>>>(Q, KC, VC, block_tables, context_lens, part, S, Hq, Hkv, block_size, max_blocks, splits, scale, status);
    else paged_decode_gqa_kernel<128><<<ctas, kPdWarps * 32, PdCfg<128>::kSmemBytes, st>>>(Q, KC, VC, block_tables, context_lens, part, S, Hq, Hkv, block_size, max_blocks, splits, scale, status);
  } else if (D == 64) { if (kv_fp8) LT_PD(64, true); else LT_PD(64, false); }
  else { if (kv_fp8) LT_PD(128, true); else LT_PD(128, false); }
#undef LT_PD
  LT_LAUNCH_CHECK();
  return merge_splits(part, static_cast<__nv_bfloat16*>(o), S * Hq, splits, D, static_cast<const __nv_bfloat16*>(gate), ldg, Hq, vdim, st);
}

// One decode step's attention (see PdStep): qkv [S, ld] bf16 rows [q | k | v], the newest token of every sequence, which is the last of its context;
// o [S, Hq, D].  part: scratch [S, Hq, splits, D + 2] fp32, or nullptr: the splits, at most 16, are a cluster.  early: block tables, lengths and every cached row but the newest were complete before the kernels in
// front of this one that may still run.  Caches as in lt_paged_decode, in blocks of 8, 16 or a multiple of 32 keys.
int lt_paged_decode_step(const void* qkv, long long ld, const float* cos_t, const float* sin_t, const int* pos, const int* slots, void* k_cache, void* v_cache,
                         const int* block_tables, const int* context_lens, float* part, void* o, int S, int Hq, int Hkv, int D, int block_size,
                         int max_blocks, int num_blocks, int splits, float scale, int kv_fp8, float k_scale, float v_scale, int early, void* stream) {
  using namespace lt;
  if ((D != 64 && D != 128) || Hkv < 1 || Hq % Hkv != 0 || Hq / Hkv > kPdMmaMaxG || splits < 1 || (!part && splits > kPdMaxCluster) || (ld & 7) || num_blocks < 1 ||
      block_size < 8 || !(32 % block_size == 0 || block_size % 32 == 0) || (long long)num_blocks * Hkv * block_size >= (1ll << 31))
    return -int(kStatusBadArgument);
  for (const void* p : {qkv, static_cast<const void*>(cos_t), static_cast<const void*>(sin_t), static_cast<const void*>(k_cache), static_cast<const void*>(v_cache)})
    if (!p || (reinterpret_cast<uintptr_t>(p) & 15)) return -int(kStatusBadArgument);
  if (S == 0) return 0;
  const uint64_t rows = uint64_t(num_blocks) * Hkv * block_size;
  const uint32_t run = block_size < 32 ? block_size : 32;
  const int bytes = kv_fp8 ? 1 : 2;
  CUtensorMap tmK, tmV;
  int r = encode_tmap_2d(&tmK, k_cache, bytes, D, rows, uint64_t(D) * bytes, kv_fp8 ? D : 64, run, !kv_fp8 || D == 128);
  if (r == 0) r = encode_tmap_2d(&tmV, v_cache, bytes, D, rows, uint64_t(D) * bytes, kv_fp8 ? D : 64, run, !kv_fp8 || D == 128);
  if (r) return r > 0 ? 1000 + r : r;
  const PdStep step{static_cast<const __nv_bfloat16*>(qkv), ld, cos_t, sin_t, pos, slots, k_cache, v_cache, kv_fp8 ? 1.f / k_scale : 1.f, kv_fp8 ? 1.f / v_scale : 1.f,
                    static_cast<__nv_bfloat16*>(o), early};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = launch_tensor_decode<true>(tmK, tmV, nullptr, block_tables, context_lens, part, S, Hq, Hkv, D, block_size, max_blocks, splits,
                                            kv_fp8 ? scale * k_scale : scale, kv_fp8, v_scale, 0, device_status_word(), step, S * Hkv * splits, part ? 1 : splits, st);
  if (rc) return rc;
  return part ? merge_splits(part, static_cast<__nv_bfloat16*>(o), S * Hq, splits, D, nullptr, 0, Hq, D, st) : 0;
}

// How many clusters of `cluster` CTAs (1 .. 16) of the step's kernel for these heads the current GPU holds at once; negative: an error.
int lt_paged_decode_places(int Hq, int Hkv, int D, int kv_fp8, int cluster) {
  using namespace lt;
  if ((D != 64 && D != 128) || Hkv < 1 || Hq % Hkv != 0 || Hq / Hkv > kPdMmaMaxG || cluster < 1 || cluster > kPdMaxCluster) return -int(kStatusBadArgument);
#define LT_PLACES(DD, NT) \
  (kv_fp8 ? clusters_at_once(paged_decode_f8_kernel<DD, NT, true>, PdF8Cfg<DD>::kWarps, PdF8Cfg<DD>::kSmemBytes, cluster) \
          : clusters_at_once(paged_decode_mma_kernel<DD, NT, true>, PdMmaCfg<DD>::kWarps, PdMmaCfg<DD>::kSmemBytes, cluster))
  if (Hq / Hkv <= 8) return D == 64 ? LT_PLACES(64, 1) : LT_PLACES(128, 1);
  return D == 64 ? LT_PLACES(64, 2) : LT_PLACES(128, 2);
#undef LT_PLACES
}

int lt_kv_append(const void* k_new, const void* v_new, void* k_cache, void* v_cache, const int* slots, long long n_tok, int Hkv,
                 int D, int block_size, int kv_fp8, float k_scale, float v_scale, void* stream) {
  using namespace lt;
  if (n_tok == 0) return 0;
  const long long total = n_tok * Hkv * D;
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto KN = static_cast<const __nv_bfloat16*>(k_new);
  auto VN = static_cast<const __nv_bfloat16*>(v_new);
  if (kv_fp8) kv_append_kernel<true><<<(unsigned)blocks, 256, 0, st>>>(KN, VN, k_cache, v_cache, slots, n_tok, Hkv, D, block_size, 1.f / k_scale, 1.f / v_scale);
  else kv_append_kernel<false><<<(unsigned)blocks, 256, 0, st>>>(KN, VN, k_cache, v_cache, slots, n_tok, Hkv, D, block_size, 1.f, 1.f);
  LT_LAUNCH_CHECK();
  return 0;
}

}  // extern "C"
