// FlashAttention backward for sm_100a: causal or full, grouped-query heads, bf16, head_dim 64 or 128.
//
// The reference backward recomputes S and P with cuBLAS into B*H*Tq*Tk fp32 scratch and runs five batched
// GEMMs plus two kernels (src/backend/gpu_native/nn/flash_attention.cu:395-713); GQA is only handled on the
// CPU by expanding K/V per head (src/ops/attention.cpp:88-175).  Here one CTA owns a block of 128 keys of one
// KV head and keeps dK and dV for it in tensor memory while it walks over every query head of the group and
// every query block that can see those keys:
//
//   S  = Q_i K^T        dP = dO_i V^T                 (tcgen05.mma into TMEM, 128 x 128 x D)
//   P  = exp2(S*c - lse),  dS = P * (dP - delta) * scale   (one query row per thread, written to shared
//                                                           memory in the swizzled operand layout)
//   dV += P^T dO_i      dK += dS^T Q_i                (A read M-major from the same P / dS tiles)
//   dQ_i = dS K         -> red.global.add into an fp32 accumulator, converted to bf16 by a last kernel
//
// What bounds it: a serial chain.  S and dP, their exponentials (1024 clocks for 128 x 128 on one SM's special function units, about
// 2100 with the loads from tensor memory and the stores around them), and, with head_dim 128, dQ, which shares tensor memory with dP and
// shared memory with P and dS.  So what need not be on the chain is not: four warps of their own take dQ from tensor memory to the
// accumulator under the next block's products; Q is loaded a block ahead, and dV is the first product of a block, which frees dO for
// the next load and P for the first half of dQ; P and dS are made in registers before their tiles are waited for.
// Measured with the pre-pass and the conversion, causal, L2 flushed, against one set of warps doing both parts: D 128, 8192 tokens, 32 / 8
// heads 2191 -> 1711 us (7700 -> 6000 clocks a block; 40 MMAs take 2560); D 64, 4 x 2048 tokens, 32 / 4 heads 359 -> 325 us (3690 -> 3400).
//
// delta = rowsum(O * dO) comes from a small pre-pass.  All waits are bounded (see common/ptx.cuh).
#include "lt_cuda.h"
#include "common/host.h"
#include "common/ptx.cuh"

#include <type_traits>

namespace lt {

constexpr int kFbBlock = 128;
constexpr int kFbThreads = 512;   // warp 0 producer, warps 1 / 10 MMA issuers (S, dP / dQ, dV, dK), warps 2-9 compute, 12-15 write dQ
constexpr int kFbComputeThreads = 256;

constexpr int kFbMaxRanks = 8;
struct FlashBwdParams {
  // Per query-owning rank (index 0 only without context parallelism); peer-mapped pointers under CP:
  const float* lse[kFbMaxRanks];    // [B, Hq, Tq] natural log
  const float* delta[kFbMaxRanks];  // [B, Hq, Tq]
  float* dq_acc[kFbMaxRanks];       // [B, Tq, Hq, D] fp32, zero-initialised; remote ranks receive red.add over NVLink
  // Context parallelism: this rank's keys meet the queries of every rank; dK/dV stay local, dQ goes to its owner.
  int cp_world, cp_rank, zigzag;
  __nv_bfloat16* dK;
  __nv_bfloat16* dV;   // [B, Tk, Hkv, D] with strides sdk_b / sdk_t
  long long sdk_b, sdk_t;
  int B, Tq, Tk, Hq, Hkv;
  float scale, scale_log2;
  int causal;
  int* status;
  // Optional phase timing (nullptr: off): the CTA of key block 0 / head 0 / batch 0 adds the SM cycles its compute
  // warp 2 and its MMA thread spend in each phase to trace[0..15] and counts iterations in trace[15].
  long long* trace;
  // Tables of cosines and sines [., D / 2] by position: dK is turned back by the angles of its rows (nullptr: it is not).
  const float* cos_t;
  const float* sin_t;
};

struct QMaps {
  CUtensorMap q[kFbMaxRanks];
  CUtensorMap d_o[kFbMaxRanks];
};
struct QSeg {
  int n, owner, q0, qbase;   // a run of consecutive visible query blocks of one rank
};
constexpr int kFbMaxSegs = 2 * kFbMaxRanks;

template <int D>
struct FaBwdCfg {
  static constexpr int kTile = kFbBlock * D * 2;          // one 128 x D bf16 tile
  static constexpr int kPTile = kFbBlock * kFbBlock * 2;  // 128 x 128 bf16
  // Q is loaded a block ahead; dO too where there is room, else as soon as dV has been added (before dK and dQ).
  static constexpr int kQStages = 2, kDoStages = (D == 64) ? 2 : 1;
  static constexpr int kOffK = 0;
  static constexpr int kOffV = kTile;
  static constexpr int kOffQ = 2 * kTile;
  static constexpr int kOffDO = kOffQ + kQStages * kTile;
  static constexpr int kOffP = kOffDO + kDoStages * kTile;
  static constexpr int kOffDS = kOffP + kPTile;
  static constexpr int kOffBar = kOffDS + kPTile;
  static constexpr int kOffSeg = kOffBar + 192;
  // dQ tiles are staged in shared memory for TMA reductions into the fp32 accumulator: boxes of 32 rows x 32 columns (4 KB, 128-byte
  // swizzle), D / 32 to each of the four writing warps.  The copy engine does the atomics, not the LSU, and it is given few, large
  // operations.
  static constexpr int kDqTile = 32 * 128;                 // one 32-row x 32-column fp32 box
  static constexpr int kDqBoxes = D / 32;                  // boxes per warp: its 32 rows
  // head_dim 64: a staging area of its own.  head_dim 128: shared memory is full, so the staging area IS the P and dS
  // tiles (free between the MMAs of one iteration and the stores of the next): columns 0 .. 63 in the P tile, which is free first.
  static constexpr bool kStageAliasesP = (D != 64);
  static constexpr int kOffDqStage = kStageAliasesP ? kOffP : ((kOffSeg + kFbMaxSegs * 16 + 16 + 1023) / 1024) * 1024;
  static constexpr int kSmemBytes = (kStageAliasesP ? kOffSeg + kFbMaxSegs * 16 + 16 : kOffDqStage + 4 * kDqBoxes * kDqTile) + 1024;
  static_assert(kSmemBytes <= 232448, "does not fit");
  static constexpr int kColS = 0, kColDP = 128, kColDV = 256, kColDK = 256 + D;
  static constexpr int kColDQ = (D == 64) ? 384 : kColDP;  // D == 64: two buffers (384, 448); D == 128: over dP, which has been read by then
  static constexpr bool kTwoDq = (D == 64);
  static constexpr bool kDqOverDp = (D != 64);
};

// Four pairs (x, y) of neighbouring columns turned by the negative angles: (x c + y s, y c - x s).
__device__ __forceinline__ void turn_back(float (&v)[8], const float* cos_row, const float* sin_row) {
  const float4 c = *reinterpret_cast<const float4*>(cos_row), s = *reinterpret_cast<const float4*>(sin_row);
  const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = v[2 * j], y = v[2 * j + 1];
    v[2 * j] = x * cc[j] + y * ss[j];
    v[2 * j + 1] = y * cc[j] - x * ss[j];
  }
}

// delta[b,h,t] = sum_d O * dO ; D/8 threads per (b,t,h) row, 16 bytes each.  They also zero their columns of the dQ accumulator [B, Tq, Hq, D] (nullptr: the
// caller has).
__global__ void flash_bwd_delta_kernel(const __nv_bfloat16* O, const __nv_bfloat16* dO,
                                       float* __restrict__ delta, float* __restrict__ dq_acc, int B, int Tq, int Hq, int D, long long so_b,
                                       long long so_t, long long sdo_b, long long sdo_t) {
  pdl_launch_dependents();
  pdl_wait();
  const int tpr = D / 8;  // 8 or 16 threads per row
  const long long gid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long row = gid / tpr;
  const int sub = int(gid % tpr);
  const long long total = (long long)B * Tq * Hq;
  float s = 0.f;
  int h = 0, t = 0, b = 0;
  if (row < total) {
    const long long bt = row / Hq;
    h = int(row - bt * Hq);
    b = int(bt / Tq);
    t = int(bt - (long long)b * Tq);
    if (dq_acc) {
      float4* z = reinterpret_cast<float4*>(dq_acc + row * D + sub * 8);
      z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint4 a = *reinterpret_cast<const uint4*>(O + b * so_b + t * so_t + (long long)h * D + sub * 8);
    const uint4 g = *reinterpret_cast<const uint4*>(dO + b * sdo_b + t * sdo_t + (long long)h * D + sub * 8);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(av[i]), y = unpack_bf16x2(gv[i]);
      s += x.x * y.x + x.y * y.y;
    }
  }
  for (int off = tpr / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (row < total && sub == 0) delta[((long long)b * Hq + h) * Tq + t] = s;
}

// dQ leaves its accumulator as bf16, eight columns a thread; with tables [., D / 2] of cosines and sines (nullptr: as it is) turned back by the angles of
// its row's position t, pairs of neighbouring columns together.
__global__ void __launch_bounds__(256) flash_bwd_convert_dq_kernel(const float* acc, __nv_bfloat16* __restrict__ dq, long long rows, int Tq,
                                                                   int HD, int D, long long sdq_b, long long sdq_t, const float* __restrict__ cos_t,
                                                                   const float* __restrict__ sin_t) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_row = HD / 8;                          // threads of a block go through whole rows
  const int rows_at_once = max(1, 256 / per_row);
  const int r_in = threadIdx.x / per_row;
  if (r_in >= rows_at_once) return;
  for (long long r = (long long)blockIdx.x * rows_at_once + r_in; r < rows; r += (long long)gridDim.x * rows_at_once) {
    const long long b = r / Tq;
    const int t = int(r - b * Tq);
    for (int c = (threadIdx.x - r_in * per_row) * 8; c < HD; c += rows_at_once > 1 ? HD : 256 * 8) {
      const float4 lo = *reinterpret_cast<const float4*>(acc + r * HD + c), hi = *reinterpret_cast<const float4*>(acc + r * HD + c + 4);
      float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      if (cos_t) turn_back(v, cos_t + (long long)t * (D / 2) + (c % D) / 2, sin_t + (long long)t * (D / 2) + (c % D) / 2);
      const uint4 o = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
      __nv_bfloat16* to = dq + b * sdq_b + t * sdq_t + c;
      if (reinterpret_cast<uintptr_t>(to) & 15) {      // rows of dQ need 8-byte alignment only
        reinterpret_cast<uint2*>(to)[0] = make_uint2(o.x, o.y);
        reinterpret_cast<uint2*>(to)[1] = make_uint2(o.z, o.w);
      } else {
        *reinterpret_cast<uint4*>(to) = o;
      }
    }
  }
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Tiled TMA reduction shared -> global (fp32 add) of the box of `m` at coordinates (x, h, t, b).
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, uint32_t smem_src, int x, int h, int t, int b) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_src), "r"(x), "r"(h), "r"(t), "r"(b) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <int D>
__global__ void __launch_bounds__(kFbThreads, 1)
flash_bwd_kernel(const __grid_constant__ QMaps qm, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDQ, const FlashBwdParams p) {
  using Cfg = FaBwdCfg<D>;
  constexpr int QS = Cfg::kQStages, DS = Cfg::kDoStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  const uint32_t bb = smem_u32(bars);
  const uint32_t kv_full = bb;
  auto q_full = [&](int i) { return bb + 8u * (1 + i); };
  auto q_empty = [&](int i) { return bb + 8u * (3 + i); };
  auto do_full = [&](int i) { return bb + 8u * (5 + i); };
  auto do_empty = [&](int i) { return bb + 8u * (7 + i); };
  const uint32_t sdp_full = bb + 8u * 9;    // S and dP are in TMEM
  const uint32_t sdp_free = bb + 8u * 10;   // compute warps have read S and dP (one arrival per warp)
  const uint32_t pds_full = bb + 8u * 11;   // P and dS are in shared memory (one arrival per warp)
  const uint32_t ds_empty = bb + 8u * 12;   // the MMAs that read dS have executed
  auto dq_full = [&](int i) { return bb + 8u * (13 + i); };   // dQ is in TMEM (one barrier per dQ buffer, so a waiter can never be
  auto dq_free = [&](int i) { return bb + 8u * (15 + i); };   // overtaken by two completions); the writing warps have read it
  const uint32_t dkv_full = bb + 8u * 17;   // all MMAs done
  const uint32_t p_empty = bb + 8u * 18;    // the MMAs that read P have executed
  const uint32_t stg_p = bb + 8u * 19;      // dQ reductions have finished reading what they staged in the P tile
  const uint32_t stg_ds = bb + 8u * 20;     // ... and in the dS tile
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 21);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // x fastest in launch order: all (head, batch) pairs of key block 0 (seen by every query, the longest loop) first
  const int kv_blk = blockIdx.z, hkv = blockIdx.x, b = blockIdx.y;
  const int G = p.Hq / p.Hkv;
  const int kv0 = kv_blk * kFbBlock;
  QSeg* segs = reinterpret_cast<QSeg*>(smem + Cfg::kOffSeg);
  int* per_head_s = reinterpret_cast<int*>(smem + Cfg::kOffSeg + kFbMaxSegs * 16);
  // global position of this block's first key
  int k_base;
  if (p.cp_world == 1) {
    k_base = kv0 - (p.Tk - p.Tq);   // expressed on the query axis: query i sees key j iff j - (Tk - Tq) <= i
  } else if (p.zigzag) {
    const int hk = p.Tk / 2;
    k_base = kv0 < hk ? p.cp_rank * hk + kv0 : (2 * p.cp_world - 1 - p.cp_rank) * hk + (kv0 - hk);
  } else {
    k_base = p.cp_rank * p.Tk + kv0;
  }
  if (threadIdx.x == 0) {
    // query blocks that see these keys, as runs per owning rank (own rank first)
    int ns = 0, total = 0;
    for (int i = 0; i < p.cp_world; ++i) {
      const int o = (p.cp_rank + i) % p.cp_world;
      const int parts = (p.cp_world > 1 && p.zigzag) ? 2 : 1;
      for (int h2 = 0; h2 < parts; ++h2) {
        int q0s, qbase, nb;
        if (parts == 2) {
          const int hq = p.Tq / 2;
          q0s = h2 * hq;
          qbase = h2 == 0 ? o * hq : (2 * p.cp_world - 1 - o) * hq;
          nb = hq / kFbBlock;
        } else {
          q0s = 0;
          qbase = p.cp_world > 1 ? o * p.Tq : 0;
          nb = (p.Tq + kFbBlock - 1) / kFbBlock;
        }
        int skip = 0;
        if (p.causal) {
          const int first_q = k_base - qbase;   // first query position (relative to the run) that sees key k_base
          skip = first_q <= 0 ? 0 : first_q / kFbBlock;
        }
        if (nb > skip) {
          segs[ns] = QSeg{nb - skip, o, q0s + skip * kFbBlock, qbase + skip * kFbBlock};
          ++ns;
          total += nb - skip;
        }
      }
    }
    for (int i = ns; i < kFbMaxSegs; ++i) segs[i] = QSeg{0, 0, 0, 0};
    *per_head_s = total;
  }
  __syncthreads();
  const int per_head = *per_head_s;
  const int n_iter = per_head * G;
  const bool single = p.cp_world == 1;                    // a single run, kept in registers
  const int first_q0 = segs[0].q0, first_qbase = segs[0].qbase;
  auto locate = [&](int j, int& owner, int& q0, int& qbase) {
    if (single) {
      owner = 0;
      q0 = first_q0 + j * kFbBlock;
      qbase = first_qbase + j * kFbBlock;
      return;
    }
    int sidx = 0;
    while (sidx < kFbMaxSegs - 1 && j >= segs[sidx].n) { j -= segs[sidx].n; ++sidx; }
    owner = segs[sidx].owner;
    q0 = segs[sidx].q0 + j * kFbBlock;
    qbase = segs[sidx].qbase + j * kFbBlock;
  };

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full(i), 1); mbar_init(q_empty(i), 1);
      mbar_init(do_full(i), 1); mbar_init(do_empty(i), 1);
      mbar_init(dq_full(i), 1); mbar_init(dq_free(i), 4);
    }
    mbar_init(sdp_full, 1); mbar_init(sdp_free, kFbComputeThreads / 32);
    mbar_init(pds_full, kFbComputeThreads / 32); mbar_init(ds_empty, 1);
    mbar_init(p_empty, 1); mbar_init(stg_p, 4); mbar_init(stg_ds, 4);
    mbar_init(dkv_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&qm.q[p.cp_rank]); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&qm.d_o[p.cp_rank]);
    tma_prefetch_desc(&tmDQ);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (n_iter > 0 && elect_one()) {
      mbar_expect_tx(kv_full, 2 * Cfg::kTile);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        tma_load_4d(sbase + Cfg::kOffK + c * (kFbBlock * 128), &tmK, kv_full, c * 64, hkv, kv0, b);
        tma_load_4d(sbase + Cfg::kOffV + c * (kFbBlock * 128), &tmV, kv_full, c * 64, hkv, kv0, b);
      }
      for (int it = 0; it < n_iter; ++it) {
        const int qs = it % QS, ds = it % DS;
        const int h = hkv * G + it / per_head;
        int owner, q0, qbase;
        locate(it % per_head, owner, q0, qbase);
        if (!mbar_wait(q_empty(qs), (uint32_t(it / QS) & 1u) ^ 1u, abort_flag, p.status, kStatusTimeoutEmpty)) break;
        mbar_expect_tx(q_full(qs), Cfg::kTile);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(sbase + Cfg::kOffQ + qs * Cfg::kTile + c * (kFbBlock * 128), &qm.q[owner], q_full(qs), c * 64, h, q0, b);
        if (!mbar_wait(do_empty(ds), (uint32_t(it / DS) & 1u) ^ 1u, abort_flag, p.status, kStatusTimeoutEmpty)) break;
        mbar_expect_tx(do_full(ds), Cfg::kTile);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(sbase + Cfg::kOffDO + ds * Cfg::kTile + c * (kFbBlock * 128), &qm.d_o[owner], do_full(ds), c * 64, h, q0, b);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- first MMA issuer: S = Q K^T, dP = dO V^T
    // (as far ahead as the S / dP columns of tensor memory allow: they are free once the compute warps have loaded them)
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t idesc_sd = make_idesc_f16(128, 128, 1, 0, 0);  // S, dP: A K-major, B K-major
      bool ok = mbar_wait(kv_full, 0, abort_flag, p.status, kStatusTimeoutFull);
      // descriptors advance by 16-byte units: only their address field changes
      const uint64_t k_desc = make_smem_desc_sw128(sbase + Cfg::kOffK, 16, 1024), v_desc = make_smem_desc_sw128(sbase + Cfg::kOffV, 16, 1024);
      const uint64_t q_desc = make_smem_desc_sw128(sbase + Cfg::kOffQ, 16, 1024), do_desc = make_smem_desc_sw128(sbase + Cfg::kOffDO, 16, 1024);
      const bool tr = p.trace != nullptr && kv_blk == 0 && hkv == 0 && b == 0;
      long long tm[4] = {0, 0, 0, 0};
      for (int it = 0; ok && it < n_iter; ++it) {
        const int qs = it % QS, ds = it % DS;
        const uint32_t ipar = it & 1;
        const uint64_t qd = q_desc + uint64_t(qs * (Cfg::kTile >> 4)), dod = do_desc + uint64_t(ds * (Cfg::kTile >> 4));
        long long c0 = tr ? clock64() : 0;
        if (!mbar_wait(q_full(qs), uint32_t(it / QS) & 1u, abort_flag, p.status, kStatusTimeoutFull)) { ok = false; break; }
        if (tr) { const long long c1 = clock64(); tm[0] += c1 - c0; c0 = c1; }
        if (!mbar_wait(sdp_free, ipar ^ 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty)) { ok = false; break; }
        if (tr) { const long long c1 = clock64(); tm[1] += c1 - c0; c0 = c1; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = ((k / 4) * (128 * 128) + (k % 4) * 32) >> 4;
          umma_f16_ss(tmem_base + Cfg::kColS, qd + off, k_desc + off, idesc_sd, k > 0 ? 1u : 0u);
        }
        if (Cfg::kDqOverDp && !mbar_wait(dq_free(0), ipar ^ 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty)) { ok = false; break; }
        if (!mbar_wait(do_full(ds), uint32_t(it / DS) & 1u, abort_flag, p.status, kStatusTimeoutFull)) { ok = false; break; }
        if (tr) { const long long c1 = clock64(); tm[2] += c1 - c0; c0 = c1; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = ((k / 4) * (128 * 128) + (k % 4) * 32) >> 4;
          umma_f16_ss(tmem_base + Cfg::kColDP, dod + off, v_desc + off, idesc_sd, k > 0 ? 1u : 0u);
        }
        umma_commit(sdp_full);
      }
      if (tr) {
        // MMA thread: wait for Q, for S / dP (and dQ) to be read, for dO
        p.trace[8] = tm[0]; p.trace[9] = tm[1]; p.trace[10] = tm[2];
      }
    }
  } else if (warp == 10) {
    // ---------------------------------------------------------------- second MMA issuer: dV += P^T dO, dQ = dS K, dK += dS^T Q
    // dV frees dO and P, which the next block's loads and dQ's way out wait for; dQ is read and written out while the tensor core
    // works on dK, and the next dP needs its columns.
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t idesc_kv = make_idesc_f16(128, D, 1, 1, 1);    // A M-major, B N-major
      constexpr uint32_t idesc_dq = make_idesc_f16(128, D, 1, 0, 1);    // A K-major, B N-major
      const uint64_t dsq_desc = make_smem_desc_sw128(sbase + Cfg::kOffDS, 16, 1024), k_desc = make_smem_desc_sw128(sbase + Cfg::kOffK, 128 * 128, 1024);
      const uint64_t p_desc = make_smem_desc_sw128(sbase + Cfg::kOffP, 128 * 128, 1024), ds_desc = make_smem_desc_sw128(sbase + Cfg::kOffDS, 128 * 128, 1024);
      const uint64_t q_desc = make_smem_desc_sw128(sbase + Cfg::kOffQ, 128 * 128, 1024), do_desc = make_smem_desc_sw128(sbase + Cfg::kOffDO, 128 * 128, 1024);
      for (int it = 0; it < n_iter; ++it) {
        const int qs = it % QS, ds = it % DS;
        const uint32_t ipar = it & 1;
        const uint64_t qd = q_desc + uint64_t(qs * (Cfg::kTile >> 4)), dod = do_desc + uint64_t(ds * (Cfg::kTile >> 4));
        // P / dS ready implies Q / dO of this stage are in shared memory (S and dP were computed from them)
        if (!mbar_wait(pds_full, ipar, abort_flag, p.status, kStatusTimeoutTmemFull)) break;
        // two buffers: this one was last used by iteration it - 2; over dP: the scores of this iteration waited for it
        if (Cfg::kTwoDq && !mbar_wait(dq_free(it & 1), ((uint32_t(it) >> 1) & 1u) ^ 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kFbBlock / 16; ++k) {   // K dimension = the 128 query rows, 16 rows per instruction
          const uint64_t koff = k * (16 * 128) >> 4;
          umma_f16_ss(tmem_base + Cfg::kColDV, p_desc + koff, dod + koff, idesc_kv, (it > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(do_empty(ds));
        umma_commit(p_empty);
#pragma unroll
        for (int k = 0; k < kFbBlock / 16; ++k)   // K dimension = the 128 keys
          umma_f16_ss(tmem_base + Cfg::kColDQ + (Cfg::kTwoDq ? (it & 1) * D : 0), dsq_desc + uint64_t(((k / 4) * (128 * 128) + (k % 4) * 32) >> 4),
                      k_desc + uint64_t(k * (16 * 128) >> 4), idesc_dq, k > 0 ? 1u : 0u);
        umma_commit(dq_full(Cfg::kTwoDq ? it & 1 : 0));
#pragma unroll
        for (int k = 0; k < kFbBlock / 16; ++k) {
          const uint64_t koff = k * (16 * 128) >> 4;
          umma_f16_ss(tmem_base + Cfg::kColDK, ds_desc + koff, qd + koff, idesc_kv, (it > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(q_empty(qs));
        umma_commit(ds_empty);
        if (it == n_iter - 1) umma_commit(dkv_full);
      }
    }
  } else if (warp >= 12) {
    // ---------------------------------------------------------------- dQ: tensor memory -> shared memory -> added to the accumulator
    const int quarter = warp & 3;
    const uint32_t lane_base = uint32_t(quarter * 32) << 16;
    uint8_t* tile = smem + Cfg::kOffDqStage + quarter * (2 * Cfg::kDqTile);
    bool ok = true, pending = false;   // pending: a reduction that reads the staging area may be in flight
    int hh = 0, jj = 0;
    for (int it = 0; it < n_iter; ++it) {
      const int buf = Cfg::kTwoDq ? it & 1 : 0;
      const int h = hkv * G + hh;
      int owner, q0, qbase;
      locate(jj, owner, q0, qbase);
      if (++jj == per_head) { jj = 0; ++hh; }
      ok = __all_sync(0xffffffffu, mbar_wait(dq_full(buf), uint32_t(Cfg::kTwoDq ? it >> 1 : it) & 1u, abort_flag, p.status, kStatusTimeoutTmemFull));
      if (!ok) break;
      tc_fence_after();
      const bool local = owner == p.cp_rank;
      const int q_idx = q0 + quarter * 32 + lane;
      float* dq_row = (p.cp_world == 1 ? p.dq_acc[0] : p.dq_acc[owner]) + (((long long)b * p.Tq + q_idx) * p.Hq + h) * D;
#pragma unroll
      for (int half = 0; half < D / 64; ++half) {
        uint32_t dq[2][32];
        tmem_ld_32x32(tmem_base + lane_base + Cfg::kColDQ + buf * D + half * 64, dq[0]);
        tmem_ld_32x32(tmem_base + lane_base + Cfg::kColDQ + buf * D + half * 64 + 32, dq[1]);
        tmem_ld_wait();
        if (half == D / 64 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_free(buf));
        }
        if (local) {
          uint8_t* to = tile + half * Cfg::kPTile;
          if (Cfg::kStageAliasesP) {
            // the staging area is the P, then the dS tile: the MMAs of this iteration must be done with it
            ok = __all_sync(0xffffffffu, mbar_wait(half == 0 ? p_empty : ds_empty, uint32_t(it) & 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty));
            if (!ok) break;
          } else {
            if (pending && lane == 0) bulk_wait_read0();
            __syncwarp();
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int u = 0; u < 8; ++u)   // row `lane` of the box, 16-byte units swizzled like the tensor map expects
              *reinterpret_cast<uint4*>(to + x * Cfg::kDqTile + lane * 128 + ((u ^ (lane & 7)) * 16)) =
                  make_uint4(dq[x][u * 4], dq[x][u * 4 + 1], dq[x][u * 4 + 2], dq[x][u * 4 + 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
#pragma unroll
            for (int x = 0; x < 2; ++x)   // rows past Tq are clipped by the copy engine
              tma_reduce_add_4d(&tmDQ, smem_u32(to + x * Cfg::kDqTile), half * 64 + x * 32, h, q0 + quarter * 32, b);
            bulk_commit();
          }
          pending = true;
        } else if (q_idx < p.Tq) {
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int u = 0; u < 8; ++u)
              red_add_v4(dq_row + half * 64 + x * 32 + u * 4, __uint_as_float(dq[x][u * 4]), __uint_as_float(dq[x][u * 4 + 1]),
                         __uint_as_float(dq[x][u * 4 + 2]), __uint_as_float(dq[x][u * 4 + 3]));
        }
      }
      if (!ok) break;
      if (Cfg::kStageAliasesP && lane == 0) {
        bulk_wait_read1();
        mbar_arrive(stg_p);
        bulk_wait_read0();
        mbar_arrive(stg_ds);
      }
    }
    if (pending && lane == 0) bulk_wait_all0();   // shared memory must outlive the reductions that read it
  } else if (warp < 10) {
    // ---------------------------------------------------------------- compute warps
    // Two warps share each TMEM lane quarter (a warp may only touch lanes 32*(warp%4)..+31); they split the columns.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = uint32_t(quarter * 32) << 16;
    bool ok = true;
    const bool tr = p.trace != nullptr && kv_blk == 0 && hkv == 0 && b == 0 && warp == 2 && lane == 0;
    long long tc[6] = {0, 0, 0, 0, 0, 0};
    // Row statistics are fetched one iteration ahead (the global-load latency is off the chain); the position of an
    // iteration (query head, block within the head) is advanced with counters, not divisions.
    const long long stat0 = ((long long)b * p.Hq + hkv * G) * p.Tq;      // of this KV head's first query head
    const float* lse0 = p.lse[0] + stat0;
    const float* delta0 = p.delta[0] + stat0;
    auto fetch_stats = [&](int hh, int jj, float& lse_raw, float& dl) {
      lse_raw = 0.f; dl = 0.f;
      if (hh >= G) return;
      int owner, q0, qbase;
      locate(jj, owner, q0, qbase);
      const int q_idx = q0 + row;
      if (q_idx < p.Tq) {
        const int at = hh * p.Tq + q_idx;
        // (indexing the pointer arrays of the kernel parameters with a run-time rank makes the compiler copy them to
        // local memory: the single-rank case reads element 0 directly)
        lse_raw = single ? lse0[at] : p.lse[owner][stat0 + at];
        dl = single ? delta0[at] : p.delta[owner][stat0 + at];
      }
    };
    float lse_next, dlt_next;
    int hh_next = 0, jj_next = 0;   // position of the iteration whose statistics are in lse_next / dlt_next
    fetch_stats(n_iter > 0 ? 0 : G, 0, lse_next, dlt_next);
    for (int it = 0; it < n_iter; ++it) {
      long long c0 = tr ? clock64() : 0;
      const uint32_t ipar = it & 1;
      int owner, q0, qbase;
      locate(jj_next, owner, q0, qbase);
      const int q_idx = q0 + row;
      const bool q_valid = q_idx < p.Tq;
      const float lse2 = lse_next * 1.4426950408889634f, dlt = dlt_next;
      if (++jj_next == per_head) { jj_next = 0; ++hh_next; }
      fetch_stats(hh_next, jj_next, lse_next, dlt_next);
      // last visible key (index local to this rank's KV) for this query row
      const int limit = p.causal ? min(kv0 + (qbase + row - k_base), p.Tk - 1) : (p.Tk - 1);
      if (tr) { const long long c1 = clock64(); tc[0] += c1 - c0; c0 = c1; }   // lse / delta loads issued, index math
      ok = __all_sync(0xffffffffu, mbar_wait(sdp_full, ipar, abort_flag, p.status, kStatusTimeoutTmemFull));
      if (!ok) break;
      if (tr) { const long long c1 = clock64(); tc[1] += c1 - c0; c0 = c1; }   // waiting for S / dP
      tc_fence_after();
      const bool live = q_valid && lse2 != -INFINITY;
      const float dlt_s = dlt * p.scale;
      const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2), l2 = pack_f32x2(-lse2, -lse2);
      const uint64_t s2 = pack_f32x2(p.scale, p.scale), d2 = pack_f32x2(-dlt_s, -dlt_s);
      uint8_t* prow = smem + Cfg::kOffP + (row >> 3) * 1024 + (row & 7) * 128 + half * (128 * 128);
      uint8_t* dsrow = smem + Cfg::kOffDS + (row >> 3) * 1024 + (row & 7) * 128 + half * (128 * 128);
      uint32_t dw[32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[32], dp[32], pw[16];
        tmem_ld_32x32(tmem_base + lane_base + Cfg::kColS + (2 * half + c) * 32, sv);
        tmem_ld_32x32(tmem_base + lane_base + Cfg::kColDP + (2 * half + c) * 32, dp);
        tmem_ld_wait();
        if (c == 1) {   // S / dP are in registers: the next iteration's score products may overwrite them
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(sdp_free);
        }
        auto weights = [&](auto masked) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float e0, e1, g0, g1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), c2, l2), e0, e1);
            e0 = ex2_approx(e0);
            e1 = ex2_approx(e1);
            if constexpr (decltype(masked)::value) {
              const int kv_idx = kv0 + (2 * half + c) * 32 + 2 * i;
              e0 = live && kv_idx <= limit ? e0 : 0.f;
              e1 = live && kv_idx + 1 <= limit ? e1 : 0.f;
            }
            unpack_f32x2(mul_f32x2(pack_f32x2(e0, e1), fma_f32x2(pack_f32x2(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])), s2, d2)), g0, g1);
            pw[i] = pack_bf16x2(e0, e1);
            dw[c * 16 + i] = pack_bf16x2(g0, g1);
          }
        };
        // every column of the chunk is visible to every row of the warp: no per-element test
        if (__all_sync(0xffffffffu, live && kv0 + (2 * half + c) * 32 + 31 <= limit)) weights(std::false_type{});
        else weights(std::true_type{});
        if (c == 0) {
          if (tr) { const long long c1 = clock64(); tc[3] += c1 - c0; c0 = c1; }
          // The tiles are waited for only when there is something to store: they are free once the MMAs of the previous iteration have
          // executed and, where dQ is staged there, its reductions have finished reading.
          ok = __all_sync(0xffffffffu, mbar_wait(p_empty, ipar ^ 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty));
          if (ok && Cfg::kStageAliasesP && it > 0)
            ok = __all_sync(0xffffffffu, mbar_wait(stg_p, uint32_t(it - 1) & 1u, abort_flag, p.status, kStatusTimeoutLocalFlag));
          if (!ok) break;
          if (tr) { const long long c1 = clock64(); tc[2] += c1 - c0; c0 = c1; }   // waiting for the P tile
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(prow + ((c * 4 + u) ^ (row & 7)) * 16) = make_uint4(pw[u * 4], pw[u * 4 + 1], pw[u * 4 + 2], pw[u * 4 + 3]);
      }
      if (!ok) break;
      if (tr) { const long long c1 = clock64(); tc[3] += c1 - c0; c0 = c1; }
      ok = __all_sync(0xffffffffu, mbar_wait(ds_empty, ipar ^ 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty));
      if (ok && Cfg::kStageAliasesP && it > 0)
        ok = __all_sync(0xffffffffu, mbar_wait(stg_ds, uint32_t(it - 1) & 1u, abort_flag, p.status, kStatusTimeoutLocalFlag));
      if (!ok) break;
      if (tr) { const long long c1 = clock64(); tc[4] += c1 - c0; c0 = c1; }   // waiting for the dS tile
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(dsrow + (u ^ (row & 7)) * 16) = make_uint4(dw[u * 4], dw[u * 4 + 1], dw[u * 4 + 2], dw[u * 4 + 3]);
      // one arrival per warp: 256 same-address arrivals on a shared-memory barrier serialise
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      if (tr) { const long long c1 = clock64(); tc[3] += c1 - c0; c0 = c1; }   // exp / dS / stores to shared memory
    }
    if (tr) {
      for (int i = 0; i < 6; ++i) p.trace[i] = tc[i];
      p.trace[15] = n_iter;
    }
    // ---------------------------------------------------------------- dK / dV epilogue (row = key index)
    if (ok && n_iter > 0) ok = __all_sync(0xffffffffu, mbar_wait(dkv_full, 0, abort_flag, p.status, kStatusTimeoutTmemFull));
    if (ok) {
      if (n_iter > 0) tc_fence_after();
      const int kv_idx = kv0 + row;
      __nv_bfloat16* dk_row = p.dK + b * p.sdk_b + (long long)kv_idx * p.sdk_t + (long long)hkv * D;
      __nv_bfloat16* dv_row = p.dV + b * p.sdk_b + (long long)kv_idx * p.sdk_t + (long long)hkv * D;
#pragma unroll 1
      for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
        uint32_t a[32], g[32];
        if (n_iter > 0) {
          tmem_ld_32x32(tmem_base + lane_base + Cfg::kColDK + c * 32, a);
          tmem_ld_32x32(tmem_base + lane_base + Cfg::kColDV + c * 32, g);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) { a[i] = 0u; g[i] = 0u; }
        }
        if (kv_idx < p.Tk) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w, z;
            float k8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) k8[i] = __uint_as_float(a[u * 8 + i]);
            if (p.cos_t) {
              const long long at = (long long)kv_idx * (D / 2) + (c * 32 + u * 8) / 2;
              turn_back(k8, p.cos_t + at, p.sin_t + at);
            }
            w.x = pack_bf16x2(k8[0], k8[1]);
            w.y = pack_bf16x2(k8[2], k8[3]);
            w.z = pack_bf16x2(k8[4], k8[5]);
            w.w = pack_bf16x2(k8[6], k8[7]);
            z.x = pack_bf16x2(__uint_as_float(g[u * 8 + 0]), __uint_as_float(g[u * 8 + 1]));
            z.y = pack_bf16x2(__uint_as_float(g[u * 8 + 2]), __uint_as_float(g[u * 8 + 3]));
            z.z = pack_bf16x2(__uint_as_float(g[u * 8 + 4]), __uint_as_float(g[u * 8 + 5]));
            z.w = pack_bf16x2(__uint_as_float(g[u * 8 + 6]), __uint_as_float(g[u * 8 + 7]));
            *reinterpret_cast<uint4*>(dk_row + c * 32 + u * 8) = w;
            *reinterpret_cast<uint4*>(dv_row + c * 32 + u * 8) = z;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int spin = 0; spin < 2000; ++spin) __nanosleep(100);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
static int launch_flash_bwd(const QMaps& qm, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdq,
                            const FlashBwdParams& p, cudaStream_t st) {
  using Cfg = FaBwdCfg<D>;
  static OncePerDevice configured;
  auto kern = flash_bwd_kernel<D>;
  if (configured.pending()) {
    LT_RETURN_IF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    configured.finish();
  }
  dim3 grid(p.Hkv, p.B, (p.Tk + kFbBlock - 1) / kFbBlock);
  LT_RETURN_IF_CUDA(launch_chained(kern, grid, kFbThreads, Cfg::kSmemBytes, st, qm, tk, tv, tdq, p));
  LT_LAUNCH_CHECK();
  return 0;
}

static int bwd_delta(const void* o, const void* d_o, float* delta, float* dq_acc, int B, int Tq, int Hq, int D, long long so_b, long long so_t,
                     long long sdo_b, long long sdo_t, cudaStream_t st) {
  const long long rows = (long long)B * Tq * Hq;
  const int threads = 256;
  const long long blocks = (rows * (D / 8) + threads - 1) / threads;
  LT_RETURN_IF_CUDA(launch_chained(flash_bwd_delta_kernel, (unsigned)blocks, threads, 0, st, static_cast<const __nv_bfloat16*>(o),
                                                               static_cast<const __nv_bfloat16*>(d_o), delta, dq_acc, B, Tq, Hq, D, so_b,
                                                               so_t, sdo_b, sdo_t));
  LT_LAUNCH_CHECK();
  return 0;
}

static int bwd_convert(const float* dq_acc, void* dq, int B, int Tq, int Hq, int D, long long sdq_b, long long sdq_t,
                       cudaStream_t st, const float* cos_t = nullptr, const float* sin_t = nullptr) {
  const long long rows = (long long)B * Tq, at_once = 256 / (Hq * D / 8) > 1 ? 256 / (Hq * D / 8) : 1;
  long long blocks = (rows + at_once - 1) / at_once;
  const long long cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  LT_RETURN_IF_CUDA(launch_chained(flash_bwd_convert_dq_kernel, (unsigned)blocks, 256, 0, st, dq_acc, static_cast<__nv_bfloat16*>(dq), rows, Tq, Hq * D, D, sdq_b,
                                   sdq_t, cos_t, sin_t));
  return 0;
}

// Main kernel.  q/d_o/lse/delta/dq_acc are given per query-owning rank (cp_world entries; peer-mapped under CP).
static long long* g_bwd_trace = nullptr;

static int bwd_main(const void* const* q_ptrs, const void* k, const void* v, const void* const* do_ptrs,
                    const float* const* lse_ptrs, const float* const* delta_ptrs, float* const* dq_acc_ptrs, void* dk, void* dv,
                    int B, int Tq, int Tk, int Hq, int Hkv, int D, long long sq_b, long long sq_t, long long sk_b, long long sk_t,
                    long long sv_b, long long sv_t, long long sdo_b, long long sdo_t, long long sdk_b, long long sdk_t,
                    float scale, int causal, int cp_world, int cp_rank, int zigzag, cudaStream_t st, const float* cos_t = nullptr,
                    const float* sin_t = nullptr) {
  if (cp_world < 1 || cp_world > kFbMaxRanks) return -int(kStatusBadArgument);
  if (cp_world > 1 && zigzag && ((Tq / 2) % kFbBlock != 0 || (Tk / 2) % kFbBlock != 0)) return -int(kStatusBadArgument);
  if (cp_world > 1 && !zigzag && (Tq % kFbBlock != 0 || Tk % kFbBlock != 0)) return -int(kStatusBadArgument);
  QMaps qm;
  CUtensorMap tk, tv;
  int r;
  for (int i = 0; i < kFbMaxRanks; ++i) {
    const int src = i < cp_world ? i : 0;
    r = encode_tmap_4d(&qm.q[i], q_ptrs[src], 2, D, Hq, Tq, B, (uint64_t)D * 2, (uint64_t)sq_t * 2, (uint64_t)sq_b * 2, 64, 1,
                       kFbBlock, 1, 1);
    if (r) return 1000 + r;
    r = encode_tmap_4d(&qm.d_o[i], do_ptrs[src], 2, D, Hq, Tq, B, (uint64_t)D * 2, (uint64_t)sdo_t * 2, (uint64_t)sdo_b * 2, 64,
                       1, kFbBlock, 1, 1);
    if (r) return 4000 + r;
  }
  r = encode_tmap_4d(&tk, k, 2, D, Hkv, Tk, B, (uint64_t)D * 2, (uint64_t)sk_t * 2, (uint64_t)sk_b * 2, 64, 1, kFbBlock, 1, 1);
  if (r) return 2000 + r;
  r = encode_tmap_4d(&tv, v, 2, D, Hkv, Tk, B, (uint64_t)D * 2, (uint64_t)sv_t * 2, (uint64_t)sv_b * 2, 64, 1, kFbBlock, 1, 1);
  if (r) return 3000 + r;
  FlashBwdParams p{};
  for (int i = 0; i < cp_world; ++i) {
    p.lse[i] = lse_ptrs[i];
    p.delta[i] = delta_ptrs[i];
    p.dq_acc[i] = dq_acc_ptrs[i];
  }
  p.cp_world = cp_world; p.cp_rank = cp_rank; p.zigzag = zigzag;
  p.dK = static_cast<__nv_bfloat16*>(dk);
  p.dV = static_cast<__nv_bfloat16*>(dv);
  p.sdk_b = sdk_b; p.sdk_t = sdk_t;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.status = device_status_word();
  p.trace = g_bwd_trace;
  p.cos_t = cos_t; p.sin_t = sin_t;
  // fp32 dQ accumulator of this rank, [B, Tq, Hq, D]: boxes of 32 rows x 32 columns (128 bytes, swizzled)
  CUtensorMap tdq;
  r = encode_tmap_4d(&tdq, dq_acc_ptrs[cp_rank], 4, D, Hq, Tq, B, (uint64_t)D * 4, (uint64_t)Hq * D * 4,
                     (uint64_t)Tq * Hq * D * 4, 32, 1, 32, 1, 1);
  if (r) return 5000 + r;
  return (D == 64) ? launch_flash_bwd<64>(qm, tk, tv, tdq, p, st) : launch_flash_bwd<128>(qm, tk, tv, tdq, p, st);
}

}  // namespace lt

extern "C" {

// Debug aid: a device buffer of 16 int64 that the next backward launches fill with per-phase SM cycle counts of one
// CTA (see FlashBwdParams::trace); nullptr switches it off.
void lt_flash_bwd_set_trace(void* buf) { lt::g_bwd_trace = static_cast<long long*>(buf); }

// Shapes as lt_flash_fwd.  delta: scratch [B, Hq, Tq] fp32.  dq_acc: scratch [B, Tq, Hq, D] fp32.
// dk and dv share the strides sdk_b / sdk_t.  cos_t, sin_t (fp32 [>= Tq, D / 2], 16-byte aligned, Tq = Tk; or both nullptr): q and k are pairs of neighbouring
// columns turned by the angles of their rows 0, 1, ..; dq and dk are turned back by these.
int lt_flash_bwd_rope(const void* q, const void* k, const void* v, const void* o, const float* lse, const void* d_o, void* dq,
                      void* dk, void* dv, float* delta, float* dq_acc, int B, int Tq, int Tk, int Hq, int Hkv, int D,
                      long long sq_b, long long sq_t, long long sk_b, long long sk_t, long long sv_b, long long sv_t,
                      long long so_b, long long so_t, long long sdo_b, long long sdo_t, long long sdq_b, long long sdq_t,
                      long long sdk_b, long long sdk_t, float scale, int causal, const float* cos_t, const float* sin_t, void* stream) {
  using namespace lt;
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || !cos_t != !sin_t || (cos_t && Tq != Tk) ||
      ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15))
    return -int(kStatusBadArgument);
  if (B == 0 || Tq == 0 || Tk == 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = bwd_delta(o, d_o, delta, dq_acc, B, Tq, Hq, D, so_b, so_t, sdo_b, sdo_t, st);
  if (rc) return rc;
  const void* qs[1] = {q};
  const void* dos[1] = {d_o};
  const float* lses[1] = {lse};
  const float* deltas[1] = {delta};
  float* accs[1] = {dq_acc};
  rc = bwd_main(qs, k, v, dos, lses, deltas, accs, dk, dv, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t, sv_b, sv_t, sdo_b, sdo_t,
                sdk_b, sdk_t, scale, causal, 1, 0, 0, st, cos_t, sin_t);
  if (rc) return rc;
  return bwd_convert(dq_acc, dq, B, Tq, Hq, D, sdq_b, sdq_t, st, cos_t, sin_t);
}

// The same without angles.
int lt_flash_bwd(const void* q, const void* k, const void* v, const void* o, const float* lse, const void* d_o, void* dq,
                 void* dk, void* dv, float* delta, float* dq_acc, int B, int Tq, int Tk, int Hq, int Hkv, int D,
                 long long sq_b, long long sq_t, long long sk_b, long long sk_t, long long sv_b, long long sv_t,
                 long long so_b, long long so_t, long long sdo_b, long long sdo_t, long long sdq_b, long long sdq_t,
                 long long sdk_b, long long sdk_t, float scale, int causal, void* stream) {
  return lt_flash_bwd_rope(q, k, v, o, lse, d_o, dq, dk, dv, delta, dq_acc, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t, sv_b, sv_t, so_b, so_t, sdo_b,
                           sdo_t, sdq_b, sdq_t, sdk_b, sdk_t, scale, causal, nullptr, nullptr, stream);
}

// Context-parallel backward in three stream-ordered phases; the caller crosses a rank barrier between them.
//   phase 0: delta = rowsum(O * dO) of the local queries (into symmetric memory); the caller also zeroes dq_acc.
//   phase 1: main kernel - this rank's keys against every rank's queries: Q / dO tiles by TMA from peer memory, lse / delta
//            by peer loads, dK / dV accumulated locally, dQ added to the owner's fp32 accumulator with red.add over NVLink.
//   phase 2: dq = bf16(dq_acc) once every peer's phase 1 is complete.
int lt_flash_bwd_cp(int phase, const void* const* q_ptrs, const void* k, const void* v, const void* o, const void* const* do_ptrs,
                    const float* const* lse_ptrs, const float* const* delta_ptrs, float* const* dq_acc_ptrs, void* dq, void* dk,
                    void* dv, int B, int Tq, int Tk, int Hq, int Hkv, int D, long long sq_b, long long sq_t, long long sk_b,
                    long long sk_t, long long sv_b, long long sv_t, long long so_b, long long so_t, long long sdo_b,
                    long long sdo_t, long long sdq_b, long long sdq_t, long long sdk_b, long long sdk_t, float scale, int causal,
                    int cp_world, int cp_rank, int zigzag, void* stream) {
  using namespace lt;
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || cp_rank < 0 || cp_rank >= cp_world) return -int(kStatusBadArgument);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (phase == 0)
    return bwd_delta(o, do_ptrs[cp_rank], const_cast<float*>(delta_ptrs[cp_rank]), nullptr, B, Tq, Hq, D, so_b, so_t, sdo_b, sdo_t, st);
  if (phase == 1)
    return bwd_main(q_ptrs, k, v, do_ptrs, lse_ptrs, delta_ptrs, dq_acc_ptrs, dk, dv, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t,
                    sv_b, sv_t, sdo_b, sdo_t, sdk_b, sdk_t, scale, causal, cp_world, cp_rank, zigzag, st);
  return bwd_convert(dq_acc_ptrs[cp_rank], dq, B, Tq, Hq, D, sdq_b, sdq_t, st);
}

}  // extern "C"
