// FlashAttention forward for sm_100a: causal or full, grouped-query heads, bf16, head_dim 64 or 128.
//
// The reference's CUDA attention materialises S = Q K^T for all heads in fp32 (four B*H*Tq*Tk scratch
// buffers), runs a row-softmax kernel and a second batched GEMM, has no causal mask and ignores the number
// of KV heads (src/backend/gpu_native/nn/flash_attention.cu:188-299).  This kernel never leaves the chip:
//
//   warp 0    TMA producer: Q tile once, K and V blocks through one ring (128-byte swizzle, mbarrier tx)
//   warp 1    MMA issuer:   S_j = Q K_j^T  (tcgen05.mma, scores of block j + 1 issued before the softmax of block j is done)
//                           O  += P_j V_j  (A = P_j from tensor memory, B = V_j as an N-major operand)
//   warps 2-5 softmax:      one query row per thread (TMEM lane = row): tcgen05.ld of the whole row into registers, maximum,
//                           exponentials, P_j as bf16 back into tensor memory.
// The running maximum is updated lazily: O in TMEM is rescaled only when a row's maximum grew by more
// than 2^8, which keeps exp2 arguments bounded and makes the rescale (tcgen05.ld/st of O) rare.
//
// What bounds it: the exponentials, 16 a clock and SM (1024 clocks for 128 x 128 scores against 256 (D 64) or 512 (D 128) of MMA), and
// the softmax warps' waits around them.  So a CTA has a single query tile and half of an SM's tensor memory, shared memory and
// registers: two CTAs run side by side, one's exponentials under the other's loads, waits, start and end.  (Two tiles in one CTA, as
// two heads of a KV head, read K and V half as often but were slower or equal: 168 against 146 us for D 64, 4 x 2048 tokens, 32
// heads, and 56 against 33 us where their fewer CTAs end in an empty wave.)  Scores are read from tensor memory once, P never
// goes through shared memory, scale, sum and conversion work on pairs, and the body for blocks that every row sees whole
// holds no tests: with a test per score, most of the time went into branches and instruction fetches.
// Measured against the kernel before it (four softmax warps to either parity of key blocks, P through shared memory, one CTA an SM), causal,
// 32 heads, L2 flushed: D 64, 4 x 2048 tokens 363 -> 136 us; D 64, 4096 tokens 299 -> 122; D 128, 8192 tokens 1177 -> 474 to 478 (1150 TFLOP/s);
// D 128, 1337 queries on 5437 keys 301 -> 155.  (That kernel had itself been 210 us and 673 us in the first and the third of these before its
// bodies got a lower limit beside the upper one, for windows, and with it tests per score.)  With 128-key blocks a thread holds 128 scores: 168
// registers, 64 bytes spilled.  Left: 1.3 to 1.5 times the exponentials' time in the loop, and 3 to 5 us a CTA of
// start, masked blocks and end.
// Query / key size D and value size DV may differ.  SHARED: the last 64 columns of a key are the same for all heads (a rotated part beside the
// heads' own unrotated ones) and come from a tensor of their own, so that keys are never put together in memory.
// Output: O [B, Tq, Hq, D] bf16 and the natural-log LSE [B, Hq, Tq] fp32 for the backward pass.
#include "lt_cuda.h"
#include "common/host.h"
#include "common/ptx.cuh"

#include <type_traits>

namespace lt {

constexpr int kFaBlockQ = 128;
constexpr int kFaShardRows = 128;        // context-parallel shards are whole numbers of query tiles and key blocks
constexpr int kFaThreads = 192;          // warp 0 producer, warp 1 MMA issuer, warps 2-5 softmax
// Keys of a block: two score buffers of 64 columns leave room for 128 columns of O.  With O of 64 columns one buffer of 128 beside
// its weights fits, and larger blocks wait less often.
constexpr int fa_block_kv(int dv) { return dv == 64 ? 128 : 64; }

struct FlashFwdParams {
  __nv_bfloat16* O;
  float* lse;
  int B, Tq, Tk, Hq, Hkv;
  long long so_b, so_t;
  float scale_log2;  // softmax scale * log2(e)
  int causal;
  int* status;
  long long* trace;   // optional phase timing of one CTA (debug aid; nullptr = off), 16 int64
  // Context parallelism: the keys/values of cp_world ranks (Tk rows each, read through per-rank tensor maps that may
  // point at peer memory) are visited in one pass; queries and keys carry global positions (contiguous split, or
  // zigzag: rank r holds sequence chunks r and 2W-1-r of 2W).  cp_world == 1 is plain attention.
  int cp_world, cp_rank, zigzag;
  int window;   // causal only: a query sees its own position and the window - 1 before it; 0 = no limit
};

constexpr int kFaMaxRanks = 8;
struct KvMaps {
  CUtensorMap k[kFaMaxRanks];
  CUtensorMap v[kFaMaxRanks];
};

// A run of consecutive visible KV blocks of one rank.
struct KvSeg {
  int n, owner, kv0, kbase;
};
constexpr int kFaMaxSegs = 2 * kFaMaxRanks;

__device__ __forceinline__ float ex2_approx_f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// Shared memory: the query tile, then a ring that K and V blocks go through in turn.
template <int D, int DV, int BKV>
struct FaFwdCfg {
  static constexpr int kQBytes = kFaBlockQ * D * 2;
  static constexpr int kKBytes = BKV * D * 2;
  static constexpr int kVBytes = BKV * DV * 2;
  static constexpr int kSlotBytes = kKBytes > kVBytes ? kKBytes : kVBytes;
  static constexpr int kFit = (113 * 1024 - 2560 - kQBytes) / kSlotBytes;     // two CTAs share an SM
  static constexpr int kSlots = kFit < 4 ? kFit : 4;
  static constexpr int kOffRing = kQBytes;
  static constexpr int kOffBar = kOffRing + kSlots * kSlotBytes;
  static constexpr int kOffSeg = kOffBar + 160;                               // KvSeg table (16 entries) + block count
  static constexpr int kSmemBytes = kOffSeg + kFaMaxSegs * 16 + 16 + 1024;    // 1 KB for the 1024-byte alignment
  // 256 columns of tensor memory.  With 64-key blocks two score buffers fit beside O; the softmax weights P (two bf16 a column)
  // go over their own scores, which the threads have in registers by then, and the next scores into the other buffer.  With
  // 128-key blocks (head size 64) P has columns of its own, and the next scores are made as soon as these have been read.
  static constexpr bool kTwoS = 2 * BKV + DV <= 256;
  static constexpr int kColP = kTwoS ? 0 : BKV;      // from the score buffer's first column
  static constexpr int kColO = 256 - DV;
  static constexpr int kTmemCols = 256;
  static_assert(kSlots >= 2 && (kTwoS || BKV + BKV / 2 + DV <= 256), "does not fit");
};

template <int D, int DV, int BKV, bool SHARED>
__global__ void __launch_bounds__(kFaThreads, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ KvMaps maps, const FlashFwdParams p) {
  using Cfg = FaFwdCfg<D, DV, BKV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  const uint32_t bb = smem_u32(bars);
  const uint32_t q_full = bb;
  auto full = [&](int i) { return bb + 8u * (1 + i); };      // ring slots, up to four
  auto empty = [&](int i) { return bb + 8u * (5 + i); };
  // One barrier for blocks of either parity: with two score buffers the softmax and the MMA issuer may be a block ahead of each
  // other, and a phase bit tells only neighbouring phases of one barrier apart.
  auto s_full = [&](int j) { return bb + 8u * (9 + (j & 1)); };    // scores of block j are in tensor memory
  auto p_full = [&](int j) { return bb + 8u * (11 + (j & 1)); };   // its softmax weights are
  auto o_full = [&](int j) { return bb + 8u * (13 + (j & 1)); };   // its PV product has been added
  const uint32_t s_free = bb + 8u * 15;                            // scores have been read (only where P has columns of its own)
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Launch order is x fastest: every head and batch entry of the heaviest (latest) query block runs before any
  // lighter block, and neighbouring CTAs are the query heads that share one KV head (the K/V tiles stay in L2).
  const int q_blk = gridDim.z - 1 - blockIdx.z;
  const int h = blockIdx.x, b = blockIdx.y;
  const int hkv = h / (p.Hq / p.Hkv);
  const int q0 = q_blk * kFaBlockQ;
  KvSeg* segs = reinterpret_cast<KvSeg*>(smem + Cfg::kOffSeg);
  int* n_blocks_s = reinterpret_cast<int*>(smem + Cfg::kOffSeg + kFaMaxSegs * 16);
  // global position of this block's first query
  int q_base;
  if (p.cp_world == 1) {
    q_base = q0 + (p.Tk - p.Tq);  // key index visible to query i is <= i + (Tk - Tq)
  } else if (p.zigzag) {
    const int hq = p.Tq / 2;
    q_base = q0 < hq ? p.cp_rank * hq + q0 : (2 * p.cp_world - 1 - p.cp_rank) * hq + (q0 - hq);
  } else {
    q_base = p.cp_rank * p.Tq + q0;
  }
  if (threadIdx.x == 0) {
    // visible KV blocks as runs: own rank first (local memory), then the other ranks
    const int q_last = q_base + kFaBlockQ - 1;
    const int nb_all = (p.Tk + BKV - 1) / BKV;
    int ns = 0, total = 0;
    for (int i = 0; i < p.cp_world; ++i) {
      const int o = (p.cp_rank + i) % p.cp_world;
      const int parts = (p.cp_world > 1 && p.zigzag) ? 2 : 1;
      for (int h2 = 0; h2 < parts; ++h2) {
        int kv0, kbase, nb;
        if (parts == 2) {
          const int hk = p.Tk / 2;
          kv0 = h2 * hk;
          kbase = h2 == 0 ? o * hk : (2 * p.cp_world - 1 - o) * hk;
          nb = hk / BKV;
        } else {
          kv0 = 0;
          kbase = p.cp_world > 1 ? o * p.Tk : 0;
          nb = nb_all;
        }
        if (p.causal) {
          const int vis = q_last < kbase ? 0 : (q_last - kbase) / BKV + 1;
          nb = nb < vis ? nb : vis;
        }
        if (p.window > 0 && p.cp_world == 1) {
          // blocks that end before the first query's window are skipped
          const int first = max(0, q_base - p.window + 1) / BKV;
          kv0 += first * BKV;
          kbase += first * BKV;
          nb -= first;
        }
        if (nb > 0) {
          segs[ns] = KvSeg{nb, o, kv0, kbase};
          ++ns;
          total += nb;
        }
      }
    }
    for (int i = ns; i < kFaMaxSegs; ++i) segs[i] = KvSeg{0, 0, 0, 0};
    *n_blocks_s = total;
    mbar_init(q_full, 1);
    for (int j = 0; j < 2; ++j) {
      mbar_init(s_full(j), 1);
      mbar_init(p_full(j), 4);
      mbar_init(o_full(j), 1);
    }
    mbar_init(s_free, 4);
    for (int i = 0; i < Cfg::kSlots; ++i) { mbar_init(full(i), 1); mbar_init(empty(i), 1); }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&maps.k[p.cp_rank]); tma_prefetch_desc(&maps.v[p.cp_rank]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  pdl_launch_dependents();
  pdl_wait();
  const int n_blocks = *n_blocks_s;
  // block j of the schedule -> (owner rank, first local key row, global position of its first key)
  auto locate = [&](int j, int& owner, int& kv0, int& kbase) {
    int sidx = 0;
    if (p.cp_world > 1)
      while (sidx < kFaMaxSegs - 1 && j >= segs[sidx].n) { j -= segs[sidx].n; ++sidx; }
    owner = segs[sidx].owner;
    kv0 = segs[sidx].kv0 + j * BKV;
    kbase = segs[sidx].kbase + j * BKV;
  };
  // K and V blocks in the order in which they go through the ring: K0, K1, V0, K2, V1, ...
  auto k_seq = [](int j) { return j == 0 ? 0 : 2 * j - 1; };
  auto v_seq = [&](int j) { return j + 1 < n_blocks ? 2 * j + 2 : 2 * j + 1; };

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (n_blocks > 0 && elect_one()) {
      auto load = [&](int i, int j, bool is_k) -> bool {
        const int s = i % Cfg::kSlots;
        int owner, kv0, kbase;
        locate(j, owner, kv0, kbase);
        if (!mbar_wait(empty(s), (uint32_t(i / Cfg::kSlots) & 1u) ^ 1u, abort_flag, p.status, kStatusTimeoutEmpty)) return false;
        const uint32_t dst = sbase + Cfg::kOffRing + s * Cfg::kSlotBytes;
        mbar_expect_tx(full(s), is_k ? Cfg::kKBytes : Cfg::kVBytes);
        if (is_k) {
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            if (SHARED && c == D / 64 - 1)
              tma_load_4d(dst + c * (BKV * 128), &maps.k[1], full(s), 0, 0, kv0, b);
            else
              tma_load_4d(dst + c * (BKV * 128), &maps.k[owner], full(s), c * 64, hkv, kv0, b);
        } else {
#pragma unroll
          for (int c = 0; c < DV / 64; ++c) tma_load_4d(dst + c * (BKV * 128), &maps.v[owner], full(s), c * 64, hkv, kv0, b);
        }
        return true;
      };
      mbar_expect_tx(q_full, Cfg::kQBytes);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) tma_load_4d(sbase + c * (kFaBlockQ * 128), &tmQ, q_full, c * 64, h, q0, b);
      bool ok = load(0, 0, true);
      for (int j = 0; ok && j < n_blocks; ++j) {
        if (j + 1 < n_blocks) ok = load(k_seq(j + 1), j + 1, true);
        ok = ok && load(v_seq(j), j, false);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer: S = Q K^T, O += P V
    if (n_blocks > 0 && elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_f16(kFaBlockQ, BKV, 1, 0, 0);
      constexpr uint32_t idesc_o = make_idesc_f16(kFaBlockQ, DV, 1, 0, 1);
      auto wait_ring = [&](int i) {
        return mbar_wait(full(i % Cfg::kSlots), uint32_t(i / Cfg::kSlots) & 1u, abort_flag, p.status, kStatusTimeoutFull);
      };
      const uint64_t q_desc = make_smem_desc_sw128(sbase, 16, 1024);
      const uint64_t k_desc = make_smem_desc_sw128(sbase + Cfg::kOffRing, 16, 1024);
      const uint64_t v_desc = make_smem_desc_sw128(sbase + Cfg::kOffRing, BKV * 128, 1024);
      auto scores = [&](int j) {
        const int slot = k_seq(j) % Cfg::kSlots;
        const uint64_t kd = k_desc + uint64_t(slot * (Cfg::kSlotBytes >> 4));
        const uint32_t d = tmem_base + (Cfg::kTwoS ? (j & 1) * BKV : 0);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t q_off = uint64_t(((k / 4) * (kFaBlockQ * 128) + (k % 4) * 32) >> 4);   // 16-byte units
          const uint64_t k_off = uint64_t(((k / 4) * (BKV * 128) + (k % 4) * 32) >> 4);
          umma_f16_ss(d, q_desc + q_off, kd + k_off, idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full(j));
        umma_commit(empty(slot));
      };
      auto values = [&](int j) {
        const int slot = v_seq(j) % Cfg::kSlots;
        const uint64_t vd = v_desc + uint64_t(slot * (Cfg::kSlotBytes >> 4));
        const uint32_t a = tmem_base + (Cfg::kTwoS ? (j & 1) * BKV : 0) + Cfg::kColP;
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)
          umma_f16_ts(tmem_base + Cfg::kColO, a + k * 8, vd + uint64_t((k * (16 * 128)) >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(o_full(j));
        umma_commit(empty(slot));
      };
      bool ok = wait_ring(0) && mbar_wait(q_full, 0, abort_flag, p.status, kStatusTimeoutFull);
      if (ok) scores(0);
      for (int j = 0; ok && j < n_blocks; ++j) {
        if (j + 1 < n_blocks) {
          // Two buffers: the other one held the weights of block j - 1, whose product was issued before and so reads them first.
          ok = wait_ring(k_seq(j + 1)) &&
               (Cfg::kTwoS || mbar_wait(s_free, uint32_t(j) & 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty));
          if (!ok) break;
          tc_fence_after();
          scores(j + 1);
        }
        ok = wait_ring(v_seq(j)) && mbar_wait(p_full(j), uint32_t(j >> 1) & 1u, abort_flag, p.status, kStatusTimeoutTmemFull);
        if (!ok) break;
        tc_fence_after();
        values(j);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax + epilogue: one query row per thread
    const int quarter = warp & 3;          // TMEM lanes this warp may touch
    const int row = quarter * 32 + lane;
    const int q_idx = q0 + row;
    const uint32_t tm = tmem_base + (uint32_t(quarter * 32) << 16);
    const uint32_t o_mine = tm + Cfg::kColO;
    const float scale = p.scale_log2;
    float m_used = 0.f, l = 0.f;
    bool seen = false;   // this row has met a visible key (with a window, whole blocks may lie before it)
    bool ok = true;
    const bool tr = p.trace != nullptr && blockIdx.z == 0 && h == 0 && b == 0 && threadIdx.x == 64;
    long long waited = 0, t0 = tr ? clock64() : 0;
    for (int j = 0; j < n_blocks; ++j) {
      const long long c0 = tr ? clock64() : 0;
      ok = __all_sync(0xffffffffu, mbar_wait(s_full(j), uint32_t(j >> 1) & 1u, abort_flag, p.status, kStatusTimeoutTmemFull));
      if (!ok) break;
      if (tr) waited += clock64() - c0;
      tc_fence_after();
      const uint32_t s_mine = tm + (Cfg::kTwoS ? (j & 1) * BKV : 0);
      uint32_t r[BKV / 32][32];
#pragma unroll
      for (int c = 0; c < BKV / 32; ++c) tmem_ld_32x32(s_mine + c * 32, r[c]);
      int owner, kv0b, kbase;
      locate(j, owner, kv0b, kbase);
      // last visible column of this block for this row: causal position and end of the rank's keys
      int limit = p.Tk - 1 - kv0b;
      if (p.causal) limit = min(limit, q_base + row - kbase);
      const int lower = p.window > 0 ? q_base + row - kbase - p.window + 1 : 0;   // first visible column
      // columns of a 32-key chunk that this row sees; chunks that no row of the warp sees are skipped
      auto visible = [&](int c) {
        const int lo = max(lower - c * 32, 0), hi = min(limit - c * 32, 31);
        return hi < lo ? 0u : (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo);
      };
      const bool whole = __all_sync(0xffffffffu, limit >= BKV - 1 && lower <= 0);
      tmem_ld_wait();
      if constexpr (!Cfg::kTwoS) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
      }
      float mx;
      if (whole) {
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 8)
#pragma unroll
            for (int u = 0; u < 4; ++u) m4[u] = max3(m4[u], __uint_as_float(r[c][i + u]), __uint_as_float(r[c][i + u + 4]));
        mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      } else {
        mx = -INFINITY;
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c) {
          const uint32_t vis = visible(c);
          if (__any_sync(0xffffffffu, vis != 0u)) {
#pragma unroll
            for (int i = 0; i < 32; ++i) mx = fmaxf(mx, (vis >> i) & 1u ? __uint_as_float(r[c][i]) : -INFINITY);
          }
        }
      }
      const float m_blk = mx == -INFINITY ? -INFINITY : mx * scale;   // a row that sees nothing here, whatever the scale
      if (!seen) {
        // nothing accumulated for this row yet (its weights were zero): take the block's maximum as it is
        m_used = (m_blk == -INFINITY) ? 0.f : m_blk;
        seen = m_blk != -INFINITY;
      }
      if (j > 0) {
        const float m_new = fmaxf(m_used, m_blk);
        const bool need = m_new - m_used > 8.f;
        const bool any = __any_sync(0xffffffffu, need);
        if (!Cfg::kTwoS || any) {
          // the product of the block before has read its weights and is in O
          ok = __all_sync(0xffffffffu, mbar_wait(o_full(j - 1), uint32_t((j - 1) >> 1) & 1u, abort_flag, p.status, kStatusTimeoutTmemEmpty));
          if (!ok) break;
          tc_fence_after();
        }
        if (any) {
          const float alpha = need ? ex2_approx_f(m_used - m_new) : 1.f;
#pragma unroll 1
          for (int c = 0; c < DV / 16; ++c) {
            uint32_t o[16];
            tmem_ld_32x16(o_mine + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x16(o_mine + c * 16, o);
          }
          tmem_st_wait();
          l *= alpha;
          if (need) m_used = m_new;
        }
      }
      // exponentials two at a time, row sum, weights as bf16 into tensor memory
      const uint64_t scale2 = pack_f32x2(scale, scale), minus2 = pack_f32x2(-m_used, -m_used);
      uint64_t sum2[2] = {0ull, 0ull};
      auto weights = [&](auto masked) {
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c) {
          uint32_t w[16];
          const uint32_t vis = decltype(masked)::value ? visible(c) : ~0u;
          if (decltype(masked)::value && !__any_sync(0xffffffffu, vis != 0u)) {
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = 0u;
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float e0, e1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), scale2, minus2), e0, e1);
              e0 = ex2_approx_f(e0);
              e1 = ex2_approx_f(e1);
              if constexpr (decltype(masked)::value) {
                e0 = (vis >> (2 * i)) & 1u ? e0 : 0.f;
                e1 = (vis >> (2 * i + 1)) & 1u ? e1 : 0.f;
              }
              sum2[i & 1] = add_f32x2(sum2[i & 1], pack_f32x2(e0, e1));
              w[i] = pack_bf16x2(e0, e1);
            }
          }
          tmem_st_32x16(s_mine + Cfg::kColP + c * 16, w);
        }
      };
      // two bodies: a test inside would be a branch per pair of keys
      if (whole) weights(std::false_type{});
      else weights(std::true_type{});
      float s0, s1;
      unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
      l += s0 + s1;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(j));   // one arrival per warp
    }
    if (tr) {
      p.trace[0] = waited;              // waiting for scores
      p.trace[4] = clock64() - t0;      // the whole loop
      p.trace[15] = n_blocks;
    }
    if (ok && n_blocks > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(o_full(n_blocks - 1), uint32_t((n_blocks - 1) >> 1) & 1u, abort_flag, p.status, kStatusTimeoutTmemFull));
      tc_fence_after();
    }
    if (ok) {
      const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
      __nv_bfloat16* orow = p.O + (long long)b * p.so_b + (long long)q_idx * p.so_t + (long long)h * DV;
#pragma unroll 1
      for (int c = 0; c < DV / 32; ++c) {
        uint32_t o[32];
        if (n_blocks > 0) {
          tmem_ld_32x32(o_mine + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        if (q_idx < p.Tq) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[u * 8 + 0]) * inv_l, __uint_as_float(o[u * 8 + 1]) * inv_l);
            w.y = pack_bf16x2(__uint_as_float(o[u * 8 + 2]) * inv_l, __uint_as_float(o[u * 8 + 3]) * inv_l);
            w.z = pack_bf16x2(__uint_as_float(o[u * 8 + 4]) * inv_l, __uint_as_float(o[u * 8 + 5]) * inv_l);
            w.w = pack_bf16x2(__uint_as_float(o[u * 8 + 6]) * inv_l, __uint_as_float(o[u * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 32 + u * 8) = w;
          }
        }
      }
      if (q_idx < p.Tq)
        p.lse[((long long)b * p.Hq + h) * p.Tq + q_idx] = (l > 0.f) ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int spin = 0; spin < 2000; ++spin) __nanosleep(100);  // bounded grace period for copies in flight
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

static long long* g_fwd_trace = nullptr;

template <int D, int DV, int BKV, bool SHARED = false>
static int launch_flash_fwd(const CUtensorMap& tq, const KvMaps& maps, const FlashFwdParams& p, cudaStream_t st) {
  using Cfg = FaFwdCfg<D, DV, BKV>;
  static OncePerDevice configured;
  auto kern = flash_fwd_kernel<D, DV, BKV, SHARED>;
  if (configured.pending()) {
    LT_RETURN_IF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    configured.finish();
  }
  dim3 grid(p.Hq, p.B, (p.Tq + kFaBlockQ - 1) / kFaBlockQ);
  LT_RETURN_IF_CUDA(launch_chained(kern, grid, kFaThreads, Cfg::kSmemBytes, st, tq, maps, p));
  LT_LAUNCH_CHECK();
  return 0;
}

static int flash_fwd_common(const void* q, const void* const* k_ptrs, const void* const* v_ptrs, void* o, float* lse, int B,
                            int Tq, int Tk, int Hq, int Hkv, int D, long long sq_b, long long sq_t, long long sk_b,
                            long long sk_t, long long sv_b, long long sv_t, long long so_b, long long so_t, float scale,
                            int causal, int cp_world, int cp_rank, int zigzag, int window, void* stream) {
  if (window < 0 || (window > 0 && (!causal || cp_world != 1))) return -int(kStatusBadArgument);
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || cp_world < 1 || cp_world > kFaMaxRanks) return -int(kStatusBadArgument);
  if (cp_world > 1 && zigzag && ((Tq / 2) % kFaBlockQ != 0 || (Tk / 2) % kFaShardRows != 0)) return -int(kStatusBadArgument);
  if (cp_world > 1 && !zigzag && (Tq % kFaBlockQ != 0 || Tk % kFaShardRows != 0)) return -int(kStatusBadArgument);
  if (B == 0 || Tq == 0) return 0;
  CUtensorMap tq;
  KvMaps maps;
  int r = encode_tmap_4d(&tq, q, 2, D, Hq, Tq, B, (uint64_t)D * 2, (uint64_t)sq_t * 2, (uint64_t)sq_b * 2, 64, 1, kFaBlockQ, 1, 1);
  if (r) return 1000 + r;
  for (int i = 0; i < kFaMaxRanks; ++i) {
    const int src = i < cp_world ? i : 0;
    r = encode_tmap_4d(&maps.k[i], k_ptrs[src], 2, D, Hkv, Tk, B, (uint64_t)D * 2, (uint64_t)sk_t * 2, (uint64_t)sk_b * 2, 64, 1,
                       fa_block_kv(D), 1, 1);
    if (r) return 2000 + r;
    r = encode_tmap_4d(&maps.v[i], v_ptrs[src], 2, D, Hkv, Tk, B, (uint64_t)D * 2, (uint64_t)sv_t * 2, (uint64_t)sv_b * 2, 64, 1,
                       fa_block_kv(D), 1, 1);
    if (r) return 3000 + r;
  }
  FlashFwdParams p{};
  p.O = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv;
  p.so_b = so_b; p.so_t = so_t;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.cp_world = cp_world; p.cp_rank = cp_rank; p.zigzag = zigzag;
  p.window = window;
  p.status = device_status_word();
  p.trace = g_fwd_trace;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return D == 64 ? launch_flash_fwd<64, 64, 128>(tq, maps, p, st) : launch_flash_fwd<128, 128, 64>(tq, maps, p, st);
}

// One sequence whose keys are [the head's own columns | 64 columns shared by all heads].
static int flash_fwd_shared(const void* q, const void* k, const void* k_shared, const void* v, void* o, float* lse, int Tq, int Tk, int H,
                            int D, int DV, long long sq_t, long long sk_t, long long ss_t, long long sv_t, float scale, int window,
                            cudaStream_t st) {
  const bool wide = D == 192 && DV == 128, mid = D == 128 && (DV == 64 || DV == 128);
  if ((!wide && !mid) || H < 1 || Tk < Tq || window < 0) return -int(kStatusBadArgument);
  if (Tq == 0) return 0;
  const int block_kv = fa_block_kv(DV), dk = D - 64;
  // one batch entry: its stride is never used, but has to be a valid one
  auto map = [&](CUtensorMap* m, const void* base, int cols, int heads, int rows, long long pitch, int box_rows) {
    return encode_tmap_4d(m, base, 2, cols, heads, rows, 1, (uint64_t)cols * 2, (uint64_t)pitch * 2, (uint64_t)pitch * rows * 2, 64, 1,
                          box_rows, 1, 1);
  };
  CUtensorMap tq;
  KvMaps maps;
  int r = map(&tq, q, D, H, Tq, sq_t, kFaBlockQ);
  if (r) return 1000 + r;
  for (int i = 0; i < kFaMaxRanks; ++i) {
    r = i == 0 ? map(&maps.k[i], k, dk, H, Tk, sk_t, block_kv) : map(&maps.k[i], k_shared, 64, 1, Tk, ss_t, block_kv);
    if (r) return 2000 + r;
    r = map(&maps.v[i], v, DV, H, Tk, sv_t, block_kv);
    if (r) return 3000 + r;
  }
  FlashFwdParams p{};
  p.O = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.B = 1; p.Tq = Tq; p.Tk = Tk; p.Hq = H; p.Hkv = H;
  p.so_b = (long long)Tq * H * DV; p.so_t = (long long)H * DV;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = 1;
  p.cp_world = 1;
  p.window = window;
  p.status = device_status_word();
  if (wide) return launch_flash_fwd<192, 128, 64, true>(tq, maps, p, st);
  return DV == 64 ? launch_flash_fwd<128, 64, 128, true>(tq, maps, p, st) : launch_flash_fwd<128, 128, 64, true>(tq, maps, p, st);
}

}  // namespace lt

extern "C" {

// q: [B, Tq, Hq, D], k/v: [B, Tk, Hkv, D], o: [B, Tq, Hq, D]; strides in elements for the batch and time
// dimensions, heads are D apart, D contiguous.  lse: [B, Hq, Tq] fp32 (natural log).
// Debug aid: a device buffer of 16 int64 that the next forward launches fill with per-phase SM cycle counts of the
// CTA of the last query block of head 0 / batch 0 (warp 2, lane 0); nullptr switches it off.
void lt_flash_fwd_set_trace(void* buf) { lt::g_fwd_trace = static_cast<long long*>(buf); }

int lt_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Tq, int Tk, int Hq, int Hkv,
                 int D, long long sq_b, long long sq_t, long long sk_b, long long sk_t, long long sv_b, long long sv_t,
                 long long so_b, long long so_t, float scale, int causal, void* stream) {
  const void* ks[1] = {k};
  const void* vs[1] = {v};
  return lt::flash_fwd_common(q, ks, vs, o, lse, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t, sv_b, sv_t, so_b, so_t, scale,
                              causal, 1, 0, 0, 0, stream);
}

// Causal attention in which query i sees key j only when 0 <= i - j < window (positions counted as in lt_flash_fwd, the
// last query on the last key): key blocks outside every row's window are never loaded.
int lt_flash_fwd_window(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Tq, int Tk, int Hq, int Hkv,
                        int D, long long sq_b, long long sq_t, long long sk_b, long long sk_t, long long sv_b, long long sv_t,
                        long long so_b, long long so_t, float scale, int window, void* stream) {
  const void* ks[1] = {k};
  const void* vs[1] = {v};
  return lt::flash_fwd_common(q, ks, vs, o, lse, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t, sv_b, sv_t, so_b, so_t, scale,
                              1, 1, 0, 0, window, stream);
}

// Causal attention of one sequence with keys in two parts: q [Tq, H, D], k [Tk, H, D - 64], k_shared [Tk, 64] (the last 64 columns of
// every head's keys), v [Tk, H, DV], o [Tq, H, DV] packed; heads are packed, rows at the given pitches (multiples of 8 elements).
// The last query stands on the last key; window as above, 0: none.  (D, DV) is (128, 64), (128, 128) or (192, 128).
int lt_flash_fwd_shared(const void* q, const void* k, const void* k_shared, const void* v, void* o, float* lse, int Tq, int Tk, int H,
                        int D, int DV, long long sq_t, long long sk_t, long long ss_t, long long sv_t, float scale, int window,
                        void* stream) {
  return lt::flash_fwd_shared(q, k, k_shared, v, o, lse, Tq, Tk, H, D, DV, sq_t, sk_t, ss_t, sv_t, scale, window, static_cast<cudaStream_t>(stream));
}

// Context-parallel forward: k_ptrs[r] / v_ptrs[r] are rank r's KV shards [B, Tk, Hkv, D] (peer-mapped pointers, all with
// the same strides); the local queries attend to every rank's keys in one pass, the KV tiles of other ranks being
// read from peer memory by non-multicast TMA loads inside the kernel.
int lt_flash_fwd_cp(const void* q, const void* const* k_ptrs, const void* const* v_ptrs, void* o, float* lse, int B, int Tq,
                    int Tk, int Hq, int Hkv, int D, long long sq_b, long long sq_t, long long sk_b, long long sk_t,
                    long long sv_b, long long sv_t, long long so_b, long long so_t, float scale, int causal, int cp_world,
                    int cp_rank, int zigzag, void* stream) {
  return lt::flash_fwd_common(q, k_ptrs, v_ptrs, o, lse, B, Tq, Tk, Hq, Hkv, D, sq_b, sq_t, sk_b, sk_t, sv_b, sv_t, so_b, so_t,
                              scale, causal, cp_world, cp_rank, zigzag, 0, stream);
}

}  // extern "C"
