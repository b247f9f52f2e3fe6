// Flash attention backward on tcgen05 tensor cores (packed variable-length, causal or full, grouped-query, head_dim 128).
//
// Two kernels, both with every contraction on `tcgen05.mma`, every accumulator in tensor memory, and P and dS as the A operand from
// tensor memory:
//
//   dK/dV kernel   CTA = 128 keys of one (sequence, kv head).  K_j and V_j stay in shared memory; the CTA walks the query
//                  heads of the group and their 128-row query blocks (Q_i, dO_i through a 2-stage TMA ring):
//                      Sᵀ  = K_j · Q_iᵀ      dPᵀ = V_j · dO_iᵀ            (128 columns each)
//                      Pᵀ  = exp2(Sᵀ·scale·log2e − lse_i·log2e)          dSᵀ = Pᵀ ∘ (dPᵀ − Δ_i) · scale
//                      dV += Pᵀ · dO_i        dK += dSᵀ · Q_i             (128 columns each, live for the whole CTA)
//                  The transposed products put the KEY on the TMEM lane: a softmax thread writes the bf16 of its Pᵀ (dSᵀ) columns
//                  over the Sᵀ (dPᵀ) columns it read.  dO_i and Q_i are read a second time through an MN-major descriptor.
//   dQ kernel      persistent, item = 128 queries of one (sequence, query head); K_j, V_j blocks of 128 keys through a ring:
//                      S = Q_i · K_jᵀ   dP = dO_i · V_jᵀ   dS = P ∘ (dP − Δ) · scale   dQ += dS · K_j
//
// Warp roles in both: warps 0..7 softmax / dS: thread = TMEM lane, two warps per lane quadrant with 64 of a block's 128 columns each;
// warp 8 TMA producer, warp 9 MMA issue + TMEM owner.
//
// What bounds them: 128 × 128 blocks of 2048 (dK/dV) and 1536 (dQ) tensor clocks against 1024 clocks of the special-function unit for
// P and about as many issue slots for dS.  The products are issued so that the tensor pipe always has two of them while the softmax warps
// work: dK/dV  dV_i, S_{i+1} | dK_i, dP_{i+1};  dQ  S_{i+1} | dQ_i, dP_{i+1}.  MMAs of one thread execute in issue order, so S_{i+1}
// may overwrite P_i behind dV_i without a wait.
// Measured: 8 × 4096 causal, 32 / 4 heads: 4164 µs, 660 TFLOP/s of the counted products (64-row blocks, P and dS through shared memory:
// 432 TFLOP/s); 24 × 1536: 486 TFLOP/s.
// S and dP are recomputed in both kernels (7 tile products per (i, j) pair instead of 5): the price of not accumulating dQ with
// atomics; results are deterministic.  Every barrier wait is bounded.
#include "attention_items.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);

namespace fab {

static constexpr int D = 128, B = 128;              // head dim; rows of a query or key block
static constexpr int kTile = B * D * 2;             // 32 KB: two 64-column atoms of 128 rows × 128 B
static constexpr int kAtom = B * 128;               // 16 KB
static constexpr int kThreads = 320;
static constexpr float kLog2e = 1.4426950408889634f;
static constexpr uint32_t kTmemCols = 512;

struct Params {
  const float* lse;     // [Hq, T]
  const float* delta;   // [Hq, T]
  __nv_bfloat16* dq;    // [T, Hq, 128]
  __nv_bfloat16* dk;    // [T, Hkv, 128]
  __nv_bfloat16* dv;
  const int* cu_seqlens;
  int Hq, Hkv, total_tokens;
  float scale;
  int causal;
  int* error_flag;
};

// TMEM accumulator row (32·chunks fp32 columns) → bf16 in global memory
__device__ __forceinline__ void store_acc_cols(uint32_t taddr, __nv_bfloat16* dst, bool valid, int chunks) {
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    uint32_t o[32];
    tmem_ld_32x32(taddr + c * 32, o);
    tmem_ld_wait();
    if (valid) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 w;
        w.x = pack_bf16x2(__uint_as_float(o[i]), __uint_as_float(o[i + 1]));
        w.y = pack_bf16x2(__uint_as_float(o[i + 2]), __uint_as_float(o[i + 3]));
        w.z = pack_bf16x2(__uint_as_float(o[i + 4]), __uint_as_float(o[i + 5]));
        w.w = pack_bf16x2(__uint_as_float(o[i + 6]), __uint_as_float(o[i + 7]));
        *reinterpret_cast<uint4*>(dst + c * 32 + i) = w;
      }
    }
  }
}

__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* full, int head, int row) {
  tma_load_2d(dst, tm, full, head * D, row);
  tma_load_2d(dst + kAtom, tm, full, head * D + 64, row);
}

// D[128 × 128] (+)= A · Bᵀ, both K-major tiles in shared memory (the contraction runs over the head dim)
__device__ __forceinline__ void mma_scores(uint32_t d, uint32_t a_addr, uint32_t b_addr) {
  constexpr uint32_t idesc = make_idesc_bf16(B, B, 0, 0);
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks)
    umma_bf16(d, make_smem_desc_sw128(a_addr + (ks >> 2) * kAtom + (ks & 3) * 32, 16, 1024),
              make_smem_desc_sw128(b_addr + (ks >> 2) * kAtom + (ks & 3) * 32, 16, 1024), idesc, ks != 0);
}
// D[128 × 128 d] (+)= A · tile with A (bf16) in tensor memory, the columns of rows 0..63 of the tile at a, those of rows 64..127 at a + 64
// (each half where its warps read the fp32 values); `steps` of 16 rows
__device__ __forceinline__ void mma_grad(uint32_t d, uint32_t a, uint32_t tile_addr, int steps, bool add) {
  constexpr uint32_t idesc = make_idesc_bf16(B, D, 0, 1);
  for (int ks = 0; ks < steps; ++ks)
    umma_bf16_ts(d, a + (ks >> 2) * 64 + (ks & 3) * 8, make_smem_desc_sw128(tile_addr + ks * (16 * 128), kAtom, 1024), idesc, add || ks != 0);
}

// =================================================================================================================
// dK / dV
// =================================================================================================================
namespace kv {

struct Smem {
  static constexpr int k = 0;
  static constexpr int v = k + kTile;
  static constexpr int q = v + kTile;               // 2 stages
  static constexpr int dout = q + 2 * kTile;        // 2 stages
  static constexpr int stats = dout + 2 * kTile;    // 2 stages × 8 warps × (64 lse + 64 delta) floats: a private copy per warp
  static constexpr int bars = stats + 2 * 8 * 128 * 4;
  static constexpr int total = bars + 256;
};

// grid (Hkv · batch, key blocks): the first key blocks, whose causal range is the longest, start first
__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_dkdv_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                         const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(p.error_flag, 0, 35);
    return;
  }
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x / p.Hkv, hk = blockIdx.x % p.Hkv;
  const int seq_start = p.cu_seqlens[b], L = p.cu_seqlens[b + 1] - seq_start;
  const int kv0 = blockIdx.y * B;
  if (kv0 >= L) return;
  const int G = p.Hq / p.Hkv;
  const int i_lo = p.causal ? static_cast<int>(blockIdx.y) : 0;
  const int n_i = (L + B - 1) / B - i_lo;
  const int n_it = n_i * G;

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::bars);
  uint64_t* kv_full = bars;             // 1
  uint64_t* q_full = bars + 1;          // 2
  uint64_t* q_empty = bars + 3;         // 2
  uint64_t* s_full = bars + 5;          // 1
  uint64_t* dp_full = bars + 6;         // 1
  uint64_t* p_ready = bars + 7;         // 1
  uint64_t* ds_ready = bars + 8;        // 1
  uint64_t* done = bars + 9;            // 1
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_ptr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  const uint32_t tmem_s = tmem, tmem_dp = tmem + 128, tmem_dk = tmem + 256, tmem_dv = tmem + 384;

  if (warp == 8) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * kTile);
      load_tile(smem + Smem::k, &tm_k, kv_full, hk, seq_start + kv0);
      load_tile(smem + Smem::v, &tm_v, kv_full, hk, seq_start + kv0);
      for (int it = 0; it < n_it && !*abort_flag; ++it) {
        const int st = it & 1;
        const int h = hk * G + it / n_i, row = seq_start + (i_lo + it % n_i) * B;
        if (!mbar_wait(&q_empty[st], ((it >> 1) & 1) ^ 1)) { *abort_flag = 1; atomicCAS(p.error_flag, 0, 31); break; }
        mbar_expect_tx(&q_full[st], 2 * kTile);
        load_tile(smem + Smem::q + st * kTile, &tm_q, &q_full[st], h, row);
        load_tile(smem + Smem::dout + st * kTile, &tm_do, &q_full[st], h, row);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      const uint32_t k_addr = smem_u32(smem + Smem::k), v_addr = smem_u32(smem + Smem::v);
      const uint32_t q_base = smem_u32(smem + Smem::q), d_base = smem_u32(smem + Smem::dout);
      auto issue_s = [&](int it) -> bool {
        if (!mbar_wait(&q_full[it & 1], (it >> 1) & 1)) return false;
        tc_fence_after();
        mma_scores(tmem_s, k_addr, q_base + (it & 1) * kTile);
        umma_commit(s_full);
        return true;
      };
      auto issue_dp = [&](int it) {
        mma_scores(tmem_dp, v_addr, d_base + (it & 1) * kTile);
        umma_commit(dp_full);
      };
      bool ok = mbar_wait(kv_full, 0) && issue_s(0);
      if (ok) issue_dp(0);
      for (int it = 0; it < n_it && ok && !*abort_flag; ++it) {
        const int st = it & 1;
        const int steps = min(B / 16, (L - (i_lo + it % n_i) * B + 15) / 16);      // query rows behind the sequence have weight 0
        if (!mbar_wait(p_ready, it & 1)) { ok = false; break; }
        tc_fence_after();
        mma_grad(tmem_dv, tmem_s, d_base + st * kTile, steps, it != 0);            // dV += Pᵀ · dO
        if (it + 1 < n_it && !issue_s(it + 1)) { ok = false; break; }
        if (!mbar_wait(ds_ready, it & 1)) { ok = false; break; }
        tc_fence_after();
        mma_grad(tmem_dk, tmem_dp, q_base + st * kTile, steps, it != 0);           // dK += dSᵀ · Q
        umma_commit(&q_empty[st]);
        if (it + 1 < n_it) issue_dp(it + 1);
      }
      if (ok) umma_commit(done);
      else { *abort_flag = 1; atomicCAS(p.error_flag, 0, 32); }
    }
  } else {
    const int q4 = warp & 3;
    const int ch = warp >> 2;                     // which 64 of the block's 128 queries this warp handles
    const int row = q4 * 32 + lane;               // key row within the block = TMEM lane
    const int kpos = kv0 + row;
    const uint32_t at = (static_cast<uint32_t>(q4 * 32) << 16) + ch * 64;
    const float sl2 = p.scale * kLog2e;
    bool ok = true;
    // this lane's queries of the step (lane and lane + 32): lse (× −log2e) and delta (× −scale), fetched one step ahead
    float nl[2], nd[2];
    auto fetch = [&](int it) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int qpos = (i_lo + it % n_i) * B + ch * 64 + i * 32 + lane;
        nl[i] = nd[i] = 0.f;
        if (it < n_it && qpos < L) {
          const long long w = static_cast<long long>(hk * G + it / n_i) * p.total_tokens + seq_start + qpos;
          nl[i] = -p.lse[w] * kLog2e;
          nd[i] = -p.delta[w] * p.scale;
        }
      }
    };
    fetch(0);
    const float2 sl2x2 = make_float2(sl2, sl2), scx2 = make_float2(p.scale, p.scale);
    for (int it = 0; it < n_it; ++it) {
      const int qbase = (i_lo + it % n_i) * B + ch * 64;
      // every warp keeps its own copy of its 64 lse / delta values, so the softmax warps never meet at a CTA barrier (a
      // barrier has no time limit; the mbarrier waits below do)
      float* stats = reinterpret_cast<float*>(smem + Smem::stats) + ((it & 1) * 8 + warp) * 128;
      stats[lane] = nl[0];
      stats[32 + lane] = nl[1];
      stats[64 + lane] = nd[0];
      stats[96 + lane] = nd[1];
      __syncwarp();
      fetch(it + 1);
      if (__any_sync(0xffffffffu, !mbar_wait(s_full, it & 1) || *abort_flag)) { ok = false; break; }
      tc_fence_after();
      const bool need_mask = (qbase + 64 > L) || (kv0 + B > L) || (p.causal && kv0 + B - 1 > qbase);
      // queries [lo, hi) of this warp's 64 count for this key
      const int lo = p.causal ? kpos - qbase : 0, hi = kpos < L ? L - qbase : 0;
      uint32_t s[2][32];
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld_32x32(tmem_s + at + c * 32, s[c]);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(stats + c * 32 + i);
          float2 a = fma_f32x2(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), sl2x2, make_float2(l4.x, l4.y));
          float2 d = fma_f32x2(make_float2(__uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3])), sl2x2, make_float2(l4.z, l4.w));
          a.x = exp2f(a.x); a.y = exp2f(a.y); d.x = exp2f(d.x); d.y = exp2f(d.y);
          if (need_mask) {
            const int j = c * 32 + i;
            if (j < lo || j >= hi) a.x = 0.f;
            if (j + 1 < lo || j + 1 >= hi) a.y = 0.f;
            if (j + 2 < lo || j + 2 >= hi) d.x = 0.f;
            if (j + 3 < lo || j + 3 >= hi) d.y = 0.f;
          }
          s[c][i] = __float_as_uint(a.x); s[c][i + 1] = __float_as_uint(a.y);
          s[c][i + 2] = __float_as_uint(d.x); s[c][i + 3] = __float_as_uint(d.y);
          packed[i / 2] = pack_bf16x2(a.x, a.y);
          packed[i / 2 + 1] = pack_bf16x2(d.x, d.y);
        }
        tmem_st_32x16(tmem_s + at + c * 16, packed);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if (__any_sync(0xffffffffu, !mbar_wait(dp_full, it & 1) || *abort_flag)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dp[32], packed[16];
        tmem_ld_32x32(tmem_dp + at + c * 32, dp);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 d4 = *reinterpret_cast<const float4*>(stats + 64 + c * 32 + i);
          float2 a = fma_f32x2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), scx2, make_float2(d4.x, d4.y));
          float2 d = fma_f32x2(make_float2(__uint_as_float(dp[i + 2]), __uint_as_float(dp[i + 3])), scx2, make_float2(d4.z, d4.w));
          a = mul_f32x2(a, make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])));
          d = mul_f32x2(d, make_float2(__uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3])));
          if (need_mask) {                        // a query of the next sequence may hold no number: 0 · that is none either
            const int j = c * 32 + i;
            if (j < lo || j >= hi) a.x = 0.f;
            if (j + 1 < lo || j + 1 >= hi) a.y = 0.f;
            if (j + 2 < lo || j + 2 >= hi) d.x = 0.f;
            if (j + 3 < lo || j + 3 >= hi) d.y = 0.f;
          }
          packed[i / 2] = pack_bf16x2(a.x, a.y);
          packed[i / 2 + 1] = pack_bf16x2(d.x, d.y);
        }
        tmem_st_32x16(tmem_dp + at + c * 16, packed);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
    }
    if (!ok || __any_sync(0xffffffffu, !mbar_wait(done, 0))) {
      *abort_flag = 1;
      atomicCAS(p.error_flag, 0, 33);
    } else {
      tc_fence_after();
      const bool valid = kpos < L;
      const long long off = (static_cast<long long>(seq_start + kpos) * p.Hkv + hk) * D;
      const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
      if (ch == 0) store_acc_cols(tmem_dk + lane_off, p.dk + off, valid, 4);     // the two warps of a quadrant share the write-back
      else store_acc_cols(tmem_dv + lane_off, p.dv + off, valid, 4);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace kv

// =================================================================================================================
// dQ
// =================================================================================================================
namespace qq {

static constexpr int kSlots = 4;                    // ring of K and V blocks, alternating

struct Smem {
  static constexpr int q = 0;
  static constexpr int dout = q + kTile;
  static constexpr int kv = dout + kTile;
  static constexpr int bars = kv + kSlots * kTile;
  static constexpr int total = bars + 256;
};

__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, Params p, ItemList list) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(p.error_flag, 0, 45);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::bars);
  uint64_t* q_full = bars;              // 1
  uint64_t* q_empty = bars + 1;         // 1
  uint64_t* kv_full = bars + 2;         // 4
  uint64_t* kv_empty = bars + 6;        // 4
  uint64_t* s_full = bars + 10;         // 2
  uint64_t* s_empty = bars + 12;        // 2
  uint64_t* dp_full = bars + 14;        // 1
  uint64_t* ds_ready = bars + 15;       // 1
  uint64_t* dq_full = bars + 16;        // 1
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 8);
    }
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, 8);
    mbar_init(dq_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_ptr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  const uint32_t tmem_dp = tmem + 256, tmem_dq = tmem + 384;      // S in columns 0 and 128, alternating
  pdl_trigger();
  pdl_wait();

  Items items;
  items.init(list);
  int b, h;
  if (warp == 8) {
    const bool leader = elect_one();
    uint32_t c = 0, qc = 0;
    while (!__any_sync(0xffffffffu, *abort_flag) && items.next(list, b, h)) {
      const int seq_start = p.cu_seqlens[b], L = p.cu_seqlens[b + 1] - seq_start, q0 = items.level * B, hk = h / (p.Hq / p.Hkv);
      const int n = ((p.causal ? min(L, q0 + B) : L) + B - 1) / B;
      if (leader) {
        bool ok = mbar_wait(q_empty, (qc & 1) ^ 1);
        ++qc;
        if (ok) {
          mbar_expect_tx(q_full, 2 * kTile);
          load_tile(smem + Smem::q, &tm_q, q_full, h, seq_start + q0);
          load_tile(smem + Smem::dout, &tm_do, q_full, h, seq_start + q0);
        }
        for (int i = 0; i < 2 * n && ok && !*abort_flag; ++i, ++c) {
          const uint32_t slot = c % kSlots;
          ok = mbar_wait(&kv_empty[slot], ((c / kSlots) & 1) ^ 1);
          if (!ok) break;
          mbar_expect_tx(&kv_full[slot], kTile);
          load_tile(smem + Smem::kv + slot * kTile, (i & 1) ? &tm_v : &tm_k, &kv_full[slot], hk, seq_start + (i >> 1) * B);
        }
        if (!ok) { *abort_flag = 1; atomicCAS(p.error_flag, 0, 41); }
      }
      __syncwarp();
    }
  } else if (warp == 9) {
    const bool leader = elect_one();
    const uint32_t q_addr = smem_u32(smem + Smem::q), d_addr = smem_u32(smem + Smem::dout), kv_addr = smem_u32(smem + Smem::kv);
    uint32_t c = 0, qc = 0, sc = 0, dc = 0;          // ring entries of earlier items; items; blocks of S issued; blocks of dS consumed
    while (!__any_sync(0xffffffffu, *abort_flag) && items.next(list, b, h)) {
      const int L = p.cu_seqlens[b + 1] - p.cu_seqlens[b], q0 = items.level * B;
      const int kv_end = p.causal ? min(L, q0 + B) : L, n = (kv_end + B - 1) / B;
      if (leader) {
        auto issue_s = [&](int j) -> bool {          // K of block j in ring entry c + 2j, V in c + 2j + 1
          const uint32_t e = c + 2 * j, slot = e % kSlots, buf = sc & 1;
          if (!mbar_wait(&kv_full[slot], (e / kSlots) & 1) || !mbar_wait(&s_empty[buf], ((sc >> 1) & 1) ^ 1)) return false;
          tc_fence_after();
          mma_scores(tmem + buf * 128, q_addr, kv_addr + slot * kTile);
          umma_commit(&s_full[buf]);
          ++sc;
          return true;
        };
        auto issue_dp = [&](int j) -> bool {
          const uint32_t e = c + 2 * j + 1, slot = e % kSlots;
          if (!mbar_wait(&kv_full[slot], (e / kSlots) & 1)) return false;
          tc_fence_after();
          mma_scores(tmem_dp, d_addr, kv_addr + slot * kTile);
          umma_commit(dp_full);
          umma_commit(&kv_empty[slot]);
          if (j + 1 == n) umma_commit(q_empty);      // the last use of Q and dO
          return true;
        };
        bool ok = mbar_wait(q_full, qc & 1) && issue_s(0) && issue_dp(0);
        ++qc;
        for (int j = 0; j < n && ok && !*abort_flag; ++j) {
          if (j + 1 < n) ok = issue_s(j + 1);
          if (!ok || !mbar_wait(ds_ready, dc & 1)) { ok = false; break; }
          ++dc;
          tc_fence_after();
          const uint32_t slot = (c + 2 * j) % kSlots;
          mma_grad(tmem_dq, tmem_dp, kv_addr + slot * kTile, min(B / 16, (kv_end - j * B + 15) / 16), j != 0);
          umma_commit(&kv_empty[slot]);
          if (j + 1 < n) ok = issue_dp(j + 1);
        }
        if (ok) umma_commit(dq_full);
        else { *abort_flag = 1; atomicCAS(p.error_flag, 0, 42); }
      }
      c += 2 * n;
      __syncwarp();
    }
  } else {
    const int q4 = warp & 3;
    const int ch = warp >> 2;                        // which 64 of a block's 128 keys this warp handles
    const int row = q4 * 32 + lane;                  // query row within the tile = TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16, at = lane_off + ch * 64;
    const float sl2 = p.scale * kLog2e;
    const float2 sl2x2 = make_float2(sl2, sl2), scx2 = make_float2(p.scale, p.scale);
    uint32_t sc = 0, dc = 0, ic = 0;
    bool ok = true;
    while (items.next(list, b, h)) {
      const int seq_start = p.cu_seqlens[b], L = p.cu_seqlens[b + 1] - seq_start, q0 = items.level * B, qpos = q0 + row;
      const int n = ((p.causal ? min(L, q0 + B) : L) + B - 1) / B;
      const int all = p.causal ? min(L, q0 + 1) : L;               // keys before this one count for every row
      const int end = p.causal ? min(L, qpos + 1) : L;             // keys that count for this row
      float l2 = 0.f, dl = 0.f;
      if (qpos < L) {
        const long long w = static_cast<long long>(h) * p.total_tokens + seq_start + qpos;
        l2 = -p.lse[w] * kLog2e;
        dl = -p.delta[w] * p.scale;
      }
      const float2 l2x2 = make_float2(l2, l2), dlx2 = make_float2(dl, dl);
      for (int j = 0; j < n; ++j) {
        const uint32_t buf = sc & 1;
        if (__any_sync(0xffffffffu, !mbar_wait(&s_full[buf], (sc >> 1) & 1) || *abort_flag)) { ok = false; break; }
        ++sc;
        tc_fence_after();
        uint32_t s[2][32];
#pragma unroll
        for (int k = 0; k < 2; ++k) tmem_ld_32x32(tmem + buf * 128 + at + k * 32, s[k]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_empty[buf]);
        const bool need_mask = (j + 1) * B > all;
        const int hi = end - j * B - ch * 64;                      // keys [0, hi) of this warp's 64 count
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float2 a = fma_f32x2(make_float2(__uint_as_float(s[k][i]), __uint_as_float(s[k][i + 1])), sl2x2, l2x2);
            s[k][i] = __float_as_uint(exp2f(a.x));
            s[k][i + 1] = __float_as_uint(exp2f(a.y));
          }
        if (__any_sync(0xffffffffu, !mbar_wait(dp_full, dc & 1) || *abort_flag)) { ok = false; break; }
        ++dc;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t dp[32], packed[16];
          tmem_ld_32x32(tmem_dp + at + k * 32, dp);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float2 a = fma_f32x2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), scx2, dlx2);
            a = mul_f32x2(a, make_float2(__uint_as_float(s[k][i]), __uint_as_float(s[k][i + 1])));
            if (need_mask) {
              if (k * 32 + i >= hi) a.x = 0.f;
              if (k * 32 + i + 1 >= hi) a.y = 0.f;
            }
            packed[i / 2] = pack_bf16x2(a.x, a.y);
          }
          tmem_st_32x16(tmem_dp + at + k * 16, packed);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_ready);
      }
      if (!ok || __any_sync(0xffffffffu, !mbar_wait(dq_full, ic & 1) || *abort_flag)) { ok = false; break; }
      ++ic;
      tc_fence_after();
      // the two warps of a quadrant share the write-back; the next item's first dS·K waits for both of them
      store_acc_cols(tmem_dq + lane_off + ch * 64, p.dq + (static_cast<long long>(seq_start + qpos) * p.Hq + h) * D + ch * 64, qpos < L, 2);
      tc_fence_before();
    }
    if (!ok) {
      *abort_flag = 1;
      atomicCAS(p.error_flag, 0, 43);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace qq
}  // namespace fab
}  // namespace mb

using namespace mb;

// q, dout [T, Hq, 128], k, v [T, Hkv, 128] (token strides q/k/v_stride elements, dout contiguous); lse, delta [Hq, T];
// dq [T, Hq, 128], dk, dv [T, Hkv, 128] contiguous bf16.
extern "C" int mb_flash_bwd_tc(const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta,
                               void* dq, void* dk, void* dv, const int* cu_seqlens, int batch, int max_seqlen, int total_tokens,
                               long long q_stride, long long k_stride, long long v_stride, int Hq, int Hkv, float scale, int causal,
                               int* error_flag, cudaStream_t s) {
  if (batch == 0 || total_tokens == 0 || max_seqlen == 0) return 0;
  if (Hq % Hkv) return -1;
  const int blocks = (max_seqlen + fab::B - 1) / fab::B;
  if (blocks > 65535) return -2;
  const long long qc = static_cast<long long>(Hq) * fab::D, kc = static_cast<long long>(Hkv) * fab::D;
  CUtensorMap tq, td, tk, tv;
  int rc = 0;
  if ((rc = make_tmap_bf16_2d(&tq, q, total_tokens, qc, q_stride, fab::B, 64))) return 1000 + rc;
  if ((rc = make_tmap_bf16_2d(&td, dout, total_tokens, qc, qc, fab::B, 64))) return 2000 + rc;
  if ((rc = make_tmap_bf16_2d(&tk, k, total_tokens, kc, k_stride, fab::B, 64))) return 3000 + rc;
  if ((rc = make_tmap_bf16_2d(&tv, v, total_tokens, kc, v_stride, fab::B, 64))) return 4000 + rc;
  static const cudaError_t configured = [] {
    const cudaError_t e = cudaFuncSetAttribute(fab::kv::flash_bwd_dkdv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fab::kv::Smem::total);
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(fab::qq::flash_bwd_dq_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fab::qq::Smem::total);
  }();
  if (configured != cudaSuccess) return static_cast<int>(configured);
  const fab::Params p{lse, delta, reinterpret_cast<__nv_bfloat16*>(dq), reinterpret_cast<__nv_bfloat16*>(dk),
                      reinterpret_cast<__nv_bfloat16*>(dv), cu_seqlens, Hq, Hkv, total_tokens, scale, causal, error_flag};
  cudaError_t e = launch_pdl(fab::kv::flash_bwd_dkdv_tc_kernel, dim3(Hkv * batch, blocks), dim3(fab::kThreads), fab::kv::Smem::total, s, tq, td, tk, tv, p);
  if (e != cudaSuccess) return static_cast<int>(e);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const ItemList list{cu_seqlens, batch, Hq, blocks, fab::B};
  const long long most = static_cast<long long>(blocks) * batch * Hq;
  e = launch_pdl(fab::qq::flash_bwd_dq_tc_kernel, dim3(static_cast<unsigned>(most < sms ? most : sms)), dim3(fab::kThreads), fab::qq::Smem::total, s, tq, td,
                 tk, tv, p, list);
  return static_cast<int>(e);
}
