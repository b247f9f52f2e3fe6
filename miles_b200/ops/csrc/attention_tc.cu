// Flash attention forward on tcgen05 tensor cores (packed variable-length, causal, grouped-query, head_dim 128).
//
// Persistent, one CTA per SM.  A work item is TWO query tiles of 128 rows that share their keys: two heads of one KV head at the same
// 128 queries (an even number of query heads per KV head), else two neighbouring tiles of one head.  Warp roles:
//   warps 0..3, 4..7   softmax of tile 0 and of tile 1: thread = query row (TMEM lane).  Read S from tensor memory, online maximum and
//                      sum in registers, write P (bf16) over S, rescale O in tensor memory when the running maximum moved, store O
//   warp 8             TMA: the two Q tiles, then K and V blocks of 128 keys through one ring of five 32 KB slots
//   warp 9             MMA issue + TMEM owner: S_t = Q_t·Kᵀ (operands in shared memory), O_t += P_t·V (P in tensor memory)
//   warps 10, 11       idle (register redistribution works on groups of four warps)
// TMEM: S0 | S1 | O0 | O1, 128 columns each; P_t takes the first 64 columns of S_t.
//
// What bounds it.  A 128×128 block costs 1024 tensor clocks (S and P·V) and 1024 clocks of the special-function unit (16 384 exp2 at
// 16 per clock), so the two have to overlap: while one tile's softmax runs, the tensor pipe works on the other tile.  The products are
// issued O0 += P0·V, S0 (next block), O1 += P1·V, S1 (next block): MMAs of one thread execute in issue order, so S_t may overwrite P_t
// without a wait, and "S_t is complete" says that O_t holds every earlier block.  P·V starts on the first 64 keys while the other 64 are
// still being exponentiated.  Two CTAs per SM with 64-key blocks and P through shared memory (the earlier form) took
// 2.56 ms (430 TFLOP/s) at 8 × 4096 causal tokens with 32 query and 4 KV heads and 1.26 ms (367) at 24 × 1536; this one takes 1.01 ms
// (1086) and 0.53 ms (883), and 0.57 ms (1143) at one sequence of 8190 and one of 3601 with 8 KV heads.  Short sequences pay for the
// half-masked diagonal blocks and the first block's latency: 450 TFLOP/s at 32 × 512.
//
// Schedule: attention_items.cuh.
// Q, K, V are read with 2-D tensor maps over [tokens, heads·128]; rows of a tile that belong to the next sequence are masked as keys and
// never stored as queries.  All barrier waits are bounded (error flag + early exit).
#include "attention_items.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);

namespace fa {

static constexpr int BQ = 128, BKV = 128, D = 128;
static constexpr int kTileBytes = 128 * D * 2;            // 32 KB: two 64-column atoms of 128 rows × 128 B (Q, K and V alike)
static constexpr int kAtom = 128 * 128;                   // 16 KB
static constexpr int kSlots = 5;                          // K/V ring
static constexpr int kThreads = 384;                      // launched with 168 registers; 2 × 208 + 88 per lane of a sub-partition afterwards
static constexpr uint32_t kTmemCols = 512;
static constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  __nv_bfloat16* o;
  float* lse;
  const int* cu_seqlens;
  const int* cu_seqlens_k;     // null: keys are the queries' own sequences.  Else sequence b has keys [cu_k[b], cu_k[b+1]) and, under
                               // the causal mask, query i sees keys ≤ i + (Lk − Lq): the queries are the LAST Lq positions of the keys
                               // (a prompt continued after a cached prefix, a later chunk of a long prompt)
  int Hq, Hkv, total_tokens;
  int pair_heads;              // the two tiles of an item: heads 2i, 2i + 1 (1) or query tiles 2i, 2i + 1 (0)
  ItemList list;               // levels of 128 or 256 queries, Hq / 2 or Hq items per sequence and level
  float scale;
  int causal;
  int* error_flag;
};

struct Smem {
  static constexpr int q = 0;                             // two tiles
  static constexpr int kv = q + 2 * kTileBytes;
  static constexpr int bars = kv + kSlots * kTileBytes;
  static constexpr int total = bars + 256;   // the dynamic segment is declared 1024-byte aligned; checked at run time
};

// One item: where its two tiles are and how many key blocks each of them takes.
struct Item {
  int seq_start, k_start, L, Lk, off, hk;
  int q0[2], h[2], n[2], kv_end[2];
  __device__ __forceinline__ Item(const Params& p, int level, int b, int sub) {
    seq_start = p.cu_seqlens[b];
    L = p.cu_seqlens[b + 1] - seq_start;
    k_start = p.cu_seqlens_k != nullptr ? p.cu_seqlens_k[b] : seq_start;
    Lk = p.cu_seqlens_k != nullptr ? p.cu_seqlens_k[b + 1] - k_start : L;
    off = Lk - L;                                        // causal diagonal shift (0 when keys and queries coincide)
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      q0[t] = p.pair_heads ? level * BQ : (2 * level + t) * BQ;
      h[t] = p.pair_heads ? 2 * sub + t : sub;
      kv_end[t] = q0[t] >= L ? 0 : (p.causal ? max(0, min(Lk, q0[t] + BQ + off)) : Lk);   // no keys: the tile is left alone
      n[t] = (kv_end[t] + BKV - 1) / BKV;
    }
    hk = h[0] / (p.Hq / p.Hkv);
  }
};

// exp2(s·scale − m) of 32 scores → P (bf16 pairs) in tensor memory; the sum is taken before rounding
__device__ __forceinline__ void exp_chunk(const uint32_t (&s)[32], float2 scale, float2 minus_m, float2 (&sum)[2], uint32_t p_addr) {
  uint32_t packed[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float2 v = fma_f32x2(make_float2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), scale, minus_m);
    v.x = exp2f(v.x);
    v.y = exp2f(v.y);
    sum[i & 1] = add_f32x2(sum[i & 1], v);
    packed[i] = pack_bf16x2(v.x, v.y);
  }
  tmem_st_32x16(p_addr, packed);
}

__global__ void __launch_bounds__(kThreads, 1)
flash_fwd_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {   // swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicExch(p.error_flag, 25);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::bars);
  uint64_t* q_full = bars;            // 2
  uint64_t* q_empty = bars + 2;       // 2
  uint64_t* kv_full = bars + 4;       // 5
  uint64_t* kv_empty = bars + 9;      // 5
  uint64_t* s_full = bars + 14;       // 2
  uint64_t* p_half = bars + 16;       // 2: keys 0..63 of P are written
  uint64_t* p_ready = bars + 18;      // 2: all of P is written
  uint64_t* o_full = bars + 20;       // 2
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_half[i], 4);
      mbar_init(&p_ready[i], 4);
      mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 9) {
    tmem_alloc(tmem_ptr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  pdl_trigger();
  pdl_wait();

  Items items;
  items.init(p.list);
  int b, sub;
  if (warp >= 8) {
    reg_dealloc<88>();
    if (warp == 8) {
      // ------------------------------ TMA producer ------------------------------
      const bool leader = elect_one();
      uint32_t c = 0, qc[2] = {0, 0};                      // ring slots filled, Q tiles loaded
      while (!__any_sync(0xffffffffu, *abort_flag) && items.next(p.list, b, sub)) {
        const Item it(p, items.level, b, sub);
        if (leader) {
          bool ok = true;
          auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* full, int head, int row) {
            mbar_expect_tx(full, kTileBytes);
            tma_load_2d(dst, tm, full, head * D, row);
            tma_load_2d(dst + kAtom, tm, full, head * D + 64, row);
          };
          auto load_q = [&](int t) {
            if (!ok || it.n[t] == 0) return;
            if (!mbar_wait(&q_empty[t], (qc[t] & 1) ^ 1)) { ok = false; return; }
            load(smem + Smem::q + t * kTileBytes, &tm_q, &q_full[t], it.h[t], it.seq_start + it.q0[t]);
            ++qc[t];
          };
          auto load_kv = [&](const CUtensorMap* tm, int j) {
            const uint32_t slot = c % kSlots;
            if (!ok) return;
            if (!mbar_wait(&kv_empty[slot], ((c / kSlots) & 1) ^ 1)) { ok = false; return; }
            load(smem + Smem::kv + slot * kTileBytes, tm, &kv_full[slot], it.hk, it.k_start + j * BKV);
            ++c;
          };
          const int n = max(it.n[0], it.n[1]);
          load_q(0);
          for (int j = 0; j < n && ok && !*abort_flag; ++j) {
            load_kv(&tm_k, j);
            if (j == 0) load_q(1);
            load_kv(&tm_v, j);
          }
          if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 21); }
        }
        __syncwarp();
      }
    } else if (warp == 9) {
      // ------------------------------ MMA issuer ------------------------------
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);   // S = Q (K-major) · K (K-major)
      constexpr uint32_t idesc_o = make_idesc_bf16(BQ, D, 0, 1);     // O = P (tensor memory) · V (MN-major, N = head dim)
      const uint32_t kv_addr = smem_u32(smem + Smem::kv);
      uint32_t c = 0, qc[2] = {0, 0}, pc[2] = {0, 0};      // ring slots consumed, Q tiles, blocks of P
      while (!__any_sync(0xffffffffu, *abort_flag) && items.next(p.list, b, sub)) {
        const Item it(p, items.level, b, sub);
        const int n = max(it.n[0], it.n[1]);
        if (leader) {
          // block j of this item: K in ring entry c + 2j, V in c + 2j + 1
          auto issue_s = [&](int t, int j) -> bool {
            const uint32_t e = c + 2 * j, slot = e % kSlots;
            if (!mbar_wait(&kv_full[slot], (e / kSlots) & 1)) return false;
            tc_fence_after();
            const uint32_t k_addr = kv_addr + slot * kTileBytes, q_addr = smem_u32(smem + Smem::q) + t * kTileBytes;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)     // 4 K-steps of 16 elements per 64-wide atom
              umma_bf16(tmem + t * 128, make_smem_desc_sw128(q_addr + (ks >> 2) * kAtom + (ks & 3) * 32, 16, 1024),
                        make_smem_desc_sw128(k_addr + (ks >> 2) * kAtom + (ks & 3) * 32, 16, 1024), idesc_s, ks != 0);
            umma_commit(&s_full[t]);
            if (t == 1 || j >= it.n[1]) umma_commit(&kv_empty[slot]);
            if (j + 1 == it.n[t]) umma_commit(&q_empty[t]);
            return true;
          };
          auto issue_pv = [&](int t, int j) -> bool {
            const uint32_t e = c + 2 * j + 1, slot = e % kSlots;
            if (!mbar_wait(&kv_full[slot], (e / kSlots) & 1) || !mbar_wait(&p_half[t], pc[t] & 1)) return false;
            tc_fence_after();
            const uint32_t v_addr = kv_addr + slot * kTileBytes, o = tmem + 256 + t * 128, pt = tmem + t * 128;
            // keys past the last one that the tile sees have weight 0: only the steps that hold others are multiplied
            const int steps = min(BKV / 16, (it.kv_end[t] - j * BKV + 15) / 16);
            auto step = [&](int ks) {
              // V: MN-major, atoms of 64 head-dim columns (LBO = one atom), 16 key rows per step
              umma_bf16_ts(o, pt + ks * 8, make_smem_desc_sw128(v_addr + ks * (16 * 128), kAtom, 1024), idesc_o, (j | ks) != 0);
            };
            for (int ks = 0; ks < min(steps, 4); ++ks) step(ks);
            if (!mbar_wait(&p_ready[t], pc[t] & 1)) return false;
            tc_fence_after();
            for (int ks = 4; ks < steps; ++ks) step(ks);
            ++pc[t];
            if (t == 1 || j >= it.n[1]) umma_commit(&kv_empty[slot]);
            if (j + 1 == it.n[t]) umma_commit(&o_full[t]);
            return true;
          };
          bool ok = true;
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (ok && it.n[t] > 0) {
              ok = mbar_wait(&q_full[t], qc[t] & 1) && issue_s(t, 0);
              ++qc[t];
            }
          for (int j = 0; j < n && ok && !*abort_flag; ++j)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (ok && j < it.n[t]) ok = issue_pv(t, j);
              if (ok && j + 1 < it.n[t]) ok = issue_s(t, j + 1);
            }
          if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 22); }
        }
        c += 2 * n;
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ softmax ------------------------------
    reg_alloc<208>();
    const int t = warp >> 2;                  // tile
    const int q4 = warp & 3;                  // TMEM lane quadrant
    const int row = q4 * 32 + lane;           // query row within the tile
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t t_s = tmem + lane_off + t * 128, t_o = tmem + lane_off + 256 + t * 128;
    const float sl2 = p.scale * kLog2e;
    uint32_t sc = 0, oc = 0;                  // blocks of S, items
    bool ok = true;
    while (items.next(p.list, b, sub)) {
      const Item it(p, items.level, b, sub);
      const int n = t ? it.n[1] : it.n[0], q0 = t ? it.q0[1] : it.q0[0], h = t ? it.h[1] : it.h[0], qpos = q0 + row;
      if (n == 0) continue;
      const int last = p.causal ? min(it.Lk - 1, qpos + it.off) : it.Lk - 1;      // last key the row sees
      const int all = p.causal ? min(it.Lk, q0 + it.off + 1) : it.Lk;             // keys before this one are seen by every row
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n; ++j) {
        if (__any_sync(0xffffffffu, !mbar_wait(&s_full[t], sc & 1) || *abort_flag)) { ok = false; break; }
        ++sc;
        tc_fence_after();
        uint32_t s[4][32];
#pragma unroll
        for (int k = 0; k < 4; ++k) tmem_ld_32x32(t_s + k * 32, s[k]);
        tmem_ld_wait();
        if ((j + 1) * BKV > all) {
          const int lim = last - j * BKV;
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (k * 32 + i > lim) s[k][i] = 0xff800000u;       // −infinity
        }
        float mx4[4] = {m_run, -INFINITY, -INFINITY, -INFINITY};   // independent chains
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int i = 0; i < 32; i += 2) mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(s[k][i]), __uint_as_float(s[k][i + 1]));
        float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]);
        // Lazy rescaling: keep the old reference maximum while the true maximum is less than 2^8 above it (P stays ≤ 256,
        // exact in the fp32 accumulator); the final O / l and the log-sum-exp are unaffected by which reference is used.
        if (m_run != -INFINITY && (mx - m_run) * sl2 <= 8.0f) mx = m_run;
        const float msc = (mx == -INFINITY) ? 0.f : mx * sl2;
        if (__any_sync(0xffffffffu, mx != m_run)) {
          const float alpha = (m_run == -INFINITY) ? 0.f : exp2f(m_run * sl2 - msc);
          l_run *= alpha;
          if (j > 0) {          // S of this block is complete, so P·V of the earlier ones is (issue order): O is stable
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
              uint32_t o[32];
              tmem_ld_32x32(t_o + k * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32(t_o + k * 32, o);
            }
          }
          m_run = mx;
        }
        float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float2 scale2 = make_float2(sl2, sl2), minus2 = make_float2(-msc, -msc);
        exp_chunk(s[0], scale2, minus2, sum, t_s);
        exp_chunk(s[1], scale2, minus2, sum, t_s + 16);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_half[t]);
        exp_chunk(s[2], scale2, minus2, sum, t_s + 32);
        exp_chunk(s[3], scale2, minus2, sum, t_s + 48);
        l_run += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[t]);
      }
      if (!ok || __any_sync(0xffffffffu, !mbar_wait(&o_full[t], oc & 1) || *abort_flag)) { ok = false; break; }
      ++oc;
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const bool valid = qpos < it.L;
      __nv_bfloat16* orow = p.o + (static_cast<long long>(it.seq_start + qpos) * p.Hq + h) * D;
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        uint32_t o[32];
        tmem_ld_32x32(t_o + k * 32, o);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + k * 32 + i) = w;
          }
        }
      }
      tc_fence_before();                      // O is read: the next item's P·V may overwrite it (it waits for that item's P)
      if (valid && p.lse != nullptr)
        p.lse[static_cast<long long>(h) * p.total_tokens + it.seq_start + qpos] = (l_run > 0.f) ? m_run * p.scale + logf(l_run) : -INFINITY;
    }
    if (!ok) {
      *abort_flag = 1;
      atomicExch(p.error_flag, 23);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace fa
}  // namespace mb

using namespace mb;

static cudaError_t fa_configure() {
  static const cudaError_t e = cudaFuncSetAttribute(fa::flash_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fa::Smem::total);
  return e;
}

// resident CTAs per SM of the forward kernel at its launch configuration (diagnostic; 1 is the design point)
extern "C" int mb_flash_fwd_tc_ctas_per_sm() {
  int n = 0;
  (void)fa_configure();
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fa::flash_fwd_tc_kernel, fa::kThreads, fa::Smem::total) != cudaSuccess) return -1;
  return n;
}

// q [T, Hq, 128] (token stride q_stride elements), k/v [T, Hkv, 128]; o [T, Hq, 128] contiguous; lse [Hq, T].
// cu_seqlens_k / total_k_tokens: optional separate key sequences (null / 0: the queries' own), see Params.
extern "C" int mb_flash_fwd_tc(const void* q, const void* k, const void* v, void* o, float* lse, const int* cu_seqlens, int batch,
                               int max_seqlen, int total_tokens, long long q_stride, long long k_stride, long long v_stride, int Hq,
                               int Hkv, float scale, int causal, int* error_flag, const int* cu_seqlens_k, int total_k_tokens,
                               cudaStream_t s) {
  if (batch == 0 || total_tokens == 0 || max_seqlen == 0) return 0;
  const int tk_rows = cu_seqlens_k != nullptr ? total_k_tokens : total_tokens;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_bf16_2d(&tq, q, total_tokens, static_cast<long long>(Hq) * fa::D, q_stride, fa::BQ, 64);
  if (rc) return 1000 + rc;
  rc = make_tmap_bf16_2d(&tk, k, tk_rows, static_cast<long long>(Hkv) * fa::D, k_stride, fa::BKV, 64);
  if (rc) return 2000 + rc;
  rc = make_tmap_bf16_2d(&tv, v, tk_rows, static_cast<long long>(Hkv) * fa::D, v_stride, fa::BKV, 64);
  if (rc) return 3000 + rc;
  if (const cudaError_t e = fa_configure(); e != cudaSuccess) return static_cast<int>(e);
  fa::Params p{};
  p.o = reinterpret_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.cu_seqlens = cu_seqlens;
  p.cu_seqlens_k = cu_seqlens_k;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.total_tokens = total_tokens;
  p.scale = scale;
  p.causal = causal;
  p.error_flag = error_flag;
  // two heads with the same keys have equal ranges; two neighbouring tiles of one head do not, but serve any number of heads
  p.pair_heads = (Hq / Hkv) % 2 == 0;
  const int rows = p.pair_heads ? fa::BQ : 2 * fa::BQ;
  p.list = ItemList{cu_seqlens, batch, p.pair_heads ? Hq / 2 : Hq, (max_seqlen + rows - 1) / rows, rows};
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long most = static_cast<long long>(p.list.levels) * batch * p.list.per_seq;
  const int grid = static_cast<int>(most < sms ? most : sms);
  return static_cast<int>(launch_pdl(fa::flash_fwd_tc_kernel, dim3(grid), dim3(fa::kThreads), fa::Smem::total, s, tq, tk, tv, p));
}
