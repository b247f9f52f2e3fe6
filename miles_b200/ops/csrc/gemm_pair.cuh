// bf16 GEMM on pairs of SMs: a cluster of two CTAs works on one 256 × BN tile with tcgen05 `cta_group::2`.
//
// Same products and operand layouts as gemm.cu (which picks between the two and holds the host code).  CTA r of a pair keeps rows
// 128·r .. 128·r + 127 of A and of the accumulator, and half of B's BN rows; the first CTA issues every MMA for both.
//   warp 0       TMA producer of the CTA's own operands; all bytes of a stage are counted on the first CTA's barrier
//   warp 1       TMEM allocation; in the first CTA also the MMA issue (one elected lane).  Commits arrive in both CTAs
//   warps 2..9   epilogue of the CTA's own 128 rows, two warps per lane quadrant (half of the columns each); the accumulator is double
//                buffered.  Four warps cannot drain a tile in the time of a short reduction (768 in the experts' second product)
//
// What bounds it.  One CTA's 128 × 256 tile reads 48 KB of operands from shared memory per 512 tensor clocks and holds 4 stages; a
// pair reads 32 KB per CTA for the same work and holds 6, and an operand row travels from L2 once per 256 rows of the other operand instead of
// once per 128 (A) or 256 (B).  Tiles run in groups of kGroupM row tiles, columns outer: the tiles that are in flight together
// cover about as many rows as columns, so that large A and B are both read from memory about once (columns-outermost over all rows
// read A again for every column tile as soon as it outgrows L2, as the expert-sorted rows do).  Measured against gemm.cu's 128 × 256
// tiles, same call: 8192³ 825 → 693 µs (1587 TFLOP/s; torch.matmul 684), 11791 × 19456 × 2560 911 → 760, weight gradient
// 16384 × 2048 over 8043 rows 448 → 356, experts' first product over 96 600 rows (16 × 1536 × 2048) 556 → 411, second (2048 × 768)
// 350 → 240 (four epilogue warps: 285).
//
// Grouped forward: segments are padded to 128 rows, so a tile's two halves may belong to two experts.  Such a tile runs twice, once
// per expert, and each CTA stores the pass that is its own: at most one tile in (experts − 1) boundaries, against padding to 256 rows.
#pragma once
#include "gemm_epilogue.cuh"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

struct GemmParams {
  int M, N, K;
  void* C;
  long long ldc;           // elements
  long long group_stride_c;  // elements between per-group outputs (grouped wgrad)
  int out_fp32;
  int accumulate;
  const __nv_bfloat16* bias;
  const int* tile_expert;  // grouped fwd: [m_tiles]
  const int* seg_offsets;  // grouped wgrad: [groups+1], multiples of BK
  int num_groups;
  int b_group_rows;        // grouped fwd: rows of B per expert (N for K-major B, K for MN-major B)
  int glu_rows;            // > 0: B is [gate; up] of this many rows each, see GluTile
  int* error_flag;
  // split-K (dense, few output tiles): `split_k` CTAs share one output tile, each writing the partial sums of its K slice
  // to its own fp32 plane of `ws` [split_k, M, N]; the last to arrive (counter per tile and 32-row quadrant) adds the
  // planes in slice order, writes C and resets the counter
  int split_k;
  float* ws;
  int* counters;
};

static inline int num_sms() {
  static int g_num_sms = 0;
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_num_sms;
}

namespace pair {

static constexpr int kBM = 128, kBK = 64, kUmmaK = 16;      // rows per CTA
static constexpr int kStages = 6;
static constexpr int kEpilogueWarps = 8, kThreads = 64 + 32 * kEpilogueWarps;
static constexpr int kGroupM = 8;                           // row tiles (of 256) per group of the tile order
// (1 / 8 / 16: 8192³ 743 / 693 / 696 µs, 16384 × 18992 × 2048 885 / 822 / 800, 16384 × 2048 × 4096 169 / 169 / 173: 8 is never far off)

template <int BN>
struct Layout {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = BN / 2 * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kBarrierBytes = 256;
  static constexpr int kTotal = kStages * kStageBytes + kBarrierBytes + kEpilogueWarps * 4096 + 1024;   // + epilogue staging + alignment slack
};

// Tile t of a group's rows and columns.
__device__ __forceinline__ void tile_of(int t, int m_tiles, int n_tiles, int& m, int& n) {
  const int per_group = kGroupM * n_tiles;
  const int first = t / per_group * kGroupM;
  const int rows = min(kGroupM, m_tiles - first);
  const int r = t % per_group;
  m = first + r % rows;
  n = r / rows;
}

// What a warp does with its 32 rows of a BN-column accumulator (columns from t_acc on; two warps per lane quadrant, `half` 0 and 1): stores
// them, makes gate · up of them, or what head.cu makes of them.
struct StoreTile {
  template <int BN>
  __device__ __forceinline__ void tile(const GemmParams& p, int group, int row0, uint32_t t_acc, uint8_t* stage, int n, int half, bool empty) const {
    const TileOut out{reinterpret_cast<uint8_t*>(p.C) + (static_cast<long long>(group) * p.group_stride_c + static_cast<long long>(row0) * p.ldc) * (p.out_fp32 ? 4 : 2),
                      p.ldc, p.M - row0, p.N, p.out_fp32, p.accumulate, p.bias};
    store_tile_staged<BN / 2>(out, t_acc + half * (BN / 2), stage, n * BN + half * (BN / 2), empty);
  }
};

// silu(gate) · up of 128 gate and 128 up columns (p.glu_rows > 0: the first CTA loads gate rows, the second up rows) → 128 bf16 columns.
// Without autograd nobody needs the pre-activations: they are neither written nor read back.  Both are rounded to bf16 first, which makes
// the result the same bits as the two kernels' (a rollout and its trainer have to agree).
struct GluTile {
  template <int BN>
  __device__ __forceinline__ void tile(const GemmParams& p, int, int row0, uint32_t t_acc, uint8_t* stage, int n, int half, bool) const {
    static_assert(BN == 256, "64 output columns per warp");
    const int lane = static_cast<int>(lane_id()), col0 = n * 128 + half * 64, F = p.glu_rows;
    if (col0 >= F) return;                                    // uniform
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t g[32], u[32];
      tmem_ld_32x32(t_acc + half * 64 + c * 32, g);
      tmem_ld_32x32(t_acc + 128 + half * 64 + c * 32, u);
      tmem_ld_wait();
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t gp = pack_bf16x2(__uint_as_float(g[2 * i]), __uint_as_float(g[2 * i + 1])), up = pack_bf16x2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
        const float g0 = __uint_as_float(gp << 16), g1 = __uint_as_float(gp & 0xffff0000u);
        o[i] = pack_bf16x2(g0 / (1.f + __expf(-g0)) * __uint_as_float(up << 16), g1 / (1.f + __expf(-g1)) * __uint_as_float(up & 0xffff0000u));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + i) ^ (lane & 7)) << 4)) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
    }
    __syncwarp();
    const int unit = lane & 7, col = col0 + unit * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int rr = k * 4 + (lane >> 3);
      if (row0 + rr < p.M && col < F)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(row0 + rr) * p.ldc + col) =
            *reinterpret_cast<const uint4*>(stage + rr * 128 + ((unit ^ (rr & 7)) << 4));
    }
    __syncwarp();
  }
};

// A_MN, B_MN, MODE: as gemm_bf16_kernel.
template <int BN, int A_MN, int B_MN, int MODE, class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmParams p, Epi epi) {
  using L = Layout<BN>;
  constexpr bool kFwd = MODE == 1, kWgrad = MODE == 2;
  constexpr uint32_t kTmemCols = 2 * BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kStages * L::kABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * L::kStageBytes);   // first CTA: both CTAs' bytes
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tmem_full = empty_bar + kStages;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;        // [2], first CTA: the epilogue warps of both CTAs
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_ptr + 1);
  uint8_t* smem_stage = smem + kStages * L::kStageBytes + L::kBarrierBytes;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int m_tiles = (p.M + 2 * kBM - 1) / (2 * kBM);
  const int n_tiles = (p.N + BN - 1) / BN;
  const int per_group = m_tiles * n_tiles;
  const int total_tiles = kWgrad ? per_group * p.num_groups : per_group;
  const int first_tile = static_cast<int>(blockIdx.x >> 1), step = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 2 * kEpilogueWarps); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) tmem_alloc_pair(tmem_base_ptr, kTmemCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                              // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_ptr;
  pdl_trigger();
  pdl_wait();

  auto k_range = [&](int group, int& k0, int& k_blocks) {
    if (kWgrad) {
      k0 = p.seg_offsets[group];
      k_blocks = (p.seg_offsets[group + 1] - k0) / kBK;
    } else {
      k0 = 0;
      k_blocks = (p.K + kBK - 1) / kBK;
    }
  };
  // Pass 0 or 1 of tile row `m`: false if there is none.  `expert`: whose weights (grouped forward), `mine`: this CTA stores the result.
  auto pass_of = [&](int m, int pass, int& expert, bool& mine) -> bool {
    expert = 0;
    mine = true;
    if (!kFwd) return pass == 0;
    const int e0 = p.tile_expert[2 * m], e1 = (2 * m + 1) * kBM < p.M ? p.tile_expert[2 * m + 1] : -1;
    expert = pass == 0 ? e0 : e1;
    mine = (rank == 0 ? e0 : e1) == expert;
    return expert >= 0 && (pass == 0 || e1 != e0);
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = first_tile; t < total_tiles && ok; t += step) {
        const int group = kWgrad ? t / per_group : 0;
        int m, n, k0, k_blocks, expert;
        bool mine;
        tile_of(kWgrad ? t % per_group : t, m_tiles, n_tiles, m, n);
        k_range(group, k0, k_blocks);
        const int a_row = (2 * m + rank) * kBM, b_row = p.glu_rows > 0 ? n * (BN / 2) + rank * p.glu_rows : n * BN + rank * (BN / 2);
        for (int pass = 0; pass < 2 && ok; ++pass) {
          if (!pass_of(m, pass, expert, mine)) continue;
          const int b_off = kFwd ? expert * p.b_group_rows : 0;
          for (int kb = 0; kb < k_blocks; ++kb) {
            if (!mbar_wait_cluster(&empty_bar[stage], phase ^ 1) || *abort_flag) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * L::kStageBytes);
            const uint32_t bar = smem_of_rank(&full_bar[stage], 0);
            const int kc = k0 + kb * kBK;
            uint8_t* sa = smem_a + stage * L::kABytes;
            uint8_t* sb = smem_b + stage * L::kBBytes;
            if (A_MN) {
#pragma unroll
              for (int a = 0; a < kBM / 64; ++a) tma_load_2d_pair(sa + a * (kBK * 128), &tmap_a, bar, a_row + a * 64, kc);
            } else {
              tma_load_2d_pair(sa, &tmap_a, bar, kc, a_row);
            }
            if (B_MN) {
#pragma unroll
              for (int b = 0; b < BN / 128; ++b) tma_load_2d_pair(sb + b * (kBK * 128), &tmap_b, bar, b_row + b * 64, kc + b_off);
            } else {
              tma_load_2d_pair(sb, &tmap_b, bar, kc, b_row + b_off);
            }
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 1); }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (first CTA) ------------------------------
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * kBM, BN, A_MN, B_MN);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int t = first_tile; t < total_tiles && ok; t += step) {
        const int group = kWgrad ? t / per_group : 0;
        int m, n, k0, k_blocks, expert;
        bool mine;
        tile_of(kWgrad ? t % per_group : t, m_tiles, n_tiles, m, n);
        k_range(group, k0, k_blocks);
        for (int pass = 0; pass < 2 && ok; ++pass) {
          if (!pass_of(m, pass, expert, mine)) continue;
          if (!mbar_wait_cluster(&tmem_empty[acc], acc_phase ^ 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          for (int kb = 0; kb < k_blocks; ++kb) {
            if (!mbar_wait_cluster(&full_bar[stage], phase) || *abort_flag) { ok = false; break; }
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem_a + stage * L::kABytes);
            const uint32_t b_addr = smem_u32(smem_b + stage * L::kBBytes);
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k) {
              const uint64_t ad = A_MN ? make_smem_desc_sw128(a_addr + k * (kUmmaK * 128), kBK * 128, 1024)
                                       : make_smem_desc_sw128(a_addr + k * (kUmmaK * 2), 16, 1024);
              const uint64_t bd = B_MN ? make_smem_desc_sw128(b_addr + k * (kUmmaK * 128), kBK * 128, 1024)
                                       : make_smem_desc_sw128(b_addr + k * (kUmmaK * 2), 16, 1024);
              umma_bf16_pair(d_tmem, ad, bd, idesc, (kb | k) != 0);
            }
            umma_commit_pair(&empty_bar[stage]);   // frees the stage in both CTAs once these MMAs have read it
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          umma_commit_pair(&tmem_full[acc]);       // an empty reduction range: nothing was issued, the epilogue writes zeros
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 2); }
    }
  } else {
    // ------------------------------ epilogue (warps 2..9) ------------------------------
    const int q = warp & 3;  // TMEM lane quadrant this warp may access
    const int half = (warp - 2) / 4;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = first_tile; t < total_tiles && ok; t += step) {
      const int group = kWgrad ? t / per_group : 0;
      int m, n, k0, k_blocks, expert;
      bool mine;
      tile_of(kWgrad ? t % per_group : t, m_tiles, n_tiles, m, n);
      k_range(group, k0, k_blocks);
      for (int pass = 0; pass < 2 && ok; ++pass) {
        if (!pass_of(m, pass, expert, mine)) continue;
        if (__any_sync(0xffffffffu, !mbar_wait_cluster(&tmem_full[acc], acc_phase) || *abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (mine)
          epi.template tile<BN>(p, group, (2 * m + rank) * kBM + q * 32, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN,
                                smem_stage + (warp - 2) * 4096, n, half, k_blocks == 0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(smem_of_rank(&tmem_empty[acc], 0));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
    if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 4); }
  }

  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync();                              // the peer has stopped reading this CTA's memory and arriving on its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

template <int BN, int A_MN, int B_MN, int MODE, class Epi>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, const Epi& epi, int tiles, cudaStream_t stream) {
  using L = Layout<BN>;
  auto kern = gemm_bf16_pair_kernel<BN, A_MN, B_MN, MODE, Epi>;
  static const cudaError_t configured = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
  if (configured != cudaSuccess) return static_cast<int>(configured);
  const int pairs = num_sms() / 2;
  return static_cast<int>(launch_pdl(kern, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kThreads), L::kTotal, stream, ta, tb, p, epi));
}

}  // namespace pair
}  // namespace mb
