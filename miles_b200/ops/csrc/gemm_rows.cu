// Projections of up to 64 tokens:  C[tokens, N] = X[tokens, K] · W[N, K]ᵀ  with every SM streaming weights.  Up to 8 tokens that is for weights
// of more than 12 Mi elements (smaller ones: gemv.cu), from 9 on for any.
//
// Up to 16 tokens with an RMSNorm in front (norm_rows): the staged operand is bf16(h · norm_w), h the sum with the residual as it is stored, and
// 1 / rms multiplies the fp32 sums in the epilogue.  That is the arithmetic of gemv.cu: one rounding of the operand where the norm weight
// is not a power of two, none where it is one; bf16(h / rms · norm_w) always has one (outputs in bf16, norm weights of one, hidden 2560: 2.4e-3
// from 64 bits, 1.7e-3 this way, which is the rounding of the output alone; fp32 router scores lose that rounding altogether).
//
// As in gemm_small.cu the weight rows are the 128-row side of the MMA and the tokens its N side (16, 32 or 64).  A projection of a model
// has 16 to 160 such tiles, so the reduction is cut as well: a CLUSTER of 1, 2, 4 or 8 CTAs shares one tile, each CTA streams its slice of
// K, and the partial accumulators meet in distributed shared memory.  CTA r of a cluster owns tokens [r · BT/S, (r + 1) · BT/S): every CTA
// stores its partial sums of those tokens into r's buffer, and after one cluster barrier r adds them in slice order and writes them out.
//   warp 0      TMA producer.  Weights that no kernel of the stream writes (`static_w`) are requested before the dependency wait: the
//               first stages arrive while the kernel in front is still running
//   warp 1      TMEM + tcgen05.mma issue
//   warps 2..5  accumulator → owners' buffers → output
//
// What bounds it: the weight bytes, and with 5 to 100 MB of them per call the time until all SMs have loads in flight.  Two CTAs fit an SM
// (72 to 90 KB in flight each), so up to 296 tiles × slices run at once and 152 tiles do not become two waves; where all of them fit with an
// SM each, the ring is as deep as the SM allows.  The earlier forms were
// 128-row token tiles (3/4 padding) with 64 columns per CTA, whose sums over K met in global memory behind atomic counters for ≤ 32 tokens.
// gate · up where the accumulator is read (kGlu) instead of a kernel behind: decode steps of 8 layers, hidden 1024, 12 / 30 / 60 rows 358 / 446 / 506 → 354 / 440 /
// 500 µs, hidden 2560, 12 layers, 19 rows 1054 → 1036.
// Measured, weights from memory, 9 / 19 / 61 tokens against the 128-row tiles: 5120 × 2048 15.4 / 14.9 / 8.8 → 6.2 / 6.3 / 8.4 µs,
// 2048 × 4096 17.0 / 13.0 / 13.1 → 6.2 / 6.8 / 8.2, 2560 × 9728 26.6 / 26.7 / 26.7 → 11.1 / 11.7 / 13.9 (7.7 at the memory's speed).
#include "launch.h"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);

namespace rows {

static constexpr int BMW = 128;     // weight rows (output features) per tile
static constexpr int BK = 64;
static constexpr int kMaxSplit = 8;
static constexpr int kSms = 148, kWideClusters = 12, kMaxExperts = 256;

struct Params {
  int tokens, N, K;
  void* C;
  long long ldc;
  int out_fp32;
  const __nv_bfloat16* bias;
  const float* row_scale;             // [tokens] factors on the sums, or null
  int static_w;
  int stages;
  int* error_flag;
  const int* slots;                   // experts: how many there are and which, see below
  int steps_per;                      // experts: 64-deep steps of one expert's share of the reduction
};

template <int BT>
struct Layout {
  static constexpr int kShallow = BT == 64 ? 3 : BT == 32 ? 4 : 5, kDeep = BT == 64 ? 8 : BT == 32 ? 10 : 12;   // stages: two CTAs per SM, one
  static constexpr int kABytes = BMW * BK * 2;         // weights: 16 KB
  static constexpr int kBBytes = BT * BK * 2;          // tokens: 2 / 4 / 8 KB
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kSumBytes = BT * BMW * 4;       // [slice][own tokens][feature] floats, where the reduction is cut
  static constexpr int total(int stages, bool cut) { return stages * kStageBytes + (cut ? kSumBytes : 0) + 256 + 1024; }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// kExperts: the weights are [E, N, K_e] and the reduction runs over the experts of `slots` one after another (X has their columns in that order).
// kGlu: the weights are [gate; up] of N / 2 rows each; a tile has 64 of both, C [tokens, N / 2] = silu(gate) · up, both rounded to bf16 first, which
// makes the result the same bits as the activation kernel's.
enum Mode { kPlain = 0, kExpertSum = 1, kGluPair = 2 };

template <int BT, int split, int mode>
__global__ void __launch_bounds__(192, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, Params p) {
  using L = Layout<BT>;
  constexpr bool kExperts = mode == kExpertSum, kGlu = mode == kGluPair;
  constexpr uint32_t kTmemCols = BT < 32 ? 32 : BT;
  const int stages = p.stages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + stages * L::kABytes;
  float* sums = reinterpret_cast<float*>(smem + stages * L::kStageBytes);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + stages * L::kStageBytes + (split > 1 ? L::kSumBytes : 0));
  uint64_t* empty_bar = full_bar + stages;
  uint64_t* tmem_full = empty_bar + stages;
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(tmem_full + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slice = static_cast<int>(blockIdx.x) % split, n_blk = static_cast<int>(blockIdx.x) / split;   // the cluster is one tile's slices

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(tmem_full, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_ptr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_ptr;
  if (split > 1) cluster_arrive();                 // "my buffer exists": waited for before the first remote store
  pdl_trigger();

  __shared__ int slot_e[kExperts ? kMaxExperts : 1];
  int total_kb = (p.K + BK - 1) / BK;
  if (kExperts) {                                  // nothing is known before the kernel in front has written the list
    pdl_wait();
    const int n = p.slots[0];
    for (int i = threadIdx.x; i < n; i += 192) slot_e[i] = p.slots[1 + i];
    __syncthreads();
    total_kb = n * p.steps_per;
  }
  const int per = (total_kb + split - 1) / split;
  const int kb0 = slice * per, kbs = max(0, min(per, total_kb - kb0));

  if (warp == 0) {
    if (elect_one()) {
      auto load_w = [&](int kb, int stage) {
        mbar_expect_tx(&full_bar[stage], L::kStageBytes);
        const int at = kb0 + kb;
        if (kExperts) tma_load_2d(smem_a + stage * L::kABytes, &tmap_w, &full_bar[stage], at % p.steps_per * BK, slot_e[at / p.steps_per] * p.N + n_blk * BMW);
        else if (!kGlu) tma_load_2d(smem_a + stage * L::kABytes, &tmap_w, &full_bar[stage], at * BK, n_blk * BMW);
        else
          for (int h = 0; h < 2; ++h)
            tma_load_2d(smem_a + stage * L::kABytes + h * (L::kABytes / 2), &tmap_w, &full_bar[stage], at * BK, n_blk * (BMW / 2) + h * (p.N / 2));
      };
      auto load_x = [&](int kb, int stage) { tma_load_2d(smem_b + stage * L::kBBytes, &tmap_x, &full_bar[stage], (kb0 + kb) * BK, 0); };
      const int early = min(kbs, stages);
      if (p.static_w)
        for (int kb = 0; kb < early; ++kb) load_w(kb, kb);
      pdl_wait();
      for (int kb = 0; kb < early; ++kb) {
        if (!p.static_w) load_w(kb, kb);
        load_x(kb, kb);
      }
      for (int kb = early; kb < kbs; ++kb) {
        const int stage = kb % stages;
        if (!mbar_wait(&empty_bar[stage], (kb / stages - 1) & 1)) { atomicExch(p.error_flag, 45); break; }
        load_w(kb, stage);
        load_x(kb, stage);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BMW, BT, 0, 0);
      for (int kb = 0; kb < kbs; ++kb) {
        const int stage = kb % stages;
        if (!mbar_wait(&full_bar[stage], (kb / stages) & 1)) { atomicExch(p.error_flag, 46); break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem_a + stage * L::kABytes);
        const uint32_t b_addr = smem_u32(smem_b + stage * L::kBBytes);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_bf16(tmem_base, make_smem_desc_sw128(a_addr + k * 32, 16, 1024), make_smem_desc_sw128(b_addr + k * 32, 16, 1024), idesc, (kb | k) != 0);
        umma_commit(&empty_bar[stage]);
      }
      umma_commit(tmem_full);
    }
    __syncwarp();
  }
  const int q = warp & 3;
  const int n = n_blk * BMW + q * 32 + lane;         // output feature of this thread (warps 2..5)
  __shared__ float scale[4][BT];                     // a copy per warp, fetched while the products run
  float v[BT];
  if (warp >= 2) {
    pdl_wait();                                      // C, the bias and the factors: after the kernels in front
    if (p.row_scale != nullptr)
      for (int i = lane; i < p.tokens; i += 32) scale[q][i] = p.row_scale[i];
    if (!mbar_wait(tmem_full, 0)) atomicExch(p.error_flag, 47);
    __syncwarp();
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < BT / 16; ++c) {
      uint32_t r[16];
      tmem_ld_32x16(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + c * 16, r);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) v[c * 16 + i] = kbs > 0 ? __uint_as_float(r[i]) : 0.f;
    }
    tc_fence_before();
  }
  const int tokens = n < p.N ? p.tokens : 0;         // a feature past the last one stores nothing
  const float bias = warp >= 2 && tokens > 0 && p.bias != nullptr ? __bfloat162float(p.bias[n]) : 0.f;
  auto put = [&](int tok, float x) {                 // lanes hold consecutive features: one 64- or 128-byte store per token and warp
    if (p.row_scale != nullptr) x *= scale[q][tok];
    if (p.bias != nullptr) x += bias;
    if (p.out_fp32) reinterpret_cast<float*>(p.C)[tok * p.ldc + n] = x;
    else reinterpret_cast<__nv_bfloat16*>(p.C)[tok * p.ldc + n] = __float2bfloat16(x);
  };
  auto put_glu = [&](int tok, float gate, float up) {        // warps on gate rows
    const float f = p.row_scale != nullptr ? scale[q][tok] : 1.f;
    gate = __bfloat162float(__float2bfloat16(gate * f));
    up = __bfloat162float(__float2bfloat16(up * f));
    reinterpret_cast<__nv_bfloat16*>(p.C)[tok * p.ldc + n_blk * (BMW / 2) + q * 32 + lane] = __float2bfloat16(gate / (1.f + __expf(-gate)) * up);
  };
  if (split == 1 && kGlu) {
    if (warp >= 2) {
      float* ups = reinterpret_cast<float*>(smem);     // [token][64]: the products are done, nothing reads or writes the ring any more
      if (q >= 2) {
#pragma unroll
        for (int i = 0; i < BT; ++i)
          if (i < p.tokens) ups[i * 64 + (q - 2) * 32 + lane] = v[i];
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (q < 2) {
#pragma unroll
        for (int i = 0; i < BT; ++i)
          if (i < p.tokens) put_glu(i, v[i], ups[i * 64 + q * 32 + lane]);
      }
    }
  } else if (split == 1) {
    if (warp >= 2) {
#pragma unroll
      for (int i = 0; i < BT; ++i)
        if (i < tokens) put(i, v[i]);
    }
  } else {
    constexpr int own = BT / split;
    cluster_wait();
    if (warp >= 2) {
#pragma unroll
      for (int o = 0; o < split; ++o) {
        const uint32_t to = smem_of_rank(sums + slice * own * BMW + q * 32 + lane, o);
#pragma unroll
        for (int i = 0; i < own; ++i)
          if (o * own + i < tokens) st_cluster(to + i * BMW * 4, v[o * own + i]);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                  // every slice's sums are in their owners' buffers; nothing remote is touched after this
    if (warp >= 2 && kGlu) {
#pragma unroll 4
      for (int i = 0; q < 2 && i < min(own, p.tokens - slice * own); ++i) {
        float gate = 0.f, up = 0.f;
#pragma unroll
        for (int s = 0; s < split; ++s) {
          gate += sums[(s * own + i) * BMW + q * 32 + lane];
          up += sums[(s * own + i) * BMW + 64 + q * 32 + lane];
        }
        put_glu(slice * own + i, gate, up);
      }
    } else if (warp >= 2) {
#pragma unroll 4
      for (int i = 0; i < min(own, tokens - slice * own); ++i) {
        float x = 0.f;
#pragma unroll
        for (int s = 0; s < split; ++s) x += sums[(s * own + i) * BMW + q * 32 + lane];
        put(slice * own + i, x);
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int BT, int split, int mode>
static int launch_as(const CUtensorMap& tw, const CUtensorMap& tx, Params p, cudaStream_t s) {
  using L = Layout<BT>;
  constexpr int kDeep = mode == kExpertSum && BT == 64 ? L::kDeep - 1 : L::kDeep;        // room for the list of experts
  auto kern = gemm_rows_kernel<BT, split, mode>;
  static const cudaError_t configured = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total(kDeep, split > 1));
  if (configured != cudaSuccess) return static_cast<int>(configured);
  const int tiles = (p.N + BMW - 1) / BMW;
  // a CTA with an SM to itself has twice the bytes in flight: the ring is deep where all clusters fit that way.  Eight neighbouring SMs are
  // found 12 times at least.  An uncut reduction has no buffers for sums: room for one stage more beside a second CTA (19456 × 2560, 19 tokens: 20.1 → 19.2 µs)
  p.stages = tiles <= (split == kMaxSplit ? kWideClusters : kSms / split) ? kDeep : L::kShallow + (split == 1 ? 1 : 0);
  return static_cast<int>(launch_pdl_cluster(kern, dim3(tiles * split), dim3(192), split, L::total(p.stages, split > 1), s, tw, tx, p));
}

template <int BT, int mode>
static int launch(const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int split, cudaStream_t s) {
  switch (split) {
    case 1: return launch_as<BT, 1, mode>(tw, tx, p, s);
    case 2: return launch_as<BT, 2, mode>(tw, tx, p, s);
    case 4: return launch_as<BT, 4, mode>(tw, tx, p, s);
    default: return launch_as<BT, 8, mode>(tw, tx, p, s);
  }
}

template <int mode>
static int launch_mode(int bt, const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int split, cudaStream_t s) {
  switch (bt) {
    case 16: return launch<16, mode>(tw, tx, p, split, s);
    case 32: return launch<32, mode>(tw, tx, p, split, s);
    default: return launch<64, mode>(tw, tx, p, split, s);
  }
}

// One row per CTA: h = bf16(x + residual) → sum (if there is a residual), bf16(h · w) → scaled, 1 / rms(h) → rstd and, if wanted, bf16(h / rms · w)
// → normed.  A handful of rows: the time is one launch and two trips to memory.
__global__ void __launch_bounds__(256) norm_rows_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual, const __nv_bfloat16* w, float eps, int K,
                                                        __nv_bfloat16* scaled, float* rstd_out, __nv_bfloat16* sum, __nv_bfloat16* normed) {
  __shared__ float part[8];
  pdl_trigger();
  pdl_wait();
  const long long row = static_cast<long long>(blockIdx.x) * K;
  auto two = [](uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); };
  auto times_w = [&](uint4 h, int at, float f) {
    const uint4 wv = *reinterpret_cast<const uint4*>(w + at);
    const uint32_t hs[4] = {h.x, h.y, h.z, h.w}, ws[4] = {wv.x, wv.y, wv.z, wv.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = two(hs[i]), b = two(ws[i]);
      o[i] = pack_bf16x2(a.x * f * b.x, a.y * f * b.y);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
  };
  float ss = 0.f;
  for (int at = threadIdx.x * 8; at < K; at += 2048) {
    uint4 h = *reinterpret_cast<const uint4*>(x + row + at);
    uint32_t* hs = &h.x;
    if (residual != nullptr) {
      const uint4 r = *reinterpret_cast<const uint4*>(residual + row + at);
      const uint32_t rs[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = two(hs[i]), b = two(rs[i]);
        hs[i] = pack_bf16x2(a.x + b.x, a.y + b.y);
      }
      *reinterpret_cast<uint4*>(sum + row + at) = h;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = two(hs[i]);
      ss += a.x * a.x + a.y * a.y;
    }
    *reinterpret_cast<uint4*>(scaled + row + at) = times_w(h, at, 1.f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) ss += part[i];
  const float rstd = rsqrtf(ss / K + eps);
  if (threadIdx.x == 0) rstd_out[blockIdx.x] = rstd;
  if (normed != nullptr)
    for (int at = threadIdx.x * 8; at < K; at += 2048)       // this thread's own pieces again
      *reinterpret_cast<uint4*>(normed + row + at) = times_w(*reinterpret_cast<const uint4*>((residual != nullptr ? sum : x) + row + at), at, rstd);
}

}  // namespace rows
}  // namespace mb

// See norm_rows_kernel; x, residual (or null), sum, scaled, normed (or null) [T, K] bf16, w [K] bf16, all 16-byte aligned, K a multiple of 8.
extern "C" int mb_norm_rows(const void* x, const void* residual, const void* w, float eps, int T, int K, void* scaled, float* rstd, void* sum, void* normed,
                            cudaStream_t s) {
  using namespace mb;
  typedef const __nv_bfloat16* cbf;
  typedef __nv_bfloat16* bf;
  if (T <= 0) return 0;
  if (K % 8 || (residual != nullptr && sum == nullptr)) return -2;
  const uintptr_t pointers = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(w) |
                             reinterpret_cast<uintptr_t>(scaled) | reinterpret_cast<uintptr_t>(sum) | reinterpret_cast<uintptr_t>(normed);
  if (pointers & 15) return -1;
  return static_cast<int>(launch_pdl(rows::norm_rows_kernel, dim3(T), dim3(256), 0, s, (cbf)x, (cbf)residual, (cbf)w, eps, K, (bf)scaled, rstd, (bf)sum,
                                     (bf)normed));
}

// C[tokens, N] (bf16 or fp32) = X[tokens, K] · W[N, K]ᵀ (· row_scale[token]) (+ bias), tokens ≤ 64.  split: 1, 2, 4 or 8 slices of K.  static_w: no
// kernel that may still run on the stream writes W.  glu: W is [gate; up] of N / 2 rows each (a multiple of 64), C [tokens, N / 2] bf16 = silu(gate) · up, no bias.
extern "C" int mb_gemm_rows(const void* X, const void* W, void* C, int tokens, int N, int K, long long ldx, long long ldw, long long ldc, int out_fp32,
                            const void* bias, const float* row_scale, int split, int static_w, int glu, int* error_flag, cudaStream_t s) {
  using namespace mb;
  if (tokens <= 0 || N <= 0) return 0;
  if (glu && (N % rows::BMW || out_fp32 || bias != nullptr)) return -3;
  if (tokens > 64 || (split != 1 && split != 2 && split != 4 && split != rows::kMaxSplit)) return -2;
  const int bt = tokens <= 16 ? 16 : tokens <= 32 ? 32 : 64;
  CUtensorMap tw, tx;
  int r = make_tmap_bf16_2d(&tw, W, N, K, ldw, glu ? rows::BMW / 2 : rows::BMW, rows::BK);
  if (r) return 1000 + r;
  r = make_tmap_bf16_2d(&tx, X, tokens, K, ldx, bt, rows::BK);
  if (r) return 2000 + r;
  const rows::Params p{tokens, N, K, C, ldc, out_fp32, reinterpret_cast<const __nv_bfloat16*>(bias), row_scale, static_w, 0, error_flag, nullptr, 0};
  return glu ? rows::launch_mode<rows::kGluPair>(bt, tw, tx, p, split, s) : rows::launch_mode<rows::kPlain>(bt, tw, tx, p, split, s);
}

// C[tokens, N] bf16 = Σ_i X[tokens, i · F ..] · W[e_i]ᵀ over the slots[0] ≤ n_max experts e_i = slots[1 + i]: X [tokens, n_max · F], W [E, N, F], F a multiple of 64.
extern "C" int mb_gemm_rows_experts(const void* X, const void* W, void* C, int tokens, int N, int F, int E, int n_max, const int* slots, int* error_flag,
                                    cudaStream_t s) {
  using namespace mb;
  if (tokens <= 0 || N <= 0) return 0;
  if (tokens > 64 || F % rows::BK || E > rows::kMaxExperts) return -2;
  const int bt = tokens <= 16 ? 16 : tokens <= 32 ? 32 : 64;
  CUtensorMap tw, tx;
  int r = make_tmap_bf16_2d(&tw, W, static_cast<long long>(E) * N, F, F, rows::BMW, rows::BK);
  if (r) return 1000 + r;
  r = make_tmap_bf16_2d(&tx, X, tokens, static_cast<long long>(n_max) * F, static_cast<long long>(n_max) * F, bt, rows::BK);
  if (r) return 2000 + r;
  const rows::Params p{tokens, N, 0, C, N, 0, nullptr, nullptr, 0, 0, error_flag, slots, F / rows::BK};
  // two CTAs per SM: their prologue runs beside the kernel in front (16 tiles, 50 MB, 16 / 61 tokens with the norm in front of it: eight slices 14.2 / 17.1 µs,
  // four with an SM each 18 / 21)
  const int tiles = (N + rows::BMW - 1) / rows::BMW;
  const int split = tiles * 8 <= 2 * rows::kSms ? 8 : tiles * 4 <= 2 * rows::kSms ? 4 : tiles * 2 <= 2 * rows::kSms ? 2 : 1;
  return rows::launch_mode<rows::kExpertSum>(bt, tw, tx, p, split, s);
}
