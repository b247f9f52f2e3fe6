// Experts of a decode step of 9 to 64 tokens without a sort: every expert that has some token multiplies ALL tokens.
//
//   moe_rows_up    act[t, s·F + f] = w(t, e_s) · silu(W13[e_s][f] · x_t) · (W13[e_s][F + f] · x_t),  0 where token t did not choose expert e_s
//   then           out[t, :] = act[t, :] · [W2[e_0] W2[e_1] …]ᵀ: one product whose reduction runs over the experts (gemm_rows.cu)
// with e_0, e_1, … the experts that have tokens, in order (`slots`).
//
// A step reads every chosen expert's weights once whatever it does with them, and the tensor cores have a token side of 64 to spare while they come: the
// sort, the gathered rows, the activation and the weighted sum of rows as kernels of their own only put launches and latencies around that.
// As in gemm_rows.cu the weight rows are the 128-row side of the MMA; a tile holds 64 gate rows and the 64 up rows of the same features, the
// activation is formed where the accumulator is read.  Two CTAs per SM and a tile each (more experts: several): with one CTA per SM the 192 tiles of 16
// experts would be two rounds.  16 experts of 2048 × 768, 8 choices, per layer of a decode step, sort + gather + products + activation + weighted sum → here: 61
// tokens 3.1 + 4.2 + 20.7 + 3.5 + 12.9 + 3.5 → 25.1 + 17.1 µs (bytes alone 15.4 + 7.7), 16 tokens 42.5 → 32.6.
//   warp 0 TMA, warp 1 tcgen05.mma (accumulator ×2), warps 2–5 epilogue: warps on the up rows hand theirs to the warps on the gate rows.
#include <cuda_bf16.h>

#include "launch.h"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);

namespace mrows {

static constexpr int kFeat = 64, BK = 64, kMaxExperts = 256;

struct Params {
  const int* topk_idx;
  const float* topk_w;
  __nv_bfloat16* act;      // [T, ld]
  int* slots;              // number of experts with tokens, then the experts
  long long ld;
  int T, k, E, offset, H, F;
  int* error_flag;
};

template <int BT>
struct Layout {
  static constexpr int kStages = BT == 64 ? 4 : 5;
  static constexpr int kABytes = 2 * kFeat * BK * 2;   // 64 gate rows, 64 up rows
  static constexpr int kBBytes = BT * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kUpBytes = BT * kFeat * 2;      // up sums on their way to the gate warps
  static constexpr int kTotal = kStages * kStageBytes + kUpBytes + 256 + 1024;
};

__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int BT>
__global__ void __launch_bounds__(192, 2)
moe_rows_up_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, Params p) {
  using L = Layout<BT>;
  constexpr int S = L::kStages;
  constexpr uint32_t kTmemCols = 2 * BT < 32 ? 32 : 2 * BT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + S * L::kABytes;
  __nv_bfloat16* ups = reinterpret_cast<__nv_bfloat16*>(smem + S * L::kStageBytes);       // [token][feature]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S * L::kStageBytes + L::kUpBytes);
  uint64_t* empty_bar = full_bar + S;
  uint64_t* tmem_full = empty_bar + S;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_ptr + 1);
  __shared__ uint32_t used[kMaxExperts / 32];
  __shared__ int slot_e[kMaxExperts], n_slots_s;
  __shared__ float weight[BT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 4); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (threadIdx.x < kMaxExperts / 32) used[threadIdx.x] = 0;
  if (warp == 1) {
    tmem_alloc(tmem_base_ptr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_ptr;
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i < p.T * p.k; i += 192) {
    const int e = p.topk_idx[i] - p.offset;
    if (e >= 0 && e < p.E) atomicOr(&used[e >> 5], 1u << (e & 31));
  }
  __syncthreads();
  if (warp == 0) {                                       // experts in order; lane l lists word l
    uint32_t bits = lane < kMaxExperts / 32 ? used[lane] : 0;
    int at = __popc(bits);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += v;
    }
    if (lane == 31) n_slots_s = at;
    for (at -= __popc(bits); bits; bits &= bits - 1) slot_e[at++] = lane * 32 + __ffs(bits) - 1;
  }
  __syncthreads();
  const int n_slots = n_slots_s, per = p.F / kFeat, total = n_slots * per, kbs = (p.H + BK - 1) / BK;
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i <= n_slots; i += 192) p.slots[i] = i == 0 ? n_slots : slot_e[i - 1];

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok && !*abort_flag; t += gridDim.x) {
        const int row = slot_e[t / per] * 2 * p.F + t % per * kFeat;
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { ok = false; break; }
          mbar_expect_tx(&full_bar[stage], L::kStageBytes);
          uint8_t* a = smem_a + stage * L::kABytes;
          tma_load_2d(a, &tmap_w, &full_bar[stage], kb * BK, row);
          tma_load_2d(a + L::kABytes / 2, &tmap_w, &full_bar[stage], kb * BK, row + p.F);
          tma_load_2d(smem_b + stage * L::kBBytes, &tmap_x, &full_bar[stage], kb * BK, 0);
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 52); }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * kFeat, BT, 0, 0);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok && !*abort_flag; t += gridDim.x) {
        if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1)) { ok = false; break; }
        tc_fence_after();
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a = smem_u32(smem_a + stage * L::kABytes), b = smem_u32(smem_b + stage * L::kBBytes);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16(tmem_base + acc * BT, make_smem_desc_sw128(a + k * 32, 16, 1024), make_smem_desc_sw128(b + k * 32, 16, 1024), idesc, (kb | k) != 0);
          umma_commit(&empty_bar[stage]);
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tmem_full[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 53); }
    }
  } else {
    const int q = warp & 3, tid = static_cast<int>(threadIdx.x) - 64;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const int slot = t / per, e = slot_e[slot] + p.offset;
      if (tid < p.T) {                                   // this expert's weight of every token, while the products run
        float w = 0.f;
        for (int j = 0; j < p.k; ++j)
          if (p.topk_idx[tid * p.k + j] == e) w += p.topk_w[tid * p.k + j];
        weight[tid] = w;
      }
      const bool ok = !*abort_flag && mbar_wait(&tmem_full[acc], acc_phase);       // a failure: no more waits, but every barrier below is met
      if (!ok) { *abort_flag = 1; atomicExch(p.error_flag, 54); }
      tc_fence_after();
      __syncwarp();
      const uint32_t from = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BT;
      float v[BT];
#pragma unroll
      for (int c = 0; c < BT / 16; ++c) {
        uint32_t r[16];
        tmem_ld_32x16(from + c * 16, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) v[c * 16 + i] = __uint_as_float(r[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      if (q >= 2) {
#pragma unroll
        for (int i = 0; i < BT; ++i)
          if (i < p.T) ups[i * kFeat + (q - 2) * 32 + lane] = __float2bfloat16(v[i]);
      }
      epilogue_sync();
      if (q < 2) {
        const int f = q * 32 + lane;
        __nv_bfloat16* to = p.act + static_cast<long long>(slot) * p.F + t % per * kFeat + f;
#pragma unroll
        for (int i = 0; i < BT; ++i) {
          if (i >= p.T) break;
          // gate and up are rounded to bf16 first, like the stored pre-activation of the general path
          const float g = __bfloat162float(__float2bfloat16(v[i])), w = weight[i];
          to[i * p.ld] = __float2bfloat16(w != 0.f ? g / (1.f + __expf(-g)) * __bfloat162float(ups[i * kFeat + f]) * w : 0.f);
        }
      }
      epilogue_sync();                                   // `ups` and `weight` are written again
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int BT>
static int launch(const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int tiles, cudaStream_t s) {
  static const cudaError_t configured = cudaFuncSetAttribute(moe_rows_up_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<BT>::kTotal);
  if (configured != cudaSuccess) return static_cast<int>(configured);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return static_cast<int>(launch_pdl(moe_rows_up_kernel<BT>, dim3(tiles < 2 * sms ? tiles : 2 * sms), dim3(192), Layout<BT>::kTotal, s, tw, tx, p));
}

}  // namespace mrows
}  // namespace mb

// out [T, H] = Σ_j w[t, j] · W2[e] · (silu(W13[e][:F] · x_t) · (W13[e][F:] · x_t)), e = idx[t, j] − offset in [0, E), 1 to 64 tokens.  act: [T, n · F] scratch with
// n = min(E, T · k), slots: 1 + n ints of scratch.  E ≤ 256, H a multiple of 8, F of 64; x, act and the weights 16-byte aligned.
extern "C" int mb_moe_rows(const void* x, const void* w13, const void* w2, const int* topk_idx, const float* topk_w, void* act, int* slots, void* out, int T,
                           int k, int E, int offset, int H, int F, int* error_flag, cudaStream_t s) {
  using namespace mb;
  if (T <= 0) return 0;
  if (T > 64 || k < 1 || E < 1 || E > mrows::kMaxExperts || H % 8 || F % mrows::kFeat) return -1;
  const int bt = T <= 16 ? 16 : T <= 32 ? 32 : 64, n = T * k < E ? T * k : E;
  CUtensorMap tw, tx;
  int r = make_tmap_bf16_2d(&tw, w13, 2ll * E * F, H, H, mrows::kFeat, mrows::BK);
  if (r) return 1000 + r;
  r = make_tmap_bf16_2d(&tx, x, T, H, H, bt, mrows::BK);
  if (r) return 2000 + r;
  const mrows::Params p{topk_idx, topk_w, reinterpret_cast<__nv_bfloat16*>(act), slots, static_cast<long long>(n) * F, T, k, E, offset, H, F, error_flag};
  const int tiles = n * (F / mrows::kFeat);
  r = bt == 16 ? mrows::launch<16>(tw, tx, p, tiles, s) : bt == 32 ? mrows::launch<32>(tw, tx, p, tiles, s) : mrows::launch<64>(tw, tx, p, tiles, s);
  if (r) return r;
  return mb_gemm_rows_experts(act, w2, out, T, H, F, E, n, slots, error_flag, s);
}
