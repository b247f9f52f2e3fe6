// Vocabulary head without logits in memory: hidden · Wᵀ on pairs of SMs (gemm_pair.cuh) whose epilogue reduces or differentiates the
// accumulator where it is.
//
//   head_stats   per row and 128 columns: {reference m, Σ 2^(z·log2e − m), Σ 2^(…)·z} with z = logit / temperature; the target's z
//   head_finish  the parts of a row → log p(target), entropy, log-sum-exp
//   head_grad    d logits (bf16) of (log p, entropy) for a range of the vocabulary, from the saved log-sum-exp
//
// What bounds it: the product itself.  The earlier form wrote fp32 logits for 16 384 columns at a time and read them back in kernels of
// their own: 1.2 MB per row and pass over the vocabulary, twice in a training step (statistics, gradients).
// Measured: log-probs of 17 829 tokens (hidden 2048, vocabulary 151 936, six MoE layers in front) 25.6 → 23.5 ms; a training step of 12 075
// tokens of the same model 76.0 → 72.8 ms.
// The exponentials (32 768 per 128 × 256 tile and CTA: 2048 clocks of the special-function unit) hide behind the product, which takes 8 192
// clocks or more for hidden sizes from 1024.
#include "gemm_pair.cuh"
#include "launch.h"

namespace mb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, long long rows, long long cols, long long ld, int box_rows, int box_cols);

namespace head {

static constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
static constexpr int kPart = 128;        // columns per part: half of a tile, what one epilogue warp holds of a row

struct Stats {
  const long long* targets;              // [M] (out of range: no target here)
  float4* parts;                         // [⌈N / 128⌉][M]: m (base 2), Σ, Σ·z
  float* target_z;                       // [M], written where the target is in range
  float inv_temp;

  template <int BN>
  __device__ __forceinline__ void tile(const GemmParams& p, int, int row0, uint32_t t_acc, uint8_t*, int n, int half, bool) const {
    constexpr int COLS = BN / 2;
    static_assert(COLS == kPart, "one part per warp");
    const uint32_t t_row = t_acc + half * COLS;
    const int col0 = n * BN + half * COLS;
    if (col0 >= p.N) return;                                  // uniform
    const int row = row0 + static_cast<int>(lane_id());
    const long long target = row < p.M ? targets[row] - col0 : -1;
    float m = -INFINITY;
    float2 s = make_float2(0.f, 0.f), e = make_float2(0.f, 0.f);
    const float2 l2e = make_float2(kLog2e, kLog2e);
#pragma unroll 1
    for (int c = 0; c < COLS / 32 && col0 + c * 32 < p.N; ++c) {
      uint32_t r[32];
      tmem_ld_32x32(t_row + c * 32, r);
      tmem_ld_wait();
      const int left = p.N - col0 - c * 32;                   // valid columns of these 32
      float2 z[16];
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        z[i] = make_float2(__uint_as_float(r[2 * i]) * inv_temp, __uint_as_float(r[2 * i + 1]) * inv_temp);
        if (left < 32) {
          if (2 * i >= left) z[i].x = -INFINITY;
          if (2 * i + 1 >= left) z[i].y = -INFINITY;
        }
        mx[i & 1] = max3(mx[i & 1], z[i].x, z[i].y);
      }
      // the reference only has to be near the maximum: everything is relative to the rounded value itself
      const float nm = fmaxf(m, fmaxf(mx[0], mx[1]) * kLog2e);
      if (nm > m) {
        const float a = exp2f(m - nm);                        // m = −∞: 0
        s.x *= a; s.y *= a; e.x *= a; e.y *= a;
        m = nm;
      }
      const float2 minus_m = make_float2(-m, -m);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float2 w = fma_f32x2(z[i], l2e, minus_m);
        w.x = exp2f(w.x);
        w.y = exp2f(w.y);
        s = add_f32x2(s, w);
        if (left < 32) {                                      // 0 · −∞
          if (2 * i >= left) z[i].x = 0.f;
          if (2 * i + 1 >= left) z[i].y = 0.f;
        }
        e = fma_f32x2(w, z[i], e);
      }
      const long long at = target - c * 32;
      if (at >= 0 && at < 32) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) t = at == i ? __uint_as_float(r[i]) : t;
        target_z[row] = t * inv_temp;
      }
    }
    if (row < p.M) __stcs(parts + static_cast<long long>(col0 / kPart) * p.M + row, make_float4(m, s.x + s.y, e.x + e.y, 0.f));
  }
};

struct Grad {
  const long long* targets;              // [M] (outside this range: none here)
  const float *lse, *ent, *g_lp, *g_ent; // [M]; ent and g_ent null without an entropy gradient, g_lp null without one of log p
  __nv_bfloat16* out;                    // [M, ld]
  long long ld;
  int first;                             // of the range
  float inv_temp;

  //   d z_j = g_lp·(1[j = target] − p_j) − g_ent·p_j·(z_j − (lse − H)),  d logit = d z · inv_temp,  p_j = exp(z_j − lse)
  template <int BN>
  __device__ __forceinline__ void tile(const GemmParams& p, int, int row0, uint32_t t_acc, uint8_t* stage, int n, int half, bool) const {
    constexpr int COLS = BN / 2;
    const uint32_t t_row = t_acc + half * COLS;
    const int col0 = n * BN + half * COLS;
    const int lane = static_cast<int>(lane_id()), row = row0 + lane;
    const bool in = row < p.M;
    const float l = in ? lse[row] : 0.f, glp = in && g_lp != nullptr ? g_lp[row] : 0.f, ge = in && g_ent != nullptr ? g_ent[row] : 0.f;
    const float mean = in && g_ent != nullptr ? l - ent[row] : 0.f;
    const long long target = in ? targets[row] - first - col0 : -1;
    const float2 minus_l = make_float2(-l, -l), l2e = make_float2(kLog2e, kLog2e), zero = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int c2 = 0; c2 < COLS / 64; ++c2) {
      const int colr = col0 + c2 * 64;
      if (colr >= p.N) break;                                 // uniform
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c2 * 64 + half * 32, r);
        tmem_ld_wait();
        const long long at = target - c2 * 64 - half * 32;
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 z = make_float2(__uint_as_float(r[2 * i]) * inv_temp, __uint_as_float(r[2 * i + 1]) * inv_temp);
          float2 w = fma_f32x2(add_f32x2(z, minus_l), l2e, zero);
          w.x = exp2f(w.x);
          w.y = exp2f(w.y);
          float2 d = make_float2(-glp * w.x, -glp * w.y);
          if (g_ent != nullptr) {
            d.x -= ge * w.x * (z.x - mean);
            d.y -= ge * w.y * (z.y - mean);
          }
          if (at == 2 * i) d.x += glp;
          if (at == 2 * i + 1) d.y += glp;
          packed[i] = pack_bf16x2(d.x * inv_temp, d.y * inv_temp);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((half * 4 + i) ^ (lane & 7)) << 4)) =
              make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
      }
      __syncwarp();
      const int unit = lane & 7, col = colr + unit * 8;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int rr = k * 4 + (lane >> 3);
        if (row0 + rr < p.M && col < p.N)
          *reinterpret_cast<uint4*>(out + static_cast<long long>(row0 + rr) * ld + col) =
              *reinterpret_cast<const uint4*>(stage + rr * 128 + ((unit ^ (rr & 7)) << 4));
      }
      __syncwarp();
    }
  }
};

// 32 rows per CTA (lane = row), the parts dealt to 8 warps
__global__ void __launch_bounds__(256) head_finish_kernel(const float4* parts, const float* target_z, int n_parts, long long R, float* logp, float* ent,
                                                          float* lse) {
  __shared__ float4 sh[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long r = blockIdx.x * 32ll + lane;
  float m = -INFINITY, s = 0.f, e = 0.f;
  auto add = [&](float4 x) {
    const float nm = fmaxf(m, x.x);
    if (nm == -INFINITY) {                       // nothing finite yet: keep a sum that is not a number, if there is one
      s += x.y; e += x.z;
      return;
    }
    const float a = exp2f(m - nm), b = exp2f(x.x - nm);
    s = s * a + x.y * b;
    e = e * a + x.z * b;
    m = nm;
  };
  if (r < R) {
#pragma unroll 4
    for (int i = warp; i < n_parts; i += 8) add(__ldcs(parts + static_cast<long long>(i) * R + r));
  }
  sh[warp][lane] = make_float4(m, s, e, 0.f);
  __syncthreads();
  if (warp == 0 && r < R) {
    for (int w = 1; w < 8; ++w) add(sh[w][lane]);
    const float l = (m + log2f(s)) * kLn2;
    logp[r] = target_z[r] - l;
    ent[r] = l - e / s;
    lse[r] = l;
  }
}

template <class Epi>
static int launch(const void* hidden, const void* W, const GemmParams& p, const Epi& epi, cudaStream_t s) {
  CUtensorMap ta, tb;
  int r = make_tmap_bf16_2d(&ta, hidden, p.M, p.K, p.K, pair::kBM, pair::kBK);
  if (r) return 1000 + r;
  r = make_tmap_bf16_2d(&tb, W, p.N, p.K, p.K, 128, pair::kBK);
  if (r) return 2000 + r;
  return pair::launch_pair<256, 0, 0, 0>(ta, tb, p, epi, ((p.M + 255) / 256) * ((p.N + 255) / 256), s);
}

}  // namespace head
}  // namespace mb

using namespace mb;

// hidden [R, H], W [V, H] (bf16, contiguous, H a multiple of 8); targets [R] in [0, V) where there is one; parts: ⌈V / 128⌉ · R · 4 floats.
extern "C" int mb_head_stats(const void* hidden, const void* W, const long long* targets, float* parts, float* target_z, int R, int V, int H,
                             float inv_temp, int* error_flag, cudaStream_t s) {
  if (R <= 0 || V <= 0) return 0;
  GemmParams p{};
  p.M = R; p.N = V; p.K = H; p.num_groups = 1; p.error_flag = error_flag;
  return head::launch(hidden, W, p, head::Stats{targets, reinterpret_cast<float4*>(parts), target_z, inv_temp}, s);
}

extern "C" int mb_head_finish(const float* parts, const float* target_z, int n_parts, long long R, float* logp, float* ent, float* lse, cudaStream_t s) {
  if (R <= 0) return 0;
  head::head_finish_kernel<<<static_cast<unsigned>((R + 31) / 32), 256, 0, s>>>(reinterpret_cast<const float4*>(parts), target_z, n_parts, R, logp, ent, lse);
  return static_cast<int>(cudaGetLastError());
}

// W: rows of the range, Vc of them (a multiple of 8) from number `first` of the vocabulary on; out [R, ld] bf16, 16-byte aligned rows.
extern "C" int mb_head_grad(const void* hidden, const void* W, const long long* targets, const float* lse, const float* ent, const float* g_lp,
                            const float* g_ent, void* out, long long ld, int R, int Vc, int first, int H, float inv_temp, int* error_flag,
                            cudaStream_t s) {
  if (R <= 0 || Vc <= 0) return 0;
  if (Vc % 8 || ld % 8 || reinterpret_cast<uintptr_t>(out) % 16) return -2;
  GemmParams p{};
  p.M = R; p.N = Vc; p.K = H; p.num_groups = 1; p.error_flag = error_flag;
  return head::launch(hidden, W, p, head::Grad{targets, lse, ent, g_lp, g_ent, reinterpret_cast<__nv_bfloat16*>(out), ld, first, inv_temp}, s);
}
